"""The order of the calibration's adjoint sums (csrc/vt_calib.cu jacobi_t_kernel and jacobi_t_combine, with csrc/vt_float_pair.h
itself) against exact sums, beside float-pair chains that meet in FP64: the error is not the larger one."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

PROGRAM = r'''
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

#include "vt_float_pair.h"

struct P { float h, l; };
static void mac(float f, P x, P& s) {
  const float p = f * x.h, e = std::fmaf(f, x.l, std::fmaf(f, x.h, -p)), t = s.h + p, v = t - s.h;
  const float lo = s.l + (((s.h - (t - v)) + (p - v)) + e);
  s.h = t + lo;
  s.l = lo - (s.h - t);
}
static P split(double d) { const float h = float(d); return {h, float(d - double(h))}; }

int main() {
  std::mt19937_64 g(1);
  std::uniform_real_distribution<double> U(0, 1);
  int worse = 0;
  for (int sign = 0; sign < 2; sign++)
    for (int n : {1, 63, 64, 65, 130, 257, 512, 1000, 1024, 2048, 3001, 4096, 8192}) {
      double a2 = 0, b2 = 0;
      for (int rep = 0; rep < 1500; rep++) {
        const int rows = (n + 63) / 64;
        double fp64 = 0;
        vtk::Df3 warp[8] = {};
        long double exact = 0, size = 0;
        for (int s = 0; s < 64; s++) {
          P a[2] = {};
          for (int i = s * rows; i < std::min(n, (s + 1) * rows); i++) {
            const double u = U(g), d = 0.05 + 3 * U(g);
            const float F = float(u * u * u / n);
            const P x = split(sign && U(g) < 0.5 ? -d : d);
            const long double q = (long double)F * ((long double)x.h + x.l);
            exact += q;
            size += std::fabs(double(q));
            mac(F, x, a[(i - s * rows) % 2]);
          }
          fp64 += (double(a[0].h) + double(a[0].l)) + (double(a[1].h) + double(a[1].l));
          const vtk::Df3 v = vtk::df_add(vtk::Df3{a[0].h, a[0].l, 0.0f}, vtk::Df3{a[1].h, a[1].l, 0.0f});
          warp[s / 8] = vtk::df_add(warp[s / 8], v);
        }
        vtk::Df3 sum = warp[0];
        for (int w = 1; w < 8; w++) sum = vtk::df_add(sum, warp[w]);
        const double a = double((fp64 - exact) / size), b = double((vtk::df_double(sum) - exact) / size);
        a2 += a * a;
        b2 += b * b;
      }
      std::printf("%s n = %4d: chains that meet in FP64 %.2e, in three parts %.2e\n", sign ? "+-" : "+ ", n, std::sqrt(a2 / 1500), std::sqrt(b2 / 1500));
      // the same chains; what they meet in adds up to 2^-53 of the sum where it is FP64, once where it is three parts
      worse += std::sqrt(b2) > 1.02 * std::sqrt(a2);
    }
  return worse;
}
'''


@pytest.mark.skipif(shutil.which("g++") is None, reason="g++ absent")
def test_column_sums_are_as_good_as_fp64_over_the_splits(tmp_path):
    src, exe = tmp_path / "columns.cpp", tmp_path / "columns"
    src.write_text(PROGRAM)
    # every product and sum rounded by itself, as the kernel's intrinsics do
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-Wall", "-Wextra", "-Werror", "-I", os.path.join(ROOT, "veridien-twin_gb300", "csrc"),
                    str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    print(out.stdout)
    assert out.returncode == 0, out.stdout
