"""The order of the calibration's node-radiosity sums (csrc/vt_calib.cu radiosity64_kernel, with csrc/vt_float_pair.h itself) against
exact sums, beside a warp per row whose lanes' float pairs meet in FP64: at no length of a row is its error the larger one."""
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
static P add(P x, P y) {
  const float t = x.h + y.h, v = t - x.h, lo = (x.l + y.l) + ((x.h - (t - v)) + (y.h - v)), h = t + lo;
  return {h, lo - (h - t)};
}
static P split(double d) { const float h = float(d); return {h, float(d - double(h))}; }

struct Row { std::vector<float> F; std::vector<P> x; };

// a warp per row: 128-bit loads where they can be, a float pair a lane, the lanes in FP64
static double warp_per_row(const Row& r) {
  const int n = int(r.F.size());
  double s[32], t[32];
  for (int l = 0; l < 32; l++) {
    P a{0, 0};
    if (n % 4 == 0) { for (int j = l; j < n / 4; j += 32) for (int q = 0; q < 4; q++) mac(r.F[4 * j + q], r.x[4 * j + q], a); }
    else for (int j = l; j < n; j += 32) mac(r.F[j], r.x[j], a);
    s[l] = double(a.h) + double(a.l);
  }
  for (int o = 16; o; o >>= 1) {
    for (int l = 0; l < 32; l++) t[l] = s[l] + s[l ^ o];
    std::copy(t, t + 32, s);
  }
  return s[0];
}
template <typename V, typename Add>
static V tree(V* v, Add plus) {
  V t[32];
  for (int o = 16; o; o >>= 1) {
    for (int l = 0; l < 32; l++) t[l] = plus(v[l], v[l ^ o]);
    std::copy(t, t + 32, v);
  }
  return v[0];
}
// radiosity64_kernel
static double block(const Row& r) {
  const int n = int(r.F.size());
  const bool is_short = n <= 768;
  double sum = 0;
  for (int w = 0; w < 8; w++) {
    P p[32];
    vtk::Df3 d[32];
    for (int l = 0; l < 32; l++) {
      P a[2][2] = {};
      for (int j = 4 * (32 * w + l); j < n; j += 1024)
        for (int q = 0; q < 4 && j + q < n; q++) mac(r.F[j + q], r.x[j + q], a[is_short ? q / 2 : 0][q % 2]);
      auto df3 = [&](const P& s) { return vtk::Df3{s.h, s.l, 0.0f}; };
      p[l] = add(a[0][0], a[0][1]);
      d[l] = vtk::df_add(vtk::df_add(df3(a[0][0]), df3(a[0][1])), vtk::df_add(df3(a[1][0]), df3(a[1][1])));
    }
    if (is_short) {
      sum += vtk::df_double(tree(d, [](vtk::Df3 x, vtk::Df3 y) { return vtk::df_add(x, y); }));
    } else {
      const P s = tree(p, add);
      sum += double(s.h) + double(s.l);
    }
  }
  return sum;
}

int main() {
  std::mt19937_64 g(1);
  std::uniform_real_distribution<double> U(0, 1);
  int worse = 0;
  for (int sign = 0; sign < 2; sign++)
    for (int n : {1, 2, 3, 5, 16, 31, 64, 100, 130, 257, 512, 700, 768, 769, 1000, 1025, 1500, 2048, 3000, 4096}) {
      double a2 = 0, b2 = 0;
      for (int rep = 0; rep < 1500; rep++) {
        Row r;
        long double exact = 0, size = 0;
        for (int j = 0; j < n; j++) {
          const double u = U(g), d = 0.05 + 3 * U(g);
          r.F.push_back(float(u * u * u / n));
          r.x.push_back(split(sign && U(g) < 0.5 ? -d : d));
          const long double q = (long double)r.F[j] * ((long double)r.x[j].h + r.x[j].l);
          exact += q;
          size += std::fabs(double(q));
        }
        const double a = double((warp_per_row(r) - exact) / size), b = double((block(r) - exact) / size);
        a2 += a * a;
        b2 += b * b;
      }
      std::printf("%s n = %4d: a warp per row %.2e, the block %.2e\n", sign ? "+-" : "+ ", n, std::sqrt(a2 / 1500), std::sqrt(b2 / 1500));
      // the rms of 1500 rows is known to 1 / sqrt(2 x 1500) of itself, and most rounding errors of the two are the same
      worse += std::sqrt(b2) > 1.02 * std::sqrt(a2);
    }
  return worse;
}
'''


@pytest.mark.skipif(shutil.which("g++") is None, reason="g++ absent")
def test_block_sums_are_as_good_as_fp64_over_the_lanes(tmp_path):
    src, exe = tmp_path / "tree.cpp", tmp_path / "tree"
    src.write_text(PROGRAM)
    # every product and sum rounded by itself, as the kernel's intrinsics do
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-Wall", "-Wextra", "-Werror", "-I", os.path.join(ROOT, "veridien-twin_gb300", "csrc"),
                    str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    print(out.stdout)
    assert out.returncode == 0, out.stdout
