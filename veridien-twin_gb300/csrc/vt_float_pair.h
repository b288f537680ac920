// Sums of float pairs (hi, lo) that lose nothing of FP64's precision, in float32 operations. Additions alone, so that neither
// compiler has a product to contract.
#pragma once

#if defined(__CUDACC__)
#define VT_FLOAT_PAIR __host__ __device__ __forceinline__
#else
#define VT_FLOAT_PAIR inline
#endif

namespace vtk {

// the value h + m + l
struct Df3 { float h, m, l; };

// s + e = a + b exactly (Knuth)
VT_FLOAT_PAIR void two_sum(float a, float b, float& s, float& e) {
  s = a + b;
  const float v = s - a;
  e = (a - (s - v)) + (b - v);
}
// good to about 2^-70 of |x| + |y|: what the two upper parts drop goes to the third. A pair has its last bit at 2^-48, and to
// round to that at each step of a tree costs more than the products of a short row do
VT_FLOAT_PAIR Df3 df_add(const Df3& x, const Df3& y) {
  float t, e1, e2, e3;
  Df3 r;
  two_sum(x.h, y.h, r.h, e1);
  two_sum(x.m, y.m, t, e2);
  two_sum(t, e1, r.m, e3);
  r.l = (x.l + y.l) + (e2 + e3);
  return r;
}
VT_FLOAT_PAIR double df_double(const Df3& x) { return double(x.h) + (double(x.m) + double(x.l)); }

}  // namespace vtk
