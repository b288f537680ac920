// Differentiable calibration render on sm_103a. The reference has no differentiation (only the analytic dtheta_d /
// dtheta of gpu/lens.js:25); this is the project's own estimator, built from the twin's pieces so that its gradient
// with respect to material albedos and emitter radiances can be computed by path replay.
//
// Estimator (per camera sub-sample, the KB4 ray and sample numbers of the path tracer, gpu/wgsl/kernels.wgsl.js
// :34-53): up to D vertices on Lambertian surfaces (f = rho / pi). At every vertex, nL emitter samples (area CDF,
// power-heuristic MIS against cosine sampling, gpu/wgsl/shade.wgsl.js:135 lightEval); between vertices, cosine-
// weighted continuation, so the throughput gains exactly rho per bounce; at vertex D, the light the node radiosity
// carries: rho / pi x H(node), H = F B the irradiance from the other nodes. An emitter hit adds its radiance
// (MIS-weighted after the first vertex). Nothing in the sampling depends on the parameters, so the estimator is a
// polynomial in the albedos, linear in the emitter radiances and in H, and its derivative is exact by replay:
// each path's record (its vertices' materials and nodes, its light samples' contributions) is differentiated term by
// term, and the derivatives are accumulated in FP64.
//
// The paths are traced by the wavefront kernels of the path tracer (closest hit, then calib_shade, then
// calib_shadow), which write each path's record. When the records of every path fit in memory the backward reads the
// forward's records; otherwise the paths are traced again in chunks of sub-samples, each chunk's records
// differentiated before the next is traced. Both forms trace the same paths with the same kernels, so the replayed
// records are bit-identical to the forward's.
#include <utility>

#include "vt_calib.cuh"
#include "vt_calib_tan.cuh"
#include "vt_camera.cuh"
#include "vt_float_pair.h"
#include "vt_wave.cuh"

namespace vtk {
using namespace vtd;

namespace {
constexpr int CT = 128;

// append `want` lanes' items to a queue with one atomic per warp; returns the slot of this lane (if want)
__device__ __forceinline__ uint32_t warp_append_c(uint32_t* count, bool want) {
  const uint32_t act = __activemask();
  const uint32_t mask = __ballot_sync(act, want);
  if (!mask) return 0;
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t leader = __ffs(mask) - 1;
  uint32_t base = 0;
  if (lane == leader) base = atomicAdd(count, uint32_t(__popc(mask)));
  base = __shfl_sync(act, base, leader);
  return base + __popc(mask & ((1u << lane) - 1u));
}

// Path records, in 32-bit words. 32 paths' records lie together, word by word (word k of record r at 32 k + r % 32 of its
// group), so that a warp's accesses to a word are one or two lines: with a record to itself each was a line per lane, and
// calib_shade, whose bound that was, took 971 us for 2.3 M paths (now 357; a calibration step of three 480 x 300 cameras, 16 sub-samples:
// 31.6 -> 27.1 ms)
template <typename Word>
struct RecordOf {
  Word* w;
  __device__ __forceinline__ uint32_t get(uint32_t k) const { return w[32u * k]; }
  __device__ __forceinline__ float getf(uint32_t k) const { return __uint_as_float(w[32u * k]); }
  __device__ __forceinline__ float3 get3(uint32_t k) const { return f3(getf(k), getf(k + 1u), getf(k + 2u)); }
  __device__ __forceinline__ void put(uint32_t k, uint32_t v) const { w[32u * k] = v; }
  __device__ __forceinline__ void putf(uint32_t k, float v) const { w[32u * k] = __float_as_uint(v); }
  __device__ __forceinline__ void put3(uint32_t k, float3 v) const { putf(k, v.x); putf(k + 1u, v.y); putf(k + 2u, v.z); }
};
using Record = RecordOf<uint32_t>;
using ConstRecord = RecordOf<const uint32_t>;
template <typename Word>
__device__ __forceinline__ RecordOf<Word> record_at(Word* base, uint32_t words, size_t r) { return {base + (r >> 5) * 32u * words + (r & 31u)}; }

// a path: its shading vertices, the emitter hit after them (~0: none) with its MIS weight x profile, the node term at the
// last of them (~0: none); per vertex the material, and per light sample the lamp and the contribution per unit emitter
// radiance, per unit albedo (0: no contribution)
constexpr uint32_t CP_N = 0, CP_EMIT_LAMP = 1, CP_EMIT_A = 2, CP_NODE = 3, CP_VERTEX = 4, CP_VERTEX_WORDS = 1 + 2 * CAL_MAX_NL;
constexpr uint32_t CP_WORDS = CP_VERTEX + CAL_MAX_DEPTH * CP_VERTEX_WORDS;
__device__ __forceinline__ uint32_t cp_mat(uint32_t k) { return CP_VERTEX + k * CP_VERTEX_WORDS; }
__device__ __forceinline__ uint32_t cp_lamp(uint32_t k, uint32_t j) { return cp_mat(k) + 1u + j; }
__device__ __forceinline__ uint32_t cp_q(uint32_t k, uint32_t j) { return cp_mat(k) + 1u + CAL_MAX_NL + j; }

// the derivative record of a path in d0 (stored form, kept only when the intrinsics' derivative is asked for): each
// light sample's dq (per unit emitter radiance and albedo; meant where the path's q is not 0), the emitter hit's d a (meant
// where it has one), the ray's tangents between bounces, and the triangle and instance each bounce hit (~0: none)
constexpr uint32_t CT_DQ = 0, CT_DE = CAL_MAX_DEPTH * CAL_MAX_NL * 3, CT_JO = CT_DE + 3, CT_JD = CT_JO + 9, CT_DPB = CT_JD + 9, CT_TRI = CT_DPB + 3,
                   CT_INST = CT_TRI + CAL_MAX_DEPTH, CT_WORDS = CT_INST + CAL_MAX_DEPTH;
__device__ __forceinline__ uint32_t ct_dq(uint32_t k, uint32_t j) { return CT_DQ + (k * CAL_MAX_NL + j) * 3u; }
__device__ __forceinline__ Tan3 get_tan(const Record& G, uint32_t k) {
  Tan3 J;
  for (uint32_t c = 0; c < 3; c++) J.c[c] = G.get3(k + 3u * c);
  return J;
}
__device__ __forceinline__ void put_tan(const Record& G, uint32_t k, const Tan3& J) {
  for (uint32_t c = 0; c < 3; c++) G.put3(k + 3u * c, J.c[c]);
}

// a path's discrete decisions (replay form): per bounce the triangle its extension ray met (~0: none) and, a byte each, the
// instance (0xff: none), and one bit per vertex and light sample, set when that sample's shadow ray was occluded
constexpr uint32_t CD_TRI = 0, CD_INST = CAL_MAX_DEPTH, CD_OCC = CD_INST + 1, CD_WORDS = CD_OCC + 1;
static_assert(CAL_MAX_DEPTH <= 4, "a word of instance bytes");
static_assert(CAL_MAX_DEPTH * CAL_MAX_NL <= 32, "one occlusion bit per vertex and light sample");
static_assert(VT_MAX_INST < 0xff, "instances fit a byte");

// emitter sample by the area CDF, with the index of the triangle (gpu/wgsl/shade.wgsl.js:31)
__device__ __forceinline__ uint32_t sample_emitter_idx(const Scene& S, float3 u, float time, float3& p, float3& n, float3& axis) {
  uint32_t lo = 0, hi = S.emit_n - 1u;
  for (uint32_t it = 0; it < 40u && lo < hi; it++) {
    const uint32_t m = (lo + hi) >> 1;
    if (__ldg(S.params + S.emit_off + 4u * m).w < u.x) lo = m + 1u; else hi = m;
  }
  const float4* e = S.params + S.emit_off + 4u * lo;
  const float3 v0 = xyz(__ldg(e)), e1 = xyz(__ldg(e + 1)), e2 = xyz(__ldg(e + 2)), nl = xyz(__ldg(e + 3));
  const float su = sqrtf(u.y);
  const float3 pl = v0 + e1 * (su * (1.0f - u.z)) + e2 * (su * u.z);
  Rot R;
  float3 pp;
  inst_pose(S, ldu(S.su + 17), time, R, pp);
  p = rmul(R, pl) + pp;
  n = rmul(R, nl);
  axis = rmul(R, ld3(S.su + 4));
  return lo;
}

__device__ __forceinline__ float3 alb(const CalibDev& C, uint32_t m) { return f3(__ldg(C.albedo + 3 * m), __ldg(C.albedo + 3 * m + 1), __ldg(C.albedo + 3 * m + 2)); }

// the emitter hit's weight a = w prof (w = 1 at the first vertex, else pb^2 / (pb^2 + nl^2 pL^2) with
// pL = t^2 / (cosE area)) and its derivative, given the tangents of the ray, of the hit distance and of the
// previous vertex's continuation pdf pb
__device__ __forceinline__ float3 tan_emitter_hit(const Scene& S, const Hit& h, const Surf& s, float3 d, float tt, uint32_t b, float pb, float3 dpb,
                                                 float fnl, float area, const Tan3& Jd, const Tan3& Jx, float3 dt) {
  Tan3 JnE;
  const float3 nE = tan_interp_normal(S, h, s, tt, Jx, JnE);
  const float3 axis = emitter_axis_at(S, tt);
  const float c = clampf(dot(-d, axis), -1.0f, 1.0f);
  const float th = acosf(c);
  const float prof = profile(S, th), slope = profile_slope(S, th);
  const float cosE = dot(-d, nE);
  const float pL = h.t * h.t / (cosE * area);
  const float A = pb * pb, B = fnl * fnl * pL * pL, AB = A + B;
  const float w = b > 1 ? A / AB : 1.0f;
  const float dtv[3] = {dt.x, dt.y, dt.z}, dpbv[3] = {dpb.x, dpb.y, dpb.z};
  float out[3];
  for (int j = 0; j < 3; j++) {
    const float dc = -dot(axis, Jd.c[j]);
    const float dth = (1.0f - c * c) > 0.0f ? -dc / sqrtf(1.0f - c * c) : 0.0f;
    float dw = 0.0f;
    if (b > 1) {
      const float dcosE = -dot(Jd.c[j], nE) - dot(d, JnE.c[j]);
      const float dpL = (2.0f * h.t * dtv[j] * cosE - h.t * h.t * dcosE) / (cosE * cosE * area);
      const float dA = 2.0f * pb * dpbv[j], dB = 2.0f * fnl * fnl * pL * dpL;
      dw = (dA * B - A * dB) / (AB * AB);
    }
    out[j] = dw * prof + w * slope * dth;
  }
  return f3(out[0], out[1], out[2]);
}

// a path's vertices at once, before it is known how many there are: the records come from HBM
struct PathWords {
  uint32_t mat[CAL_MAX_DEPTH], lamp[CAL_MAX_DEPTH][CAL_MAX_NL];
  float q[CAL_MAX_DEPTH][CAL_MAX_NL];
};
__device__ __forceinline__ PathWords path_words(const ConstRecord& P, uint32_t depth, uint32_t nl) {
  PathWords W;
#pragma unroll
  for (uint32_t k = 0; k < CAL_MAX_DEPTH; k++) {
    W.mat[k] = k < depth ? P.get(cp_mat(k)) : 0u;
#pragma unroll
    for (uint32_t j = 0; j < CAL_MAX_NL; j++) {
      const bool on = k < depth && j < nl;
      W.q[k][j] = on ? P.getf(cp_q(k, j)) : 0.0f;
      W.lamp[k][j] = on ? P.get(cp_lamp(k, j)) : 0u;
    }
  }
  return W;
}

// one rounding each in this order, whatever the compiler knows of the operands in an unrolled loop
__device__ __forceinline__ float3 mac3(float3 a, float b, float3 c) { return f3(__fmaf_rn(a.x, b, c.x), __fmaf_rn(a.y, b, c.y), __fmaf_rn(a.z, b, c.z)); }
__device__ __forceinline__ float dot_fma(float3 a, float3 b) { return __fmaf_rn(a.z, b.z, __fmaf_rn(a.x, b.x, __fmul_rn(a.y, b.y))); }

// radiance of a recorded path
__device__ __forceinline__ float3 path_value(const CalibDev& C, const ConstRecord& P, uint32_t depth, uint32_t nl) {
  const uint32_t n = P.get(CP_N), node = P.get(CP_NODE), lamp = P.get(CP_EMIT_LAMP);
  const PathWords W = path_words(P, depth, nl);
  const float emit_a = P.getf(CP_EMIT_A);
  float3 L = f3(0, 0, 0), T = f3(1, 1, 1);
#pragma unroll
  for (uint32_t k = 0; k < CAL_MAX_DEPTH; k++) {
    if (k >= n) continue;
    const float3 rho = alb(C, W.mat[k]);
    float s = 0.0f;
#pragma unroll
    for (uint32_t j = 0; j < CAL_MAX_NL; j++) {
      const float q = W.q[k][j];
      if (j < nl && q != 0.0f) s += __ldg(C.lamp + W.lamp[k][j]) * q;
    }
    const float3 Tr = T * rho;
    L = mac3(Tr, s / float(nl), L);
    if (k + 1 == n && node != MISS) {
      const float3 Hn = f3(__ldg(C.H + node), __ldg(C.H + C.n_nodes + node), __ldg(C.H + 2 * C.n_nodes + node));
      L = mac3(Tr * Hn, INV_PI_F, L);
    }
    T = Tr;
  }
  if (lamp != MISS) L = mac3(T, emit_a * __ldg(C.lamp + lamp), L);
  return L;
}

// a path's albedo gradient: per vertex its material and g-weighted value (on: the vertex exists)
struct AlbGrad {
  uint32_t mat[CAL_MAX_DEPTH];
  float3 val[CAL_MAX_DEPTH];
  bool on[CAL_MAX_DEPTH];
};

// d loss / d parameters of one recorded path, given g = d loss / d (path radiance); FP64 into shared accumulators
__device__ __forceinline__ void path_grad(const CalibDev& C, const ConstRecord& P, uint32_t depth, uint32_t nl, float3 g, double* sh_lamp, AlbGrad& ag) {
  const uint32_t n = P.get(CP_N), node = P.get(CP_NODE), lamp = P.get(CP_EMIT_LAMP);
  const float emit_a = P.getf(CP_EMIT_A);
  const PathWords W = path_words(P, depth, nl);
  // Each term is formed in FP32 and added to the FP64 accumulators (FP64 arithmetic runs at a small fraction of
  // this part's FP32 rate; the reductions stay FP64). A term whose albedo product ends at vertex k adds
  // g o value / rho_l to every vertex l <= k: D[k] gathers the g-weighted values of the terms ending at k, and vertex
  // l receives (sum_{k >= l} D[k]) / rho_l, which the caller sums over the warp per material.
  const float fnl = float(nl);
  float3 T = f3(1, 1, 1);
  float3 D[CAL_MAX_DEPTH], rho[CAL_MAX_DEPTH];
#pragma unroll
  for (uint32_t k = 0; k < CAL_MAX_DEPTH; k++) {
    D[k] = f3(0, 0, 0);
    rho[k] = f3(1, 1, 1);
    if (k >= n) continue;
    rho[k] = alb(C, W.mat[k]);
    T = T * rho[k];
    float s = 0.0f;
#pragma unroll
    for (uint32_t j = 0; j < CAL_MAX_NL; j++) {
      const float q = W.q[k][j];
      if (j >= nl || q == 0.0f) continue;
      atomicAdd(sh_lamp + W.lamp[k][j], double(dot_fma(g, T) * q / fnl));
      s += __ldg(C.lamp + W.lamp[k][j]) * q;
    }
    if (s != 0.0f) D[k] = D[k] + g * T * (s / fnl);
    if (k + 1 == n && node != MISS) {
      const float ip = 0.318309886183790672f;
      const float3 Hn = f3(__ldg(C.H + node), __ldg(C.H + C.n_nodes + node), __ldg(C.H + 2 * C.n_nodes + node));
      atomicAdd(C.g_H + node, double(g.x * T.x * ip));
      atomicAdd(C.g_H + C.n_nodes + node, double(g.y * T.y * ip));
      atomicAdd(C.g_H + 2 * C.n_nodes + node, double(g.z * T.z * ip));
      D[k] = D[k] + g * T * Hn * ip;
    }
  }
  if (lamp != MISS && emit_a != 0.0f) {
    atomicAdd(sh_lamp + lamp, double(dot_fma(g, T) * emit_a));
    if (n) {
      const float Le = emit_a * __ldg(C.lamp + lamp);
#pragma unroll
      for (uint32_t k = 0; k < CAL_MAX_DEPTH; k++)
        if (k + 1 == n) D[k] = D[k] + g * T * Le;
    }
  }
  float3 acc = f3(0, 0, 0);
#pragma unroll
  for (int k = CAL_MAX_DEPTH - 1; k >= 0; k--) {
    ag.on[k] = uint32_t(k) < n;
    if (!ag.on[k]) continue;
    acc = acc + D[k];
    ag.mat[k] = W.mat[k];
    ag.val[k] = f3(acc.x / rho[k].x, acc.y / rho[k].y, acc.z / rho[k].z);
  }
}

// Adds each lane's value (on: it has one) to sh[3 key + c]: the lanes with the same key are summed over the warp in
// FP32 (a fixed butterfly, so the sum depends only on the warp's lanes), then one FP64 shared atomic per key and
// channel. Called by all 32 lanes of the warp.
__device__ __forceinline__ void warp_key_add3(double* sh, uint32_t key, float3 v, bool on) {
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t pending = __ballot_sync(0xffffffffu, on);
  while (pending) {
    const uint32_t leader = __ffs(pending) - 1;
    const uint32_t k0 = __shfl_sync(0xffffffffu, key, leader);
    const bool in = on && key == k0;
    pending &= ~__ballot_sync(0xffffffffu, in);
    float a = in ? v.x : 0.0f, b = in ? v.y : 0.0f, c = in ? v.z : 0.0f;
    for (int o = 16; o > 0; o >>= 1) {
      a += __shfl_xor_sync(0xffffffffu, a, o);
      b += __shfl_xor_sync(0xffffffffu, b, o);
      c += __shfl_xor_sync(0xffffffffu, c, o);
    }
    if (lane < 3u) atomicAdd(sh + 3 * k0 + lane, double(lane == 0u ? a : lane == 1u ? b : c));   // one compare-and-swap loop, not three
    if (in) on = false;
  }
}

// ------------------------------------------------------------------------------------ the wavefront estimator
// The estimator split like the path tracer: the closest-hit kernel of the wavefront, then calib_shade (one vertex:
// the record of the vertex, its light samples' unshadowed contributions and shadow segments, the cosine
// continuation), then calib_shadow (any hit per light sample; an occluded sample's contribution is cleared in the
// record). Each path's record stays in HBM, so the backward evaluates path_grad on the records without
// tracing again. The record of path (i, id) of a camera's sub-samples [i0, i1) is record (i - i0) n_pix + id; a wave's
// begin at r0.
constexpr int WT = 256;

template <bool TAN>
__global__ void __launch_bounds__(WT, 3) calib_shade_kernel(const Scene S, const CamParams cp, const CalibDev C, WaveBufs wb, uint32_t* rec,
                                                        uint32_t* tan, size_t r0, uint32_t b, uint32_t* dec, size_t d0, int dmode) {
  const uint32_t n = *wb.count_in;
  const uint32_t nl = cp.n_light;
  const float fnl = float(nl);
  const float area = __ldg(S.su + 3);
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    const uint32_t p = wb.q_in[k];
    const Record P = record_at(rec, CP_WORDS, r0 + p);
    if (b == 1) { P.put(CP_N, 0u); P.put(CP_EMIT_LAMP, MISS); P.putf(CP_EMIT_A, 0.0f); P.put(CP_NODE, MISS); }
    const uint4 meta = wb.meta[p];
    const uint32_t i = meta.y, hs = meta.z;
    const float4 o4 = wb.o[p], d4 = wb.d[p], hv = wb.hit[p];
    const float3 o = xyz(o4), d = xyz(d4);
    const float tt = o4.w, pb_prev = d4.w;
    const Hit h{hv.x, hv.y, hv.z, __float_as_uint(hv.w), wb.hinst[p]};
    const Record D = record_at(dec, CD_WORDS, d0 + p);
    if (dmode == 1) {
      // every bounce of the path starts as none: a replay whose path continues where the recorded one stopped (its
      // rays can differ from the recorded ones in the last bits) meets nothing there, never a stale triangle
      if (b == 1) {
        D.put(CD_OCC, 0u);
        for (uint32_t a = 1; a < CAL_MAX_DEPTH; a++) D.put(CD_TRI + a, MISS);
      }
      D.put(CD_TRI + b - 1, h.tri);
      const uint32_t at = 8u * (b - 1u), inst = h.inst == MISS ? 0xffu : h.inst;
      D.put(CD_INST, ((b == 1 ? MISS : D.get(CD_INST)) & ~(0xffu << at)) | inst << at);
    }
    const uint32_t occ = dmode == 2 ? D.get(CD_OCC) : 0u;
    bool cont = false, shadow = false;
    const Record G = record_at(tan, CT_WORDS, r0 + p);
    Tan3 Jo, Jd, Jx;
    float3 dpb, dt;
    if (TAN) {
      if (b == 1) {
        for (uint32_t a = 1; a < cp.max_depth; a++) { G.put(CT_TRI + a, MISS); G.put(CT_INST + a, MISS); }
        Jo = tan_zero(); Jd = tan_identity(); dpb = f3(0, 0, 0);
      } else {
        Jo = get_tan(G, CT_JO); Jd = get_tan(G, CT_JD); dpb = G.get3(CT_DPB);
      }
      G.put(CT_TRI + b - 1, h.tri);
      G.put(CT_INST + b - 1, h.inst);
    }
    if (h.tri != MISS) {
      const Surf s = surface(S, h, o, d, tt);
      if (TAN) tan_plane_hit(Jo, Jd, d, s.ng, h.t, Jx, dt);
      if (s.flags & VT_F_EMITTER) {
        const float3 nE = emitter_normal(S, h, s, tt);
        const float cosE = dot(-d, nE);
        if (cosE > 0.0f) {
          const float prof = profile(S, acosf(clampf(dot(-d, emitter_axis_at(S, tt)), -1.0f, 1.0f)));
          float w = 1.0f;
          if (b > 1) {
            const float pL = h.t * h.t / (cosE * area);
            w = pb_prev * pb_prev / (pb_prev * pb_prev + fnl * fnl * pL * pL);
          }
          P.put(CP_EMIT_LAMP, __ldg(C.emit_of_tri + h.tri));
          P.putf(CP_EMIT_A, w * prof);
          if (TAN) {
            const float3 de = tan_emitter_hit(S, h, s, d, tt, b, pb_prev, dpb, fnl, area, Jd, Jx, dt);
            G.put3(CT_DE, de);
          }
        }
      } else {
        const uint32_t vk = b == 1 ? 0u : P.get(CP_N);
        P.put(cp_mat(vk), s.mat);
        P.put(CP_N, vk + 1u);
        const float3 nrm = s.ns, wo = -d;
        Tan3 Jn;
        if (TAN) Jn = tan_shading_normal(S, h, s, tt, Jx);
        const float sh0 = b == 1 ? u01(pcg(hs + 3u)) : bounce_shift(hs, b, 0);
        const float sh1 = b == 1 ? u01(pcg(hs + 4u)) : bounce_shift(hs, b, 1);
        const float sh2 = b == 1 ? u01(pcg(hs + 5u)) : bounce_shift(hs, b, 2);
        float4* srec = wb.sh + size_t(p) * nl * 3;
        for (uint32_t j = 0; j < nl; j++) {
          const float3 u = f3(kr(i * nl + j, KL0, sh0), kr(i * nl + j, KL1, sh1), kr(i * nl + j, KL2, sh2));
          float3 lp, ln, la;
          P.put(cp_lamp(vk, j), sample_emitter_idx(S, u, tt, lp, ln, la));
          P.putf(cp_q(vk, j), 0.0f);
          srec[3 * j + 1] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
          float3 wi = lp - s.p;
          const float d2 = dot(wi, wi), dist = sqrtf(d2);
          wi = wi / dist;
          const float cosE = dot(-wi, ln), cosS = dot(nrm, wi);
          if (cosE <= 0.0f || cosS <= 0.0f || dot(s.ng, wi) <= 0.0f || dot(nrm, wo) <= 0.0f) continue;
          const float prof = profile(S, acosf(clampf(dot(-wi, la), -1.0f, 1.0f)));
          if (prof <= 0.0f) continue;
          const float pdfW = d2 / (cosE * area), pb = cosS * INV_PI_F;
          const float w = fnl * fnl * pdfW * pdfW / (fnl * fnl * pdfW * pdfW + pb * pb);
          const float q = prof * cosS * w * INV_PI_F / pdfW;
          if (TAN) G.put3(ct_dq(vk, j), tan_light(S, s.p, nrm, lp, ln, la, area, fnl, q, Jx, Jn));
          // the recorded shadow ray's outcome: an occluded sample stays as calib_shadow_kernel clears it
          if (!((occ >> (vk * CAL_MAX_NL + j)) & 1u)) P.putf(cp_q(vk, j), q);
          if (dmode == 2) continue;
          const float3 so = offset_ray(s.p, s.ng, wi);
          srec[3 * j] = make_float4(so.x, so.y, so.z, dist - 2e-5f);
          srec[3 * j + 1] = make_float4(wi.x, wi.y, wi.z, 1.0f);
          srec[3 * j + 2] = make_float4(0.0f, 0.0f, __uint_as_float(vk), 0.0f);
          shadow = true;
        }
        if (shadow) wb.nee[p] = make_float4(0.0f, 0.0f, 0.0f, tt);
        if (b == cp.max_depth) {
          if (h.inst == MISS && h.tri < C.n_static_tris) P.put(CP_NODE, __ldg(C.tri_node + h.tri));
        } else if (dot(nrm, wo) > 0.0f) {
          const float u1 = b == 1 ? kr(i, KB1, u01(pcg(hs + 7u))) : kr(i, KB1, bounce_shift(hs, b, 4));
          const float u2 = b == 1 ? kr(i, KB2, u01(pcg(hs + 8u))) : kr(i, KB2, bounce_shift(hs, b, 5));
          const float3 t = basis_t(nrm), bb = basis_b(nrm);
          const float r = sqrtf(u1);
          float sp, cpz;
          sincosf(2.0f * PI_F * u2, &sp, &cpz);
          const float3 l = t * (r * cpz) + bb * (r * sp) + nrm * sqrtf(fmaxf(0.0f, 1.0f - u1));
          const float cl = dot(nrm, l);
          if (cl > 0.0f && dot(s.ng, l) > 0.0f) {
            const float3 no = offset_ray(s.p, s.ng, l);
            wb.o[p] = make_float4(no.x, no.y, no.z, tt);
            wb.d[p] = make_float4(l.x, l.y, l.z, cl * INV_PI_F);
            wb.meta[p] = make_uint4(meta.x, meta.y, meta.z, b + 1u);
            cont = true;
            if (TAN) {
              const Tan3 Jl = tan_continue(nrm, Jn, r, cpz, sp, sqrtf(fmaxf(0.0f, 1.0f - u1)));
              G.put3(CT_DPB, (tan_dot(l, Jn) + tan_dot(nrm, Jl)) * INV_PI_F);
              put_tan(G, CT_JO, Jx);
              put_tan(G, CT_JD, Jl);
            }
          }
        }
      }
    }
    const uint32_t qs = warp_append_c(wb.count_out, cont);
    if (cont) wb.q_out[qs] = p;
    const uint32_t ss = warp_append_c(wb.count_sh, shadow);
    if (shadow) wb.q_sh[ss] = p;
  }
}

// any hit of the pending light samples on persistent lanes; an occluded sample's contribution is cleared in the record
__global__ void __launch_bounds__(WT, 4) calib_shadow_kernel(const Scene S, const CamParams cp, WaveBufs wb, uint32_t* rec, size_t r0, uint32_t* dec,
                                                             size_t d0) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");   // the next bounce's closest hits
  const uint32_t n = *wb.count_sh;
  const uint32_t nl = cp.n_light;
  const uint32_t skip = ldu(S.su + 7);
  __shared__ uint2 stack_sh[SH_DEPTH * WT];
  LaneStack stk;
  stk.sh = stack_sh; stk.lane = threadIdx.x; stk.stride = WT;
  TraceState st;
  float3 o = f3(0, 0, 0), d = f3(0, 0, 1);
  float tt = 0.0f;
  uint32_t p = 0, j = 0, state = LANE_IDLE;
  bool exhausted = false;
  const float4* srec = nullptr;
  auto next_sample = [&]() -> bool {
    for (; j < nl; j++) {
      const float4 a = srec[3 * j], w = srec[3 * j + 1];
      if (w.w == 0.0f) continue;
      o = xyz(a); d = xyz(w);
      st.best = Hit{a.w, 0.0f, 0.0f, MISS, MISS};
      if (trace_phase(S, cp.root, o, d, 0.0f, tt, 3u, skip, st, -1)) return true;
    }
    return false;
  };
  auto start = [&](uint32_t idx) {
    p = wb.q_sh[idx];
    tt = wb.nee[p].w;
    srec = wb.sh + size_t(p) * nl * 3;
    j = 0;
    state = next_sample() ? LANE_NODE : LANE_IDLE;
  };
  auto next = [&]() {
    if (st.best.tri == MISS && trace_phase(S, cp.root, o, d, 0.0f, tt, 3u, skip, st, st.k + 1)) { state = LANE_NODE; return; }
    if (st.best.tri != MISS) {
      const uint32_t vk = __float_as_uint(srec[3 * j + 2].z);
      record_at(rec, CP_WORDS, r0 + p).putf(cp_q(vk, j), 0.0f);
      if (dec) {
        const Record D = record_at(dec, CD_WORDS, d0 + p);
        D.put(CD_OCC, D.get(CD_OCC) | 1u << (vk * CAL_MAX_NL + j));
      }
    }
    j++;
    state = next_sample() ? LANE_NODE : LANE_IDLE;
  };
  const uint32_t lanes = lanes_of(n);
  while (serve_lanes(state, exhausted, wb.fetch_sh, n, cp.refill, lanes, next, start)) trace_round<true>(S, 0.0f, st, stk, state);
}

// the derivative in d0 of a recorded path's radiance, per channel, from its derivative record
__device__ __forceinline__ void path_tangent(const CalibDev& C, const ConstRecord& P, const ConstRecord& G, uint32_t nl, float3* dL) {
  const uint32_t n = P.get(CP_N), lamp = P.get(CP_EMIT_LAMP);
  dL[0] = dL[1] = dL[2] = f3(0, 0, 0);
  float3 T = f3(1, 1, 1);
  for (uint32_t k = 0; k < n; k++) {
    T = mul3(T, alb(C, P.get(cp_mat(k))));
    for (uint32_t j = 0; j < nl; j++) {
      if (P.getf(cp_q(k, j)) == 0.0f) continue;
      const float3 dq = G.get3(ct_dq(k, j)) * (__ldg(C.lamp + P.get(cp_lamp(k, j))) / float(nl));
      dL[0] = dL[0] + dq * T.x; dL[1] = dL[1] + dq * T.y; dL[2] = dL[2] + dq * T.z;
    }
  }
  if (lamp != MISS) {
    const float3 de = G.get3(CT_DE) * __ldg(C.lamp + lamp);
    dL[0] = dL[0] + de * T.x; dL[1] = dL[1] + de * T.y; dL[2] = dL[2] + de * T.z;
  }
}

// the derivative of the loss in the camera's intrinsics from one sub-sample: G = g . dL / d d0 (FP64), chained
// through d d0 / d K at the sub-sample's image position
__device__ __forceinline__ void add_intrinsics_grad(const CamParams& cp, uint32_t id, uint32_t i, const float3* dL, double3 g, float* kacc) {
  uint32_t x, y;
  if (!pixel_xy(cp, id, x, y)) return;
  // the term in FP32, its accumulation in FP64
  const float gx = float(g.x), gy = float(g.y), gz = float(g.z);
  const float G[3] = {gx * dL[0].x + gy * dL[1].x + gz * dL[2].x, gx * dL[0].y + gy * dL[1].y + gz * dL[2].y,
                      gx * dL[0].z + gy * dL[1].z + gz * dL[2].z};
  if (G[0] == 0.0f && G[1] == 0.0f && G[2] == 0.0f) return;
  const uint32_t hs = hash3(x, y, cp.seed * 64u + cp.cam_index);
  const float2 uv = subsample_uv(x, y, i, hs);
  float J[3][8];
  kb4_ray_jacobian(cp.lens, uv.x, uv.y, f3(cp.rx[0], cp.rx[1], cp.rx[2]), f3(cp.ry[0], cp.ry[1], cp.ry[2]), f3(cp.rz[0], cp.rz[1], cp.rz[2]), J);
#pragma unroll
  for (int k = 0; k < 8; k++) kacc[k] += G[0] * J[0][k] + G[1] * J[1][k] + G[2] * J[2][k];
}

// Per pixel over the records of sub-samples [i0, i1): backward 0 adds their values to the pixel's running sum (kept in
// the image between chunks; the chunk that ends at spp writes the image and the loss partials), 1 / 2 accumulate the
// gradients (2: with the intrinsics' derivative)
__global__ void __launch_bounds__(CT) calib_records_kernel(const CamParams cp, const CalibDev C, const uint32_t* __restrict__ rec,
                                                          const uint32_t* __restrict__ tan, uint32_t n_pix, int backward, uint32_t i0,
                                                          uint32_t i1) {
  extern __shared__ double sm[];
  double* sh_alb = sm;
  double* sh_lamp = sm + 3 * C.n_mat;
  __shared__ double red[CT / 32];
  __shared__ double sh_k[8];
  if (backward) {
    for (uint32_t k = threadIdx.x; k < 3 * C.n_mat + C.n_lamps; k += blockDim.x) sm[k] = 0.0;
    if (threadIdx.x < 8) sh_k[threadIdx.x] = 0.0;
    __syncthreads();
  }
  double loss = 0.0;
  // the thread's intrinsics terms (one pixel's sub-samples of the launch) summed in FP32 registers, then one FP64 warp
  // sum and 8 shared atomics per warp at the end: all lanes add to the same 8 words, where per-path atomics would
  // contend, and FP64 issues at a small fraction of FP32 on this part
  float kacc[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
  const float sc = cp.scale / float(cp.spp);
  // the block's threads take pixels base + threadIdx.x together, so that a warp's lanes stay together for the
  // per-material warp sums of the backward
  for (uint32_t base = blockIdx.x * blockDim.x; base < n_pix; base += gridDim.x * blockDim.x) {
    const uint32_t id = base + threadIdx.x;
    uint32_t x = 0, y = 0;
    const bool valid = id < n_pix && pixel_xy(cp, id, x, y);
    const size_t px = size_t(y) * cp.w + x;
    if (backward) {
      double3 g = make_double3(0.0, 0.0, 0.0);
      if (valid) {
        const float4 I = C.image[px], Tg = C.target ? C.target[px] : make_float4(0.f, 0.f, 0.f, 0.f);
        const double k = 2.0 * C.inv_count * double(sc);
        g = make_double3(k * (double(I.x) - Tg.x), k * (double(I.y) - Tg.y), k * (double(I.z) - Tg.z));
      }
      const float3 gf = f3(float(g.x), float(g.y), float(g.z));
      for (uint32_t i = i0; i < i1; i++) {
        const size_t r = size_t(i - i0) * n_pix + id;
        AlbGrad ag;
#pragma unroll
        for (uint32_t k = 0; k < CAL_MAX_DEPTH; k++) { ag.on[k] = false; ag.mat[k] = 0u; ag.val[k] = f3(0, 0, 0); }
        if (valid) path_grad(C, record_at(rec, CP_WORDS, r), cp.max_depth, cp.n_light, gf, sh_lamp, ag);
#pragma unroll
        for (uint32_t k = 0; k < CAL_MAX_DEPTH; k++) warp_key_add3(sh_alb, ag.mat[k], ag.val[k], ag.on[k]);
        if (backward == 2 && valid) {
          float3 dL[3];
          path_tangent(C, record_at(rec, CP_WORDS, r), record_at(tan, CT_WORDS, r), cp.n_light, dL);
          add_intrinsics_grad(cp, id, i, dL, g, kacc);
        }
      }
    } else {
      if (!valid) continue;
      // the sum over sub-samples in order, carried across chunks exactly (a float in the image)
      float3 s = f3(0, 0, 0);
      if (i0 > 0) s = xyz(C.image[px]);
      for (uint32_t i = i0; i < i1; i++) s = s + path_value(C, record_at(rec, CP_WORDS, size_t(i - i0) * n_pix + id), cp.max_depth, cp.n_light);
      if (i1 < cp.spp) {
        C.image[px] = make_float4(s.x, s.y, s.z, 0.0f);
        continue;
      }
      const float4 I = make_float4(s.x * sc, s.y * sc, s.z * sc, 1.0f);
      C.image[px] = I;
      if (C.target) {
        const float4 Tg = C.target[px];
        const double dx = double(I.x) - Tg.x, dy = double(I.y) - Tg.y, dz = double(I.z) - Tg.z;
        loss += dx * dx + dy * dy + dz * dz;
      }
    }
  }
  if (backward) {
    if (backward == 2) {
#pragma unroll
      for (int k = 0; k < 8; k++) {
        double v = double(kacc[k]);
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if ((threadIdx.x & 31u) == 0u && v != 0.0) atomicAdd(sh_k + k, v);
      }
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < 3 * C.n_mat; k += blockDim.x) if (sm[k] != 0.0) atomicAdd(C.g_albedo + k, sm[k]);
    for (uint32_t k = threadIdx.x; k < C.n_lamps; k += blockDim.x) if (sh_lamp[k] != 0.0) atomicAdd(C.g_lamp + k, sh_lamp[k]);
    if (backward == 2 && threadIdx.x < 8 && sh_k[threadIdx.x] != 0.0) atomicAdd(C.g_K + threadIdx.x, sh_k[threadIdx.x]);
    return;
  }
  for (int o = 16; o > 0; o >>= 1) loss += __shfl_down_sync(0xffffffffu, loss, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = loss;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < CT / 32; w++) t += red[w];
    C.partials[blockIdx.x] = t * C.inv_count;
  }
}

// one thread per (node, emitter triangle): stratified points (Kronecker in the unit square, the sampler's
// triangle warp), cosines, profile, visibility through the BVH
__global__ void direct_transfer_kernel(const Scene S, const float* __restrict__ C, const float* __restrict__ N, uint32_t n, uint32_t n_lamps,
                                       uint32_t samples, float* __restrict__ D) {
  const size_t total = size_t(n) * n_lamps;
  const uint32_t skip = ldu(S.su + 7);
  for (size_t k = size_t(blockIdx.x) * blockDim.x + threadIdx.x; k < total; k += size_t(gridDim.x) * blockDim.x) {
    const uint32_t i = uint32_t(k / n_lamps), t = uint32_t(k % n_lamps);
    const float3 c = f3(C[3 * i], C[3 * i + 1], C[3 * i + 2]), nn = f3(N[3 * i], N[3 * i + 1], N[3 * i + 2]);
    const float4* e = S.params + S.emit_off + 4u * t;
    const float3 v0 = xyz(__ldg(e)), e1 = xyz(__ldg(e + 1)), e2 = xyz(__ldg(e + 2)), nl0 = xyz(__ldg(e + 3));
    const float At = 0.5f * length(cross(e1, e2));
    Rot R;
    float3 pp;
    inst_pose(S, ldu(S.su + 17), 0.5f, R, pp);
    const float3 nl = rmul(R, nl0), axis = rmul(R, ld3(S.su + 4));
    const float3 org = c + nn * 1e-4f;
    float acc = 0.0f;
    for (uint32_t s = 0; s < samples; s++) {
      const float u1 = kr(s, R2A, 0.5f), u2 = kr(s, R2B, 0.5f);
      const float su = sqrtf(u1);
      const float3 lp = rmul(R, v0 + e1 * (su * (1.0f - u2)) + e2 * (su * u2)) + pp;
      float3 w = lp - org;
      const float r2 = dot(w, w), r = sqrtf(r2);
      w = w / r;
      const float ci = dot(nn, w), ct = dot(nl, -w);
      if (ci <= 0.0f || ct <= 0.0f) continue;
      const float prof = profile(S, acosf(clampf(dot(-w, axis), -1.0f, 1.0f)));
      if (prof <= 0.0f) continue;
      const Hit h = trace_scene<true>(S, 0u, org, w, 0.0f, r - 2e-5f, 0.5f, 3u, skip);
      if (h.tri == MISS) acc += prof * ci * ct / r2;
    }
    D[size_t(i) * n_lamps + t] = acc * At / float(samples);
  }
}

__global__ void dl_kernel(const float* __restrict__ D, const float* __restrict__ L, uint32_t n, uint32_t n_lamps, float* __restrict__ y) {
  const uint32_t row = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
  if (row >= n) return;
  float a = 0.0f;
  for (uint32_t t = lane; t < n_lamps; t += 32) a = fmaf(D[size_t(row) * n_lamps + t], L[t], a);
  for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
  if (lane == 0) y[row] = a;
}

// The calibration's node radiosity and its adjoint at FP64 accuracy without FP64 inner products (FP64 issues at a
// small fraction of FP32 on this part): a vector entry x is held as the float pair (hi, lo) with hi = float(x),
// lo = float(x - hi); each product F_ij x_j is formed exactly for hi by an FMA (its rounding error) plus the lo
// part's product, and the products are summed in a float pair by compensated addition (two-sum, then renormalised).
// Each step is good to about 2^-48 relative; a float32 restatement of 4096-term sums measures at most about 1e-13
// relative against exact sums (FP32 alone: 1e-6). Rows, columns and splits meet in FP64.
__device__ __forceinline__ float2 df_split(double x) {
  const float h = float(x);
  return make_float2(h, float(x - double(h)));
}
// A step of two products at once, the pair's sums apart; every product, difference and sum is rounded on its own (the _rn
// intrinsics are never contracted; x - y is x + (-y) exactly):
//   p = f xh   e = f xl + (f xh - p)   t = sh + p   v = t - sh   lo = sl + (((sh - (t - v)) + (p - v)) + e)
//   sh' = t + lo   sl' = lo - (sh' - t)       (renormalised, so that lo stays below an ulp of the sum)
// f2 and nf2 = -f2; xh, xl the vector's parts.
struct DfAcc { float2 h, l; };
__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ void df_mac2(float2 f, float2 nf, float2 xh, float2 xl, DfAcc& s) {
  const float2 m1 = f2(-1.0f, -1.0f);
  const float2 np = __fmul2_rn(nf, xh);                              // -p
  const float2 e = __ffma2_rn(f, xl, __ffma2_rn(f, xh, np));
  const float2 t = __ffma2_rn(np, m1, s.h);                          // sh + p
  const float2 nv = __ffma2_rn(t, m1, s.h);                          // -(t - sh)
  const float2 a = __ffma2_rn(__fadd2_rn(t, nv), m1, s.h);           // sh - (t - v)
  const float2 b = __ffma2_rn(np, m1, nv);                           // p - v
  const float2 lo = __fadd2_rn(s.l, __fadd2_rn(__fadd2_rn(a, b), e));
  s.h = __fadd2_rn(t, lo);
  s.l = __fadd2_rn(lo, __ffma2_rn(s.h, m1, t));                      // lo - (sh - t)
}
// the sum of two float pairs, renormalised
__device__ __forceinline__ float2 df_add(float2 x, float2 y) {
  const float t = __fadd_rn(x.x, y.x), v = __fsub_rn(t, x.x);
  const float lo = __fadd_rn(__fadd_rn(x.y, y.y), __fadd_rn(__fsub_rn(x.x, __fsub_rn(t, v)), __fsub_rn(y.x, v)));
  const float h = __fadd_rn(t, lo);
  return make_float2(h, __fsub_rn(lo, __fsub_rn(h, t)));
}

// Transposed sweep, the three channels in one pass over F: partial[split][c][part][j] = sum over rows i of the split of F[i][j]
// (g_c,i + rho_c,i lam_c,i), three float parts (Df3), rows of np. A thread takes four columns, two float-pair sums a step (f32x2), so a row of
// F is one 16-byte load for 12 products; the rows' weights lie in shared memory as the pairs the products take. The even and the odd
// rows are chains of their own (one chain for both had 1.3 to 1.8 times the error, n = 512 to 8192), which meet as three parts, like the
// splits. FP64 there, at two operations a cycle and SM, took up to 4 us a sweep: a small calibration step (100 x 100) 3.31 ms with
// 1000 nodes, 4.17 with FP64; 4.31 and 4.92 with 2048; 8.23 and 8.72 with 4096. Bound by the FMA pipe: 14 operations a product, 18 us of
// 37 with 4096 nodes, its combine 5 (a channel and a product at a time, one row in flight: 80 and 25).
constexpr uint32_t JT_SPLITS = 64, JT_THREADS = 256, JT_ROWS = 64;
__host__ __device__ constexpr uint32_t jt_pitch(uint32_t n) { return (n + 3u) / 4u * 4u; }
__global__ void __launch_bounds__(JT_THREADS) jacobi_t_kernel(const float* __restrict__ F, const double* __restrict__ g, const float* __restrict__ rho,
                                                             const double* __restrict__ lam, uint32_t n, float* __restrict__ part) {
  __shared__ float4 w[3][JT_ROWS];   // (hi, hi, lo, lo)
  const uint32_t j = 4u * (blockIdx.x * JT_THREADS + threadIdx.x);
  const uint32_t rows = (n + JT_SPLITS - 1) / JT_SPLITS, i0 = blockIdx.y * rows, i1 = min(n, i0 + rows);
  const bool vec = (n & 3u) == 0u;
  DfAcc s[2][3][2];
#pragma unroll
  for (int q = 0; q < 12; q++) s[q / 6][q / 2 % 3][q % 2].h = s[q / 6][q / 2 % 3][q % 2].l = f2(0.0f, 0.0f);
  for (uint32_t ib = i0; ib < i1; ib += JT_ROWS) {
    const uint32_t m = min(JT_ROWS, i1 - ib);
    __syncthreads();
    for (uint32_t q = threadIdx.x; q < 3u * m; q += JT_THREADS) {
      const uint32_t c = q / m, k = q % m;
      const size_t i = size_t(c) * n + ib + k;
      const float2 x = df_split(g[i] + double(rho[i]) * lam[i]);
      w[c][k] = make_float4(x.x, x.x, x.y, x.y);
    }
    __syncthreads();
    if (j < n) {
      const float* Fc = F + size_t(ib) * n + j;
      auto load = [&](const float* p) {
        if (vec) return __ldg(reinterpret_cast<const float4*>(p));
        return make_float4(p[0], j + 1 < n ? p[1] : 0.0f, j + 2 < n ? p[2] : 0.0f, j + 3 < n ? p[3] : 0.0f);
      };
      auto row = [&](float4 f, uint32_t k, DfAcc (&a)[3][2]) {
#pragma unroll
        for (int c = 0; c < 3; c++) {
          const float4 x = w[c][k];
          df_mac2(f2(f.x, f.y), f2(-f.x, -f.y), f2(x.x, x.y), f2(x.z, x.w), a[c][0]);
          df_mac2(f2(f.z, f.w), f2(-f.z, -f.w), f2(x.x, x.y), f2(x.z, x.w), a[c][1]);
        }
      };
      uint32_t k = 0;
      for (; k + 4u <= m; k += 4u, Fc += size_t(4) * n) {   // four rows in flight
        float4 f[4];
#pragma unroll
        for (int q = 0; q < 4; q++) f[q] = load(Fc + size_t(q) * n);
#pragma unroll
        for (int q = 0; q < 4; q++) row(f[q], k + q, s[q & 1]);
      }
      if (k < m) row(load(Fc), k, s[0]);
      if (k + 1u < m) row(load(Fc + n), k + 1u, s[1]);
      if (k + 2u < m) row(load(Fc + size_t(2) * n), k + 2u, s[0]);
    }
  }
  if (j >= n) return;
  const size_t np = jt_pitch(n);
#pragma unroll
  for (int c = 0; c < 3; c++) {
    Df3 v[4];
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const DfAcc &a = s[0][c][q], &b = s[1][c][q];
      v[2 * q] = df_add(Df3{a.h.x, a.l.x, 0.0f}, Df3{b.h.x, b.l.x, 0.0f});
      v[2 * q + 1] = df_add(Df3{a.h.y, a.l.y, 0.0f}, Df3{b.h.y, b.l.y, 0.0f});
    }
    float* p = part + (size_t(blockIdx.y) * 3 + c) * 3 * np + j;
    *reinterpret_cast<float4*>(p) = make_float4(v[0].h, v[1].h, v[2].h, v[3].h);
    *reinterpret_cast<float4*>(p + np) = make_float4(v[0].m, v[1].m, v[2].m, v[3].m);
    *reinterpret_cast<float4*>(p + 2 * np) = make_float4(v[0].l, v[1].l, v[2].l, v[3].l);
  }
}
// out = the sum of the partials, 3 n values: a block takes 32 of them, each warp an eighth of the splits, the warps' sums in
// order
__global__ void __launch_bounds__(256) jacobi_t_combine(const float* __restrict__ part, uint32_t n, double* __restrict__ out) {
  __shared__ Df3 red[8][32];
  const uint32_t np = jt_pitch(n), lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, j = blockIdx.x * 32u + lane, c = j / np, k = j % np;
  Df3 a{0.0f, 0.0f, 0.0f};
  if (c < 3u) {
    const float* p = part + (size_t(warp * (JT_SPLITS / 8)) * 3 + c) * 3 * np + k;
    Df3 x[JT_SPLITS / 8];
#pragma unroll
    for (uint32_t s = 0; s < JT_SPLITS / 8; s++, p += size_t(9) * np) x[s] = {p[0], p[np], p[2 * size_t(np)]};
#pragma unroll
    for (uint32_t s = 0; s < JT_SPLITS / 8; s++) a = df_add(a, x[s]);
  }
  red[warp][lane] = a;
  __syncthreads();
  if (warp || c >= 3u || k >= n) return;
  for (uint32_t w = 1; w < 8; w++) a = df_add(a, red[w][lane]);
  out[size_t(c) * n + k] = df_double(a);
}

// The three channels' B_c,out = rho_c o (DL + F B_c,in) at FP64 accuracy (F in FP32, B as float pairs, planar [c][hi | lo]
// [np]), the products summed in float pairs; with `H` set, H_c = F B_c,in (rounded to FP32) instead. A block takes
// R64_ROWS rows, a thread four columns at a time of each: a load of B serves the rows, and a step is two products (f32x2) in
// 12 independent sums. Bound by the FMA pipe (14 operations a product, 18 us at its rate). N = 4096: 37 us a sweep; a warp per
// row with one product a step and B read again for each row took 51 us.
// A row's sums over the lanes are float pairs where its length allows it: with chains of n / 512 products
// their error against exact sums stays below that of a warp per row, 32 chains of n / 32 that meet in FP64 (positive terms, rms: n =
// 769 6.1e-16, there 6.3e-16; 1025 4.8e-16 and 6.8e-16; 4096 4.6e-16 and 1.3e-15). A shorter row's error would be the tree's (n = 512 6.7e-16, there
// 5.4e-16; 31 1.5e-15 and 3.0e-16), so there (SHORT) every product is a sum of its own and the tree takes Df3 (9.9e-17, and 3.0e-16).
constexpr uint32_t R64_ROWS = 4, R64_THREADS = 256;
constexpr uint32_t R64_SHORT = 768;   // nodes, at most four a thread
__device__ __forceinline__ float2 df_shfl(float2 v, uint32_t mask) {
  return make_float2(__shfl_xor_sync(0xffffffffu, v.x, mask), __shfl_xor_sync(0xffffffffu, v.y, mask));
}
__device__ __forceinline__ Df3 df_shfl(Df3 v, uint32_t mask) {
  return {__shfl_xor_sync(0xffffffffu, v.h, mask), __shfl_xor_sync(0xffffffffu, v.m, mask), __shfl_xor_sync(0xffffffffu, v.l, mask)};
}
__device__ __forceinline__ double df_double(float2 v) { return double(v.x) + double(v.y); }
// the sums over a warp's lanes of 16 values a lane: lane 2 v ends with value v. A step halves the values that a lane still adds
template <typename V>
__device__ __forceinline__ V df_warp_sum16(V* v, uint32_t lane) {
#pragma unroll
  for (uint32_t half = 8; half > 0; half >>= 1) {
    const bool up = (lane & (2u * half)) != 0u;
#pragma unroll
    for (uint32_t q = 0; q < half; q++) {
      const V mine = up ? v[q + half] : v[q], other = up ? v[q] : v[q + half];
      v[q] = df_add(mine, df_shfl(other, 2 * half));
    }
  }
  return df_add(v[0], df_shfl(v[0], 1));
}
template <bool SHORT>
__global__ void __launch_bounds__(R64_THREADS, SHORT ? 1 : 2) radiosity64_kernel(const float* __restrict__ F, const float* __restrict__ rho,
                                                                               const float* __restrict__ DL, const float* __restrict__ Bin,
                                                                               float* __restrict__ Bout, float* __restrict__ H, uint32_t n, uint32_t np) {
  constexpr int SUMS = SHORT ? 2 : 1;
  __shared__ double red[R64_THREADS / 32][R64_ROWS * 3];
  const uint32_t row0 = blockIdx.x * R64_ROWS, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const bool vec = (n & 3u) == 0u;
  DfAcc s[R64_ROWS][3][SUMS];
#pragma unroll
  for (uint32_t r = 0; r < R64_ROWS; r++)
#pragma unroll
    for (int c = 0; c < 3; c++) {
      s[r][c][0].h = s[r][c][0].l = f2(0.0f, 0.0f);
      s[r][c][SUMS - 1] = s[r][c][0];
    }
  for (uint32_t j = 4u * threadIdx.x; j < n; j += 4u * R64_THREADS) {
    float4 f[R64_ROWS];
#pragma unroll
    for (uint32_t r = 0; r < R64_ROWS; r++) {
      const float* p = F + size_t(min(row0 + r, n - 1u)) * n + j;
      if (vec) f[r] = __ldg(reinterpret_cast<const float4*>(p));
      else f[r] = make_float4(p[0], j + 1 < n ? p[1] : 0.0f, j + 2 < n ? p[2] : 0.0f, j + 3 < n ? p[3] : 0.0f);
    }
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const float4 xh = __ldg(reinterpret_cast<const float4*>(Bin + size_t(2 * c) * np + j));
      const float4 xl = __ldg(reinterpret_cast<const float4*>(Bin + size_t(2 * c + 1) * np + j));
#pragma unroll
      for (uint32_t r = 0; r < R64_ROWS; r++) {
        df_mac2(f2(f[r].x, f[r].y), f2(-f[r].x, -f[r].y), f2(xh.x, xh.y), f2(xl.x, xl.y), s[r][c][0]);
        df_mac2(f2(f[r].z, f[r].w), f2(-f[r].z, -f[r].w), f2(xh.z, xh.w), f2(xl.z, xl.w), s[r][c][SUMS - 1]);
      }
    }
    if (SHORT) break;   // n is R64_SHORT at most
  }
  // the block's sums over a warp's lanes, then over the warps in FP64
  static_assert(R64_ROWS * 3 <= 16, "values of a lane");
  double sum = 0.0;
  if (SHORT) {
    if (128u * warp < n) {
      Df3 v[16];
#pragma unroll
      for (uint32_t q = 0; q < 16; q++) {
        v[q] = {0.0f, 0.0f, 0.0f};
        if (q >= R64_ROWS * 3) continue;
        const DfAcc &a = s[q / 3][q % 3][0], &b = s[q / 3][q % 3][SUMS - 1];
        v[q] = df_add(df_add(Df3{a.h.x, a.l.x, 0.0f}, Df3{a.h.y, a.l.y, 0.0f}), df_add(Df3{b.h.x, b.l.x, 0.0f}, Df3{b.h.y, b.l.y, 0.0f}));
      }
      sum = df_double(df_warp_sum16(v, lane));
    }
  } else {
    float2 v[16];
#pragma unroll
    for (uint32_t q = 0; q < 16; q++) {
      v[q] = make_float2(0.0f, 0.0f);
      if (q >= R64_ROWS * 3) continue;
      const DfAcc& a = s[q / 3][q % 3][0];
      v[q] = df_add(make_float2(a.h.x, a.l.x), make_float2(a.h.y, a.l.y));
    }
    sum = df_double(df_warp_sum16(v, lane));
  }
  if (!(lane & 1u) && lane / 2u < R64_ROWS * 3) red[warp][lane / 2u] = sum;
  __syncthreads();
  const uint32_t q = threadIdx.x, row = row0 + q / 3u, c = q % 3u;
  if (q >= 3u * R64_ROWS || row >= n) return;
  double a = 0.0;
  for (uint32_t w = 0; w < R64_THREADS / 32; w++) a += red[w][q];
  if (H) { H[size_t(c) * n + row] = float(a); return; }
  const float2 x = df_split(double(rho[size_t(c) * n + row]) * (double(DL[row]) + a));
  Bout[size_t(2 * c) * np + row] = x.x;
  Bout[size_t(2 * c + 1) * np + row] = x.y;
}
// the first iterate, and zeros in both arrays' tails
__global__ void radiosity64_init(const float* __restrict__ rho, const float* __restrict__ DL, float* __restrict__ B, float* __restrict__ other, uint32_t n,
                                 uint32_t np) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 3 * np) return;
  const uint32_t c = i / np, k = i % np;
  const float2 x = k < n ? df_split(double(rho[size_t(c) * n + k]) * double(DL[k])) : make_float2(0.0f, 0.0f);
  B[size_t(2 * c) * np + k] = x.x;
  B[size_t(2 * c + 1) * np + k] = x.y;
  if (k >= n) other[size_t(2 * c) * np + k] = other[size_t(2 * c + 1) * np + k] = 0.0f;
}

__global__ void mul_kernel(const float* __restrict__ a, const float* __restrict__ b, float* __restrict__ y, uint32_t n) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = a[i] * b[i];
}

__global__ void sum_kernel(const double* __restrict__ p, uint32_t n, double* __restrict__ out) {
  __shared__ double s[1024];
  double a = 0.0;
  for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) a += p[i];
  s[threadIdx.x] = a;
  __syncthreads();
  for (uint32_t o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) s[threadIdx.x] += s[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = s[0];
}
// calib_shade_kernel's grid-stride loop runs as one wave of its own occupancy (3 blocks of 256 per SM at 80
// registers) rather than on the traversal kernels' grid, a wave and a third of it (C4 forward 200 -> 196 ms)
template <bool TAN>
int calib_shade_grid() {
  static std::atomic<int> grid[MAX_DEVICES];
  return per_device_value(grid, [](int dev) {
    int per = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, calib_shade_kernel<TAN>, WT, 0);
    return device_sms(dev) * std::max(1, per);
  });
}
}  // namespace

size_t calib_record_bytes(uint32_t paths) { return size_t(paths) * CP_WORDS * 4; }

size_t calib_tan_bytes(uint32_t paths) { return size_t(paths) * CT_WORDS * 4; }

// tri_hit's arithmetic without its range checks: for a hit tri_hit accepted, the same t, u, v; a recorded hit is met
// again even when the ray moved by rounding (the derivative-record kernel's ray can differ from the plain kernel's
// in its last bits)
__device__ __forceinline__ void tri_uvt(const Scene& S, uint32_t k, float3 o, float3 d, float& t, float& u, float& v) {
  const float4* r = S.tris + 4u * k;
  const float3 v0 = xyz(__ldg(r)), e1 = xyz(__ldg(r + 1)), e2 = xyz(__ldg(r + 2));
  const float3 p = cross(d, e2);
  const float det = dot(e1, p);
  const float inv = 1.0f / det;
  const float3 s = o - v0;
  u = dot(s, p) * inv;
  const float3 q = cross(s, e1);
  v = dot(d, q) * inv;
  t = dot(e2, q) * inv;
}

// the extension rays of a replayed bounce meet the triangles the traced bounce recorded: the traversal's frame (the
// world, or the instance's pose at the path's time) and its triangle arithmetic, so t, u, v are the traced hit's
__global__ void __launch_bounds__(256) calib_rehit_kernel(const Scene S, WaveBufs wb, const uint32_t* __restrict__ dec, size_t d0, uint32_t b) {
  const uint32_t n = *wb.count_in;
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    const uint32_t p = wb.q_in[k];
    const ConstRecord D = record_at(dec, CD_WORDS, d0 + p);
    const uint32_t tri = D.get(CD_TRI + b - 1), inst = (D.get(CD_INST) >> (8u * (b - 1u))) & 0xffu;
    float4 hit = make_float4(BIG, 0.0f, 0.0f, __uint_as_float(MISS));
    uint32_t hinst = MISS;
    if (tri != MISS) {
      const float4 o4 = wb.o[p], d4 = wb.d[p];
      float3 o = xyz(o4), d = xyz(d4);
      if (inst != 0xffu) {
        Rot R;
        float3 pp;
        inst_pose(S, inst, o4.w, R, pp);
        o = rtmul(R, o - pp);
        d = rtmul(R, d);
        hinst = inst;
      }
      float t, u, v;
      tri_uvt(S, tri, o, d, t, u, v);
      hit = make_float4(t, u, v, __uint_as_float(tri));
    }
    wb.hit[p] = hit;
    wb.hinst[p] = hinst;
  }
}

// the paths of sub-samples [i0, i1) of the camera through the wavefront, their records (i - i0) n_pix + id
static void calib_trace(const Scene& S, const CamParams& cp, const CalibDev& C, WaveBufs wb, uint32_t wave_paths, uint32_t* rec, uint32_t* tan,
                        uint32_t i0, uint32_t i1, int blocks, cudaStream_t st, uint32_t* dec, int dmode) {
  const uint32_t n_pix = tiled_pixels(cp.w, cp.h, cp.tile_w, cp.tile_h);
  const uint32_t per_wave = std::max(1u, std::min(i1 - i0, wave_paths / std::max(1u, n_pix)));
  for (uint32_t w0 = i0; w0 < i1; w0 += per_wave) {
    const uint32_t n_i = std::min(per_wave, i1 - w0);
    cudaMemsetAsync(wb.counts, 0, 16, st);
    launch_wave_gen(cp, wb, w0, n_i, n_pix, blocks, st);
    const size_t r0 = size_t(w0 - i0) * n_pix, d0 = size_t(w0) * n_pix;
    const int dm = dec ? dmode : 0;
    uint32_t* db = dm ? dec : nullptr;
    for (uint32_t b = 1; b <= cp.max_depth; b++) {
      WaveBufs w = wb;
      bounce_view(w, b);
      if (dm == 2) {
        cudaMemsetAsync(w.count_out, 0, 16, st);
        calib_rehit_kernel<<<std::max(1, blocks), 256, 0, st>>>(S, w, db, d0, b);
      } else {
        launch_wave_extend(S, cp, w, blocks, st, b > 1);   // over the light samples' tail
      }
      if (tan) calib_shade_kernel<true><<<calib_shade_grid<true>(), WT, 0, st>>>(S, cp, C, w, rec, tan, r0, b, db, d0, dm);
      else calib_shade_kernel<false><<<calib_shade_grid<false>(), WT, 0, st>>>(S, cp, C, w, rec, nullptr, r0, b, db, d0, dm);
      if (dm == 2) continue;   // the recorded shadow outcomes were applied by the shading
      calib_shadow_kernel<<<blocks, WT, 0, st>>>(S, cp, w, rec, r0, db, d0);
    }
  }
}

uint32_t calib_wave_forward(const Scene& S, const CamParams& cp, const CalibDev& C, WaveBufs wb, uint32_t wave_paths, void* records, void* tangents,
                            int blocks, cudaStream_t st) {
  return calib_wave_chunk(S, cp, C, wb, wave_paths, records, tangents, 0, cp.spp, 0, blocks, st);
}

size_t calib_dec_bytes(uint32_t paths) { return size_t(paths) * CD_WORDS * 4; }

uint32_t calib_wave_chunk(const Scene& S, const CamParams& cp, const CalibDev& C, WaveBufs wb, uint32_t wave_paths, void* records, void* tangents,
                          uint32_t i0, uint32_t i1, int mode, int blocks, cudaStream_t st, void* decisions, int dec_mode) {
  uint32_t *rec = static_cast<uint32_t*>(records), *tan = static_cast<uint32_t*>(tangents);
  calib_trace(S, cp, C, wb, wave_paths, rec, tan, i0, i1, blocks, st, static_cast<uint32_t*>(decisions), dec_mode);
  const uint32_t n_pix = tiled_pixels(cp.w, cp.h, cp.tile_w, cp.tile_h);
  const uint32_t grid = std::max(1u, std::min(uint32_t(blocks), (n_pix + CT - 1) / CT));
  const size_t smem = mode ? size_t(3 * C.n_mat + C.n_lamps) * 8 : 0;
  calib_records_kernel<<<grid, CT, smem, st>>>(cp, C, rec, tan, n_pix, mode, i0, i1);
  return grid;
}

void calib_records_backward(const CamParams& cp, const CalibDev& C, const void* records, const void* tangents, int blocks, cudaStream_t st) {
  const uint32_t n_pix = tiled_pixels(cp.w, cp.h, cp.tile_w, cp.tile_h);
  const uint32_t grid = std::max(1u, std::min(uint32_t(blocks), (n_pix + CT - 1) / CT));
  calib_records_kernel<<<grid, CT, size_t(3 * C.n_mat + C.n_lamps) * 8, st>>>(cp, C, static_cast<const uint32_t*>(records),
                                                                             static_cast<const uint32_t*>(tangents), n_pix, tangents ? 2 : 1,
                                                                             0, cp.spp);
}

// per path of the camera's records, in (row, column, sub-sample) order: the triangle and instance of each bounce
// (~0: none) and each vertex's light samples' q (0: occluded or no contribution)
__global__ void calib_export_paths_kernel(const CamParams cp, const uint32_t* __restrict__ rec, const uint32_t* __restrict__ tan, uint32_t n_pix,
                                          uint32_t* __restrict__ tri_inst, float* __restrict__ q) {
  const uint32_t id = blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t x, y;
  if (id >= n_pix || !pixel_xy(cp, id, x, y)) return;
  for (uint32_t i = 0; i < cp.spp; i++) {
    const size_t r = size_t(i) * n_pix + id, o = (size_t(y) * cp.w + x) * cp.spp + i;
    const ConstRecord P = record_at(rec, CP_WORDS, r), G = record_at(tan, CT_WORDS, r);
    const uint32_t n = P.get(CP_N);
    for (uint32_t b = 0; b < CAL_MAX_DEPTH; b++) {
      tri_inst[(o * CAL_MAX_DEPTH + b) * 2] = b < cp.max_depth ? G.get(CT_TRI + b) : MISS;
      tri_inst[(o * CAL_MAX_DEPTH + b) * 2 + 1] = b < cp.max_depth ? G.get(CT_INST + b) : MISS;
      for (uint32_t j = 0; j < CAL_MAX_NL; j++) q[(o * CAL_MAX_DEPTH + b) * CAL_MAX_NL + j] = b < n && j < cp.n_light ? P.getf(cp_q(b, j)) : 0.0f;
    }
  }
}

void calib_export_paths(const CamParams& cp, const void* records, const void* tangents, uint32_t* tri_inst, float* q, cudaStream_t st) {
  const uint32_t n_pix = tiled_pixels(cp.w, cp.h, cp.tile_w, cp.tile_h);
  calib_export_paths_kernel<<<(n_pix + 127) / 128, 128, 0, st>>>(cp, static_cast<const uint32_t*>(records), static_cast<const uint32_t*>(tangents),
                                                                n_pix, tri_inst, q);
}

void launch_direct_transfer(const Scene& S, const float* centres, const float* normals, uint32_t n, uint32_t n_lamps, uint32_t samples, float* D,
                            cudaStream_t st) {
  const size_t total = size_t(n) * n_lamps;
  const uint32_t grid = uint32_t(std::min<size_t>((total + 127) / 128, 65535));
  direct_transfer_kernel<<<grid, 128, 0, st>>>(S, centres, normals, n, n_lamps, samples, D);
}

void launch_dl(const float* D, const float* L, uint32_t n, uint32_t n_lamps, float* y, cudaStream_t st) {
  dl_kernel<<<(n + 7) / 8, 256, 0, st>>>(D, L, n, n_lamps, y);
}

size_t jacobi_t_work(uint32_t n) { return size_t(JT_SPLITS) * 9 * jt_pitch(n) * 4; }

void launch_jacobi_t(const float* F, const double* g, const float* rho, const double* lam_in, double* lam_out, uint32_t n, double* work,
                     cudaStream_t st) {
  float* part = reinterpret_cast<float*>(work);   // the arena's places are 256-byte aligned
  jacobi_t_kernel<<<dim3((n + 4 * JT_THREADS - 1) / (4 * JT_THREADS), JT_SPLITS), JT_THREADS, 0, st>>>(F, g, rho, lam_in, n, part);
  jacobi_t_combine<<<(3 * jt_pitch(n) + 31) / 32, 256, 0, st>>>(part, n, lam_out);
}

void launch_sum(const double* p, uint32_t n, double* out, cudaStream_t st) { sum_kernel<<<1, 1024, 0, st>>>(p, n, out); }

void launch_mul(const float* a, const float* b, float* y, uint32_t n, cudaStream_t st) { mul_kernel<<<(n + 255) / 256, 256, 0, st>>>(a, b, y, n); }

void launch_radiosity64(const float* F, const float* rho, const float* DL, uint32_t n, uint32_t iters, void* work, float* H,
                        cudaStream_t st) {
  // the three channels' iterates as float pairs, two planar arrays in `work`, rows of a multiple of 4
  const uint32_t np = (n + 3u) / 4u * 4u;
  float* cur = static_cast<float*>(work);
  float* nxt = cur + size_t(6) * np;
  const uint32_t blocks = (n + R64_ROWS - 1) / R64_ROWS;
  radiosity64_init<<<(3 * np + 255) / 256, 256, 0, st>>>(rho, DL, cur, nxt, n, np);
  const auto kernel = n <= R64_SHORT ? radiosity64_kernel<true> : radiosity64_kernel<false>;
  for (uint32_t it = 0; it < iters; it++) {
    kernel<<<blocks, R64_THREADS, 0, st>>>(F, rho, DL, cur, nxt, nullptr, n, np);
    std::swap(cur, nxt);
  }
  kernel<<<blocks, R64_THREADS, 0, st>>>(F, rho, DL, cur, nullptr, H, n, np);
}

}  // namespace vtk
