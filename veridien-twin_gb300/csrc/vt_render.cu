// Ray queries on sm_103a: traceTest (gpu/wgsl/kernels.wgsl.js:535) and visible (gpu/renderer.js:1238). Camera
// rendering is the wavefront path tracer in vt_wave.cu.
#include <algorithm>

#include "vt_kernels.cuh"

namespace vtk {
using namespace vtd;

// Traversal layout of a node (64 B): per axis the planes (child 0 lo, child 1 lo, child 0 hi, child 1 hi), then the
// children's words (child 0 ref, count, child 1 ref, count), so that a load leaves the two children's planes as the
// register pairs of slab_pair's f32x2 operations. gpu/bvh.js numbers a child above its parent; an interior child that is not gets
// the count BAD_CHILD, and a leaf beside it comes first (traverse tests a node's leaves before it descends)
__global__ void pack_nodes_kernel(float4* __restrict__ nodes, uint32_t n) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float4* nb = nodes + size_t(4) * i;
  float4 a0 = nb[0], a1 = nb[1], a2 = nb[2], a3 = nb[3];   // c0.lo|ref, c0.hi|count, c1.lo|ref, c1.hi|count
  const bool bad0 = fu(a1.w) == 0u && fu(a0.w) <= i, bad1 = fu(a3.w) == 0u && fu(a2.w) <= i;
  if (bad0) a1.w = __uint_as_float(BAD_CHILD);
  if (bad1) a3.w = __uint_as_float(BAD_CHILD);
  if (bad0 && !bad1 && fu(a3.w) != 0u) {
    const float4 lo = a0, hi = a1;
    a0 = a2; a1 = a3; a2 = lo; a3 = hi;
  }
  nb[0] = make_float4(a0.x, a2.x, a1.x, a3.x);
  nb[1] = make_float4(a0.y, a2.y, a1.y, a3.y);
  nb[2] = make_float4(a0.z, a2.z, a1.z, a3.z);
  nb[3] = make_float4(a0.w, a1.w, a2.w, a3.w);
}
void pack_nodes(float4* nodes, uint32_t n, cudaStream_t st) {
  if (n) pack_nodes_kernel<<<(n + 255) / 256, 256, 0, st>>>(nodes, n);
}

// gpu/wgsl/kernels.wgsl.js:535 traceTest: one ray per thread
__global__ void trace_kernel(const Scene S, const float4* __restrict__ o4, const float4* __restrict__ d4, uint32_t n, uint32_t mask,
                             uint32_t any_hit, uint32_t root, float4* __restrict__ out4, float* __restrict__ out_v) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float4 o = o4[i], d = d4[i];
  const Hit h = any_hit ? trace_scene<true>(S, root, xyz(o), xyz(d), 0.0f, BIG, o.w, mask, 0u)
                        : trace_scene<false>(S, root, xyz(o), xyz(d), 0.0f, BIG, o.w, mask, 0u);
  out4[i] = make_float4(h.t, __uint_as_float(h.tri), __uint_as_float(h.inst), h.u);
  if (out_v) out_v[i] = h.v;
}

void launch_trace(const Scene& S, const float4* o4, const float4* d4, uint32_t n, uint32_t mask, uint32_t any_hit, uint32_t root,
                  float4* out4, float* out_v, cudaStream_t st) {
  if (!n) return;
  trace_kernel<<<(n + 127) / 128, 128, 0, st>>>(S, o4, d4, n, mask, any_hit, root, out4, out_v);
}

// gpu/renderer.js:1238 visible: occlusion between the camera centre and each point (static BVH from its full root,
// then every posed body at `time`, the camera's own bodies skipped)
__global__ void visible_kernel(const Scene S, float3 c, const float3* __restrict__ pts, uint32_t n, float tol, float time, uint32_t skip,
                               uint8_t* __restrict__ out) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float3 v = pts[i] - c;
  const float dist = length(v);
  if (!(dist > tol)) { out[i] = 1; return; }
  const float3 d = v / dist;
  const Hit h = trace_scene<true>(S, 0u, c, d, 0.0f, dist - tol, time, 3u, skip);
  out[i] = h.tri == MISS ? 1 : 0;
}

void launch_visible(const Scene& S, float3 c, const float3* pts, uint32_t n, float tol, float time, uint32_t skip, uint8_t* out,
                    cudaStream_t st) {
  if (!n) return;
  visible_kernel<<<(n + 127) / 128, 128, 0, st>>>(S, c, pts, n, tol, time, skip, out);
}

}  // namespace vtk
