// Path queues filled by whole warps.
#pragma once

#include <cstdint>

namespace vtk {

// A path with a next ray, with light samples or both to the next bounce's queue and the bounce's shadow queue (WaveBufs, whose
// counts of the two are neighbours): one atomic a warp for both. A warp waits for its answer at the end of each 32 paths, and the
// counter's line takes one in ~1.3 ns (one for each queue, 640x480, 16 spp: 14.42 ms, pose batch
// 83.9; now 14.32, 83.0)
template <typename Bufs>
__device__ __forceinline__ void append_path(const Bufs& wb, uint32_t p, bool cont, bool shadow) {
  const uint32_t act = __activemask(), lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
  const uint32_t mc = __ballot_sync(act, cont), ms = __ballot_sync(act, shadow);
  if (!(mc | ms)) return;
  const uint32_t leader = __ffs(act) - 1;
  unsigned long long base = 0;
  if (lane == leader) base = atomicAdd(reinterpret_cast<unsigned long long*>(wb.count_out), (unsigned long long)__popc(ms) << 32 | uint32_t(__popc(mc)));
  const uint32_t b0 = __shfl_sync(act, uint32_t(base), leader), b1 = __shfl_sync(act, uint32_t(base >> 32), leader);
  if (cont) wb.q_out[b0 + __popc(mc & below)] = p;
  if (shadow) wb.q_sh[b1 + __popc(ms & below)] = p;
}

// A warp's entries for a queue, kept in shared memory and appended by one atomic when they are many (or at the end): for the
// short kernels, which with an atomic a warp for each 32 paths were bound by the counter's line, ~1.3 ns each (camera rays
// of 4.3 M paths 176 us, now 97; bytes 50). In the shading the queue's state costs more registers than the atomics time
// (640x480, 16 spp: 2.8 -> 4.5 ms).
constexpr uint32_t WQ_CAP = 128;
struct WarpQueue {
  uint32_t* buf;       // WQ_CAP words of the warp's own
  uint32_t fill = 0;   // the same in all lanes
  __device__ __forceinline__ explicit WarpQueue(uint32_t* b) : buf(b) {}
  // all 32 lanes together
  __device__ __forceinline__ void push(bool want, uint32_t v, uint32_t* count, uint32_t* q) {
    const uint32_t lane = threadIdx.x & 31u, mask = __ballot_sync(0xffffffffu, want);
    if (want) buf[fill + __popc(mask & ((1u << lane) - 1u))] = v;
    fill += __popc(mask);
    __syncwarp();
    if (fill > WQ_CAP - 32u) flush(count, q);
  }
  __device__ __forceinline__ void flush(uint32_t* count, uint32_t* q) {
    if (!fill) return;
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(count, fill);
    base = __shfl_sync(0xffffffffu, base, 0);
    for (uint32_t i = lane; i < fill; i += 32u) q[base + i] = buf[i];
    fill = 0;
    __syncwarp();
  }
};

// A warp's share of n items: the runs of 32 from `first`, `runs` of them side by side (so that what the warp appends at once
// lay side by side too) where there is more than a run for each warp, then `stride` on
struct WarpShare {
  uint32_t first, runs, stride;
  __device__ __forceinline__ explicit WarpShare(uint32_t n) {
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    runs = min(max(n / (warps * 32u), 1u), WQ_CAP / 32u) * 32u;
    first = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * runs;
    stride = warps * runs;
  }
};

}  // namespace vtk
