// Multi-right-hand-side node radiosity sweeps on the 5th-generation tensor cores (tcgen05) of sm_103a.
//
// tc_gemm_kernel: one CTA per SM takes a run of the (128 rows, 128 bytes of K) tiles of F. One warp feeds a ring of
// shared-memory stages with TMA (cp.async.bulk.tensor, 128-byte swizzle; a stage is 128 rows x 128 B of F and 64 rows x 128 B
// of the transposed right-hand sides Bt), one issues tcgen05.mma (M = 128, N = 64, K = 16 bf16 / 32 e4m3 per instruction)
// into two accumulators in tensor memory (TMEM) in turn and releases each stage with tcgen05.commit, and four read the
// accumulators back with tcgen05.ld and sum them in registers, into a partial per row tile that the run meets. The
// combine kernels (CUDA cores, HBM-bound and small) apply the Jacobi epilogue or the accurate residual in FP64.
//
// The sweep streams F once: 2 B per element in BF16, 1 B in FP8, so it is HBM-bound (64 flop/B at 64 right-hand
// sides in BF16, 128 in FP8, both under the tensor ridge). Every wait on an mbarrier is bounded by a clock limit:
// a wait that runs out sets *err and the kernel drains its TMA copies, frees its TMEM and returns.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp8.h>

#include <algorithm>
#include <cstring>
#include <mutex>

#include "vt_async.cuh"
#include "vt_kernels.cuh"
#include "vt_tc.cuh"

namespace vtk {

namespace {

constexpr uint32_t A_BYTES = 128 * 128;   // 128 rows x 128 B
constexpr uint32_t B_BYTES = 64 * 128;    // 64 rows x 128 B
using namespace async;

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const TcMap* map, int32_t c0, int32_t c1, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
               "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// shared-memory matrix descriptor: K-major, 128-byte swizzle, 8-row atoms 1024 B apart
__device__ __forceinline__ uint64_t sw128_desc(uint32_t saddr) {
  uint64_t d = uint64_t((saddr & 0x3FFFFu) >> 4);
  d |= uint64_t(1) << 16;                 // leading byte offset (unused for swizzled K-major)
  d |= uint64_t(1024 >> 4) << 32;         // stride byte offset: one 8-row atom
  d |= uint64_t(1) << 46;                 // descriptor version
  d |= uint64_t(2) << 61;                 // 128-byte swizzle
  return d;
}
// instruction descriptor: D f32, A/B type, K-major A and B, N = 64, M = 128
__host__ __device__ constexpr uint32_t idesc_of(uint32_t ab_type) {
  return (1u << 4) | (ab_type << 7) | (ab_type << 10) | ((64u >> 3) << 17) | ((128u >> 4) << 24);
}
constexpr uint32_t IDESC_BF16 = idesc_of(1);   // kind::f16, bf16 x bf16
constexpr uint32_t IDESC_E4M3 = idesc_of(0);   // kind::f8f6f4, e4m3 x e4m3

template <int MODE>
__device__ __forceinline__ void mma(uint32_t tmem, uint64_t a, uint64_t b, uint32_t accumulate) {
  if (MODE == TC_FP8) {
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n}" ::"r"(tmem),
                 "l"(a), "l"(b), "r"(IDESC_E4M3), "r"(accumulate)
                 : "memory");
  } else {
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(tmem),
                 "l"(a), "l"(b), "r"(IDESC_BF16), "r"(accumulate)
                 : "memory");
  }
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ bool elect_one() {
  uint32_t r;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(r));
  return r != 0u;
}
// two floats' bf16 parts, packed (the first in the low half); x becomes the remainder
__device__ __forceinline__ uint32_t take_bf16x2(float& x0, float& x1) {
  uint32_t w;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(w) : "f"(x1), "f"(x0));
  x0 -= __uint_as_float(w << 16);
  x1 -= __uint_as_float(w & 0xffff0000u);
  return w;
}

// the same of a pair (x - h as one f32x2 multiply-add, exact as the two differences are)
__device__ __forceinline__ uint32_t take_bf16x2(float2& x) {
  uint32_t w;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(w) : "f"(x.y), "f"(x.x));
  x = __ffma2_rn(make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)), make_float2(-1.0f, -1.0f), x);
  return w;
}

// One CTA per SM takes an equal run of the (row tile, K stage) pairs in tile order, across tiles without a break in the
// pipeline (a CTA's start and end cost ~5 us); a tile's sum is then that of the few CTAs whose runs meet it, each in a
// partial of its own. Stage g belongs to CTA run_cta(g). Stages x CTAs stay below 2^32 (run_ctas; n = 480,000 and more): the
// divisions of 64 bits took up to 1 us of a small sweep's kernels.
__device__ __forceinline__ uint32_t run_cta(uint32_t g, uint32_t total, uint32_t ctas) { return ((g + 1u) * ctas - 1u) / total; }
// the CTAs whose runs meet row tile `tile` of KT stages
__device__ __forceinline__ uint32_t run_segments(uint32_t tile, uint32_t KT, uint32_t n, uint32_t ctas) {
  const uint32_t total = (n + 127u) / 128u * KT, g = tile * KT;
  return run_cta(g + KT - 1u, total, ctas) - run_cta(g, total, ctas) + 1u;
}

// Bound: F from HBM. n = 32768, 64 columns: 323 us a BF16 sweep, 2.1 GB of F at 0.98 of the measured copy rate, and 640 us the accurate
// product's 4.3 GB (0.99); 361 and 660 by a CTA per row tile and quarter of K, whose starts and ends lay bare.
//
// The accumulation of the tensor cores drops what lies below the accumulator's last bit: an accumulator takes TC_CHAIN stages
// at most, the rest of a row's sum is in FP32 registers, rounded to nearest.
constexpr uint32_t TC_CHAIN = 2;
constexpr int TC_THREADS = 192;   // warps 0-3 drain, 4 TMA, 5 MMA

template <int MODE, int STAGES>
__global__ void __launch_bounds__(TC_THREADS, 1)
    tc_gemm_kernel(const __grid_constant__ TcMap mA, const __grid_constant__ TcMap mA2, const __grid_constant__ TcMap mB,
                   const __grid_constant__ TcMap mB2, uint32_t n, uint32_t R, float* __restrict__ partials, uint32_t* err) {
  constexpr bool X3 = MODE == TC_BF16X3;
  constexpr uint32_t STAGE_BYTES = (X3 ? 2 : 1) * (A_BYTES + B_BYTES);
  constexpr uint32_t K_ELEMS = MODE == TC_FP8 ? 128 : 64;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);
  // full[s]: a stage's tiles landed; empty[s]: its MMAs are done; ready[b]: accumulator b's MMAs are done; read[b]: it is
  // read back; fin: the last MMA is done
  auto full = [&](uint32_t s) { return smem_u32(bars + s); };
  auto empty = [&](uint32_t s) { return smem_u32(bars + STAGES + s); };
  auto ready = [&](uint32_t b) { return smem_u32(bars + 2 * STAGES + b); };
  auto read = [&](uint32_t b) { return smem_u32(bars + 2 * STAGES + 2 + b); };
  const uint32_t fin = smem_u32(bars + 2 * STAGES + 4);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 5);
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  const uint32_t KT = (n + K_ELEMS - 1u) / K_ELEMS;
  const uint32_t total = (n + 127u) / 128u * KT;
  const uint32_t g0 = blockIdx.x * total / gridDim.x, nkt = (blockIdx.x + 1u) * total / gridDim.x - g0;
  uint32_t tile = g0 / KT, kk = g0 % KT;   // of the role's next stage

  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < STAGES; s++) { mbar_init(full(s), 1); mbar_init(empty(s), 1); }
    for (uint32_t b = 0; b < 2; b++) { mbar_init(ready(b), 1); mbar_init(read(b), 4); }
    mbar_init(fin, 1);
    mbar_fence_init();
  }
  if (warp == 5) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 128;" ::"r"(smem_u32(tmem_slot)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 4) {
    if (lane == 0) {
      uint32_t issued = 0;
      for (uint32_t kt = 0; kt < nkt; kt++) {
        const uint32_t s = kt % STAGES;
        if (kt >= STAGES && !mbar_wait(empty(s), ((kt / STAGES) & 1u) ^ 1u, err)) break;
        mbar_expect_tx(full(s), STAGE_BYTES);
        const int32_t kx = int32_t(kk * K_ELEMS), m0 = int32_t(tile * 128u);
        const uint32_t at = smem_u32(smem + s * STAGE_BYTES), bt = at + (X3 ? 2 : 1) * A_BYTES;
        tma_load_2d(at, &mA, kx, m0, full(s));
        if (X3) tma_load_2d(at + A_BYTES, &mA2, kx, m0, full(s));
        tma_load_2d(bt, &mB, kx, 0, full(s));
        if (X3) tma_load_2d(bt + B_BYTES, &mB2, kx, 0, full(s));
        if (++kk == KT) { kk = 0; tile++; }
        issued++;
      }
      // drain: every stage this thread filled must have landed before the CTA may exit
      for (uint32_t kt = issued > STAGES ? issued - STAGES : 0; kt < issued; kt++) mbar_wait(full(kt % STAGES), (kt / STAGES) & 1u, err);
    }
  } else if (warp == 5) {
    // The whole warp runs the loop, so that the descriptors stay in uniform registers, and one elected lane issues
    const bool el = elect_one();
    const uint64_t A0 = sw128_desc(smem_u32(smem)), B0 = sw128_desc(smem_u32(smem + (X3 ? 2 : 1) * A_BYTES));
    uint32_t chain = 0;   // accumulators begun before this one
    for (uint32_t kt = 0; kt < nkt; kt++) {
      const uint32_t s = kt % STAGES, b = chain & 1u;
      const bool first = kt == 0u || kk % TC_CHAIN == 0u;
      bool ok = mbar_wait(full(s), (kt / STAGES) & 1u, err);
      if (first && chain >= 2u) ok = ok && mbar_wait(read(b), ((chain >> 1) - 1u) & 1u, err);
      if (++kk == KT) kk = 0;
      const bool last = kk % TC_CHAIN == 0u || kt + 1u == nkt;
      if (!__all_sync(0xffffffffu, ok)) break;
      tc_fence_after();
      const uint64_t A = A0 + ((s * STAGE_BYTES) >> 4), B = B0 + ((s * STAGE_BYTES) >> 4);
      const uint32_t d = tmem + 64u * b;
      if (el) {
#pragma unroll
        for (uint32_t k = 0; k < 4; k++) {   // 32 bytes of K each
          mma<MODE>(d, A + 2 * k, B + 2 * k, k || !first);
          if (X3) {
            mma<MODE>(d, A + 2 * k, B + (B_BYTES >> 4) + 2 * k, 1u);
            mma<MODE>(d, A + (A_BYTES >> 4) + 2 * k, B + 2 * k, 1u);
          }
        }
        mma_commit(empty(s));
        if (last) mma_commit(ready(b));
      }
      __syncwarp();
      if (last) chain++;
    }
    if (el) mma_commit(fin);
    mbar_wait(fin, 0, err);   // no MMA in flight when the TMEM is given back
  } else {
    // warp w reads accumulator rows 32 w .. 32 w + 31 (TMEM lanes)
    float acc[64];
#pragma unroll
    for (int c = 0; c < 64; c++) acc[c] = 0.0f;
    uint32_t chain = 0;
    for (uint32_t kt = 0; kt < nkt; kt++) {
      const bool end = ++kk == KT || kt + 1u == nkt;
      if (!end && kk % TC_CHAIN) continue;
      const uint32_t b = chain & 1u;
      if (!__all_sync(0xffffffffu, mbar_wait(ready(b), (chain >> 1) & 1u, err))) break;
      tc_fence_after();
      chain++;
#pragma unroll
      for (int q = 0; q < 4; q++) {
        float v[16];
        tmem_ld16(tmem + ((warp * 32u) << 16) + 64u * b + 16u * q, v);
#pragma unroll
        for (int c = 0; c < 16; c++) acc[16 * q + c] += v[c];
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(read(b));
      if (!end) continue;
      // the tile's end, or the run's: this CTA's partial of it
      const uint32_t row = tile * 128u + warp * 32u + lane, seg = blockIdx.x - run_cta(tile * KT, total, gridDim.x);
      if (row < n) {
        float4* dst = reinterpret_cast<float4*>(partials + (size_t(seg) * n + row) * 64);
#pragma unroll
        for (int c = 0; c < 16; c++)
          if (4u * c < R) dst[c] = make_float4(acc[4 * c], acc[4 * c + 1], acc[4 * c + 2], acc[4 * c + 3]);
      }
#pragma unroll
      for (int c = 0; c < 64; c++) acc[c] = 0.0f;
      kk = 0;
      tile++;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 5) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 128;" ::"r"(tmem) : "memory");
}

template <int MODE, int STAGES>
constexpr size_t smem_bytes() {
  return size_t(STAGES) * (MODE == TC_BF16X3 ? 2 : 1) * (A_BYTES + B_BYTES) + 1024 + 8 * (2 * STAGES + 5) + 16;
}

template <int MODE, int STAGES>
void launch_gemm(const TcMap* A, const TcMap* A2, const TcMap* B, const TcMap* B2, uint32_t n, uint32_t R, uint32_t ctas, float* partials,
                 uint32_t* err, cudaStream_t st) {
  static std::atomic<int> set[MAX_DEVICES];
  per_device_value(set, [](int) {
    cudaFuncSetAttribute(tc_gemm_kernel<MODE, STAGES>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem_bytes<MODE, STAGES>()));
    return 1;
  });
  tc_gemm_kernel<MODE, STAGES><<<ctas, TC_THREADS, smem_bytes<MODE, STAGES>(), st>>>(*A, A2 ? *A2 : *A, *B, B2 ? *B2 : *B, n, R, partials, err);
}

// ------------------------------------------------------------------------------------------------ FP32 sweeps
// F B in FP32 accuracy on the tensor cores. A float32 is the sum of three bf16 numbers (rounded to nearest at each step:
// m at most 2^-9 and l at most 2^-18 of it), so the product of two is h h' + (h m' + m h') + (h l' + l h' + m m') to
// 2^-26: six bf16 products, each exact. F stays FP32 in memory (no converted copy): its tiles arrive by TMA, converter warps
// split them in registers and store the parts to TMEM, from where tcgen05.mma takes its A operand; B's parts are K-major
// rows (h | m | l, 64 each) in shared memory.
//
// The tensor cores' accumulation drops what lies below the accumulator's last bit, which over a long sum of positive terms
// is a drift (-6.4e-8 of the sum when it is taken up every 64 of K). So the h h' sums of each 32 of K go to an accumulator of
// their own and four warps add a stage's two to FP32 registers, rounded to nearest, while the next stage's are made; the
// small products (2^-8 of the sum) stay in theirs for a tile's whole range. Error of F B against FP64 (2-norm, positive
// entries; the FMA chain of jacobi_gemm_fp32_kernel in brackets): n = 1540 6.3e-8 (6.9e-8), 4096 5.9e-8 (8.0e-8), 16384
// 1.6e-7 (1.9e-7); signed entries 9.3e-8 (2.0e-7) to 2.5e-7 (7.3e-7).
//
// A part reaches down to 2^-133, a float's last bit to 2^-149: F and B are taken FX_SCALE times each, so that the parts hold
// every bit of every float (without it 8 times the FMA chain's error where B is 2^-118), and the sums are scaled back. A
// sum past 2^96 (or a value past 2^112) overflows and takes the FMA kernel as an infinity does.
//
// Bound: F from HBM. n = 32768, 64 columns: 755 us a sweep with its combine, 4.3 GB of F in ~725 us (0.87 of the measured
// copy rate), against 3197 us on the FMA pipes. A stage is 32 KB of F, 1450 cycles of an SM's share of the bandwidth; its 24
// MMAs take 768. What held it back on the way there: one lane's MMA code (72 cycles an MMA), two waits of the MMA warp
// for each 32 of K (890 us), CTAs per tile and K split instead of one run each (a start and an end of ~5 us per 70 us).
constexpr float FX_SCALE = 65536.0f;
constexpr int FX_THREADS = 448;          // warps 0-3 drain, 4-11 convert, 12 TMA, 13 MMA
constexpr int FX_STAGES = 4;
constexpr uint32_t FX_F = 2 * 128 * 128, FX_B = 192 * 128, FX_STAGE = FX_F + FX_B;
constexpr uint32_t FX_A = 96, FX_HH = 192, FX_R = 448;   // TMEM columns: A parts (2 x 96 from 0), h h' (2 x 2 x 64), the rest (64)
constexpr size_t FX_SMEM = size_t(FX_STAGES) * FX_STAGE + 1024 + 256;

// D (+)= A B: A in TMEM (a row per lane, two bf16 of K per column), B by descriptor
__device__ __forceinline__ void mma_ta(uint32_t d, uint32_t a, uint64_t b, uint32_t accumulate) {
  asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}" ::"r"(d), "r"(a), "l"(b),
               "r"(IDESC_BF16), "r"(accumulate)
               : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr), "r"(r[0]),
      "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]),
      "r"(r[14]), "r"(r[15])
      : "memory");
}
// 16 columns of two neighbouring accumulators of 64
__device__ __forceinline__ void tmem_ld16x2(uint32_t taddr, float* v) {
  uint32_t r[32];
#pragma unroll
  for (int q = 0; q < 2; q++) {
    uint32_t* x = r + 16 * q;
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(x[0]), "=r"(x[1]), "=r"(x[2]), "=r"(x[3]), "=r"(x[4]), "=r"(x[5]), "=r"(x[6]), "=r"(x[7]), "=r"(x[8]), "=r"(x[9]), "=r"(x[10]),
          "=r"(x[11]), "=r"(x[12]), "=r"(x[13]), "=r"(x[14]), "=r"(x[15])
        : "r"(taddr + 64u * q));
  }
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; i++) v[i] = __uint_as_float(r[i]);
}
__global__ void __launch_bounds__(FX_THREADS, 1)
    tc_gemm_f32_kernel(const __grid_constant__ TcMap mF, const __grid_constant__ TcMap mB, uint32_t n, uint32_t R, float* __restrict__ partials,
                       uint32_t* err) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + FX_STAGES * FX_STAGE);
  // Stage kt has A buffer and h h' accumulators kt & 1. full[s]: a stage's tiles landed; empty[s]: its MMAs are done;
  // ready[b]: its A parts are in TMEM, its B tile landed and its accumulators are free; done[b]: its MMAs are done; drained[b]:
  // its h h' accumulators are read; rest: the small products of a tile are read; fin: the last MMA is done
  auto full = [&](uint32_t s) { return smem_u32(bars + s); };
  auto empty = [&](uint32_t s) { return smem_u32(bars + FX_STAGES + s); };
  auto ready = [&](uint32_t a) { return smem_u32(bars + 2 * FX_STAGES + a); };
  auto done = [&](uint32_t a) { return smem_u32(bars + 2 * FX_STAGES + 2 + a); };
  auto drained = [&](uint32_t b) { return smem_u32(bars + 2 * FX_STAGES + 4 + b); };
  const uint32_t rest = smem_u32(bars + 2 * FX_STAGES + 6), fin = smem_u32(bars + 2 * FX_STAGES + 7);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * FX_STAGES + 8);
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  const uint32_t KT = (n + 63u) / 64u;
  const uint32_t total = (n + 127u) / 128u * KT;
  const uint32_t g0 = blockIdx.x * total / gridDim.x, nkt = (blockIdx.x + 1u) * total / gridDim.x - g0;
  uint32_t tile = g0 / KT, kk = g0 % KT;   // of the role's next stage
  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < FX_STAGES; s++) { mbar_init(full(s), 1); mbar_init(empty(s), 1); }
    for (uint32_t b = 0; b < 2; b++) { mbar_init(ready(b), 8); mbar_init(done(b), 1); mbar_init(drained(b), 4); }
    mbar_init(rest, 4);
    mbar_init(fin, 1);
    mbar_fence_init();
  }
  if (warp == 13) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 12) {
    if (lane == 0) {
      uint32_t issued = 0;
      for (uint32_t kt = 0; kt < nkt; kt++) {
        const uint32_t s = kt % FX_STAGES;
        if (kt >= FX_STAGES && !mbar_wait(empty(s), ((kt / FX_STAGES) & 1u) ^ 1u, err)) break;
        mbar_expect_tx(full(s), FX_STAGE);
        const int32_t kx = int32_t(kk * 64u), m0 = int32_t(tile * 128u);
        const uint32_t at = smem_u32(smem + s * FX_STAGE);
        tma_load_2d(at, &mF, kx, m0, full(s));
        tma_load_2d(at + FX_F / 2, &mF, kx + 32, m0, full(s));
        tma_load_2d(at + FX_F, &mB, kx, 0, full(s));
        if (++kk == KT) { kk = 0; tile++; }
        issued++;
      }
      // drain: every stage this thread filled must have landed before the CTA may exit
      for (uint32_t kt = issued > FX_STAGES ? issued - FX_STAGES : 0; kt < issued; kt++) mbar_wait(full(kt % FX_STAGES), (kt / FX_STAGES) & 1u, err);
    }
  } else if (warp == 13) {
    // The whole warp runs the loop, so that the descriptors stay in uniform registers, and one elected lane issues (in one
    // lane's code an MMA took 72 cycles to issue; N = 64 runs in 32). A wait costs this warp ~200 cycles beside the
    // converters, so it makes one per stage: they wait for what `ready` stands for.
    const bool el = elect_one();
    const uint64_t B0 = sw128_desc(smem_u32(smem + FX_F));
    uint32_t tiles = 0;   // tiles begun before this one
    for (uint32_t kt = 0; kt < nkt; kt++) {
      const uint32_t s = kt % FX_STAGES, b = kt & 1u;
      const bool first = kt == 0u || kk == 0u;
      bool ok = mbar_wait(ready(b), (kt >> 1) & 1u, err);
      if (first) {
        if (tiles) ok = ok && mbar_wait(rest, (tiles - 1u) & 1u, err);
        tiles++;
      }
      if (++kk == KT) kk = 0;
      if (!__all_sync(0xffffffffu, ok)) break;
      tc_fence_after();
      const uint64_t Bs = B0 + ((s * FX_STAGE) >> 4);   // rows h' | m' | l', 512 units of 16 bytes each
      const uint32_t A = tmem + FX_A * b, hh = tmem + FX_HH + 128u * b, r = tmem + FX_R;
      if (el) {
#pragma unroll
        for (uint32_t k = 0; k < 4; k++) {   // 16 of K each
          const uint32_t h = A + 8 * k, m = h + 32, l = h + 64;
          const uint64_t Bh = Bs + 2 * k, Bm = Bh + 512, Bl = Bh + 1024;
          mma_ta(hh + 64u * (k >> 1), h, Bh, k & 1u);
          mma_ta(r, h, Bm, k || !first);
          mma_ta(r, m, Bh, 1u);
          mma_ta(r, h, Bl, 1u);
          mma_ta(r, l, Bh, 1u);
          mma_ta(r, m, Bm, 1u);
        }
        mma_commit(empty(s));
        mma_commit(done(b));
      }
      __syncwarp();
    }
    if (el) mma_commit(fin);
    mbar_wait(fin, 0, err);   // no MMA in flight when the TMEM is given back
  } else if (warp >= 4) {
    // converters: warps 4-7 the stage's first 32 of K, 8-11 the others; a thread takes a row (its TMEM lane)
    const uint32_t half = (warp - 4u) >> 2, row = (warp & 3u) * 32u + lane;
    for (uint32_t kt = 0; kt < nkt; kt++) {
      const uint32_t s = kt % FX_STAGES, b = kt & 1u;
      bool ok = mbar_wait(full(s), (kt / FX_STAGES) & 1u, err);
      if (kt >= 2u) ok = ok && mbar_wait(done(b), ((kt >> 1) - 1u) & 1u, err);   // the A buffer is free
      if (!__all_sync(0xffffffffu, ok)) break;
      tc_fence_after();
      const float4* src = reinterpret_cast<const float4*>(smem + s * FX_STAGE + half * (FX_F / 2) + row * 128u);
      const uint32_t taddr = tmem + FX_A * b + 16u * half + (((warp & 3u) * 32u) << 16);
      uint32_t h[16], m[16], l[16];
#pragma unroll
      for (uint32_t c = 0; c < 8; c++) {
        const float4 f = src[c ^ (row & 7u)];   // 128-byte swizzle
        float2 x = __fmul2_rn(make_float2(f.x, f.y), make_float2(FX_SCALE, FX_SCALE));
        float2 y = __fmul2_rn(make_float2(f.z, f.w), make_float2(FX_SCALE, FX_SCALE));
        h[2 * c] = take_bf16x2(x); h[2 * c + 1] = take_bf16x2(y);
        m[2 * c] = take_bf16x2(x); m[2 * c + 1] = take_bf16x2(y);
        l[2 * c] = take_bf16x2(x); l[2 * c + 1] = take_bf16x2(y);
      }
      tmem_st16(taddr, h);
      tmem_st16(taddr + 32, m);
      tmem_st16(taddr + 64, l);
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      if (kt >= 2u && !__all_sync(0xffffffffu, mbar_wait(drained(b), ((kt >> 1) - 1u) & 1u, err))) break;
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(ready(b));
    }
  } else {
    // drain: a stage's h h' sums in one rounding to nearest, in K order; at a tile's end the small products
    float acc[64];
#pragma unroll
    for (int c = 0; c < 64; c++) acc[c] = 0.0f;
    const uint32_t base = tmem + ((warp * 32u) << 16);
    for (uint32_t kt = 0; kt < nkt; kt++) {
      if (!__all_sync(0xffffffffu, mbar_wait(done(kt & 1u), (kt >> 1) & 1u, err))) break;
      tc_fence_after();
#pragma unroll
      for (int g = 0; g < 4; g++) {
        float v[32];
        tmem_ld16x2(base + FX_HH + 128u * (kt & 1u) + 16u * g, v);
#pragma unroll
        for (int c = 0; c < 16; c++) acc[16 * g + c] += v[c] + v[16 + c];
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(drained(kt & 1u));
      if (++kk < KT && kt + 1u < nkt) continue;
      // the tile's end, or the run's: this CTA's partial of it
#pragma unroll
      for (int g = 0; g < 4; g++) {
        float v[16];
        tmem_ld16(base + FX_R + 16u * g, v);
#pragma unroll
        for (int c = 0; c < 16; c++) acc[16 * g + c] += v[c];
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(rest);
      const uint32_t row = tile * 128u + warp * 32u + lane, seg = blockIdx.x - run_cta(tile * KT, total, gridDim.x);
      if (row < n) {
        float4* dst = reinterpret_cast<float4*>(partials + (size_t(seg) * n + row) * R);
#pragma unroll
        for (int c = 0; c < 16; c++)
          if (4u * c < R) dst[c] = make_float4(acc[4 * c], acc[4 * c + 1], acc[4 * c + 2], acc[4 * c + 3]);
      }
#pragma unroll
      for (int c = 0; c < 64; c++) acc[c] = 0.0f;
      kk = 0;
      tile++;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 13) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}

__device__ __forceinline__ void block_sum2(double a, double b, double* partials) {
  __shared__ double sa[32], sb[32];
  for (int o = 16; o > 0; o >>= 1) { a += __shfl_down_sync(0xffffffffu, a, o); b += __shfl_down_sync(0xffffffffu, b, o); }
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
  if (l == 0) { sa[w] = a; sb[w] = b; }
  __syncthreads();
  if (w == 0) {
    a = l < nw ? sa[l] : 0.0;
    b = l < nw ? sb[l] : 0.0;
    for (int o = 16; o > 0; o >>= 1) { a += __shfl_down_sync(0xffffffffu, a, o); b += __shfl_down_sync(0xffffffffu, b, o); }
    if (l == 0) { partials[2 * blockIdx.x] = a; partials[2 * blockIdx.x + 1] = b; }
  }
}

// A tile of 32 rows of the n x R iterate, in shared memory, to the bf16 parts of FX_SCALE times it as K-major rows: Bt (192 x np): row 64 q + c
// holds part q of column c. A thread splits two neighbours of K: a 32-bit store per part (np is even); c < R
__device__ __forceinline__ void store_parts(const float (*tile)[65], uint32_t i0, uint32_t R, uint32_t np, uint16_t* __restrict__ Bt) {
  for (uint32_t q = threadIdx.x; q < R * 16u; q += 256u) {
    const uint32_t c = q / 16u, k = 2u * (q % 16u);
    float x0 = tile[k][c] * FX_SCALE, x1 = tile[k + 1u][c] * FX_SCALE;
    uint32_t* dst = reinterpret_cast<uint32_t*>(Bt + size_t(c) * np + i0 + k);
    dst[0] = take_bf16x2(x0, x1);
    dst[size_t(32) * np] = take_bf16x2(x0, x1);
    dst[size_t(64) * np] = take_bf16x2(x0, x1);
  }
}
__global__ void __launch_bounds__(256) pack_b_f32_kernel(const float* __restrict__ X, uint32_t n, uint32_t R, uint32_t np, uint16_t* __restrict__ Bt) {
  __shared__ float tile[32][65];
  const uint32_t i0 = blockIdx.x * 32u;
  for (uint32_t q = threadIdx.x; q < 32u * R; q += 256u) tile[q / R][q % R] = i0 + q / R < n ? X[size_t(i0) * R + q] : 0.0f;
  __syncthreads();
  store_parts(tile, i0, R, np, Bt);
}

// Y = E + rho (sum of the tile's partials, in CTA order), its parts for the next sweep, and the block's
// sums of |Y - X|^2 and |Y|^2
__global__ void __launch_bounds__(256) combine_f32_kernel(const float* __restrict__ part, uint32_t ctas, const float* __restrict__ rho,
                                                          const float* __restrict__ E, const float* __restrict__ X, float* __restrict__ Y, uint32_t n,
                                                          uint32_t R, uint32_t np, uint16_t* __restrict__ Bt, double* __restrict__ norms) {
  __shared__ float tile[32][65];
  const uint32_t i0 = blockIdx.x * 32u, R4 = R / 4u;
  const size_t stride = size_t(n) * R4;
  const float4* P = reinterpret_cast<const float4*>(part);
  const uint32_t splits = i0 < n ? run_segments(i0 / 128u, (n + 63u) / 64u, n, ctas) : 0u;
  double d2 = 0.0, b2 = 0.0;
  for (uint32_t q = threadIdx.x; q < 32u * R4; q += 256u) {
    const uint32_t r = q / R4, c = 4u * (q % R4);
    float4 b = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (i0 + r < n) {
      const size_t i = size_t(i0) * R4 + q;
      float4 a = P[i];
      for (uint32_t s = 1; s < splits; s++) {
        const float4 v = P[s * stride + i];
        a.x += v.x; a.y += v.y; a.z += v.z; a.w += v.w;
      }
      constexpr float back = 1.0f / (FX_SCALE * FX_SCALE);
      a.x *= back; a.y *= back; a.z *= back; a.w *= back;
      const float rr = rho[i0 + r];
      const float4 e = reinterpret_cast<const float4*>(E)[i], x = reinterpret_cast<const float4*>(X)[i];
      b = make_float4(fmaf(rr, a.x, e.x), fmaf(rr, a.y, e.y), fmaf(rr, a.z, e.z), fmaf(rr, a.w, e.w));
      reinterpret_cast<float4*>(Y)[i] = b;
      const double dx = double(b.x) - x.x, dy = double(b.y) - x.y, dz = double(b.z) - x.z, dw = double(b.w) - x.w;
      d2 += dx * dx + dy * dy + dz * dz + dw * dw;
      b2 += double(b.x) * b.x + double(b.y) * b.y + double(b.z) * b.z + double(b.w) * b.w;
    }
    tile[r][c] = b.x; tile[r][c + 1u] = b.y; tile[r][c + 2u] = b.z; tile[r][c + 3u] = b.w;
  }
  __syncthreads();
  store_parts(tile, i0, R, np, Bt);
  block_sum2(d2, b2, norms);
}

// ------------------------------------------------------------------------------------------------ CUDA-core helpers
__global__ void split_bf16_kernel(const float* __restrict__ F, __nv_bfloat16* __restrict__ hi, __nv_bfloat16* __restrict__ lo, size_t count) {
  for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < count; i += size_t(gridDim.x) * blockDim.x) {
    const float f = F[i];
    const __nv_bfloat16 h = __float2bfloat16_rn(f);
    hi[i] = h;
    lo[i] = __float2bfloat16_rn(f - __bfloat162float(h));
  }
}

__device__ __forceinline__ float block_max(float v) {
  __shared__ float red[32];
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) red[w] = v;
  __syncthreads();
  if (w == 0) {
    v = l < int(blockDim.x >> 5) ? red[l] : 0.0f;
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    if (l == 0) red[0] = v;
  }
  __syncthreads();
  const float r = red[0];
  __syncthreads();
  return r;
}

// one block per row: s_i = max_j |F_ij| / 448 (the largest finite e4m3), q_ij = e4m3(F_ij / s_i)
__global__ void quant_rows_fp8_kernel(const float* __restrict__ F, uint8_t* __restrict__ q, float* __restrict__ row_scale, uint32_t n) {
  const size_t base = size_t(blockIdx.x) * n;
  float m = 0.0f;
  for (uint32_t j = threadIdx.x; j < n; j += blockDim.x) m = fmaxf(m, fabsf(F[base + j]));
  m = block_max(m);
  const float s = m > 0.0f ? m / 448.0f : 1.0f;
  if (threadIdx.x == 0) row_scale[blockIdx.x] = s;
  const float inv = 1.0f / s;
  for (uint32_t j = threadIdx.x; j < n; j += blockDim.x) {
    const __nv_fp8_e4m3 e(F[base + j] * inv);
    q[base + j] = *reinterpret_cast<const uint8_t*>(&e);
  }
}

// column maxima of X (n x R) for the FP8 column scales (positive floats compare as their bit patterns)
__global__ void col_max_kernel(const float* __restrict__ X, uint32_t n, uint32_t R, uint32_t* __restrict__ col_max) {
  const uint32_t c = threadIdx.x % 64u;
  float m = 0.0f;
  if (c < R)
    for (uint32_t i = blockIdx.x * (blockDim.x / 64u) + threadIdx.x / 64u; i < n; i += gridDim.x * (blockDim.x / 64u))
      m = fmaxf(m, fabsf(X[size_t(i) * R + c]));
  if (c < R && m > 0.0f) atomicMax(col_max + c, __float_as_uint(m));
}

// X (n x R) -> Bt (64 x n): transposed through a 32 x 32 shared tile; rows c >= R of Bt are zero
template <int MODE>
__global__ void pack_b_kernel(const float* __restrict__ X, uint32_t n, uint32_t R, __nv_bfloat16* __restrict__ hi, __nv_bfloat16* __restrict__ lo,
                              uint8_t* __restrict__ q8, const uint32_t* __restrict__ col_max, float* __restrict__ col_scale) {
  __shared__ float tile[32][33];
  const uint32_t i0 = blockIdx.x * 32u, c0 = blockIdx.y * 32u;
  for (uint32_t k = threadIdx.y; k < 32u; k += blockDim.y) {
    const uint32_t i = i0 + k, c = c0 + threadIdx.x;
    tile[k][threadIdx.x] = (i < n && c < R) ? X[size_t(i) * R + c] : 0.0f;
  }
  __syncthreads();
  for (uint32_t k = threadIdx.y; k < 32u; k += blockDim.y) {
    const uint32_t c = c0 + k, i = i0 + threadIdx.x;
    if (i >= n) continue;
    const float x = tile[threadIdx.x][k];
    const size_t o = size_t(c) * n + i;
    if (MODE == TC_FP8) {
      const float m = c < R ? __uint_as_float(col_max[c]) : 0.0f;
      const float s = m > 0.0f ? m / 448.0f : 1.0f;
      if (blockIdx.x == 0 && threadIdx.x == 0) col_scale[c] = s;
      const __nv_fp8_e4m3 e(x / s);
      q8[o] = *reinterpret_cast<const uint8_t*>(&e);
    } else {
      const __nv_bfloat16 h = __float2bfloat16_rn(x);
      hi[o] = h;
      lo[o] = __float2bfloat16_rn(x - __bfloat162float(h));
    }
  }
}

constexpr uint32_t CB_THREADS = 256;

// a block's sums of a and b into partials[2 block], [2 block + 1]: per thread and per warp in FP32, per block in FP64
// (a sweep's stopping test needs no more, and FP64 per element would cost more than the sweep's memory traffic)
__device__ __forceinline__ void block_sum2f(float a, float b, double* partials) {
  __shared__ double sa[32], sb[32];
  for (int o = 16; o > 0; o >>= 1) { a += __shfl_down_sync(0xffffffffu, a, o); b += __shfl_down_sync(0xffffffffu, b, o); }
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
  if (l == 0) { sa[w] = double(a); sb[w] = double(b); }
  __syncthreads();
  if (w == 0) {
    double x = l < nw ? sa[l] : 0.0, y = l < nw ? sb[l] : 0.0;
    for (int o = 16; o > 0; o >>= 1) { x += __shfl_down_sync(0xffffffffu, x, o); y += __shfl_down_sync(0xffffffffu, y, o); }
    if (l == 0) { partials[2 * blockIdx.x] = x; partials[2 * blockIdx.x + 1] = y; }
  }
}

// Rows that a block of the combining kernels takes: 32, but 8 where blocks of 32 would be fewer than the SMs and there are columns
// enough for the threads. The residual's FP64 (few units an SM) and the reads of up to nine partials then lie on four times the SMs:
// FP8 with 64 columns, n = 512, 1024, 2048, 3008 a solve: 703, 767, 769, 847 us with 32 rows, 669, 733, 731, 797 with 8; from n =
// 4864 on, and with 4 columns, 32 take the same or less (n = 4096, BF16: 595 us, 614 with 8)
constexpr uint32_t CB_FEW = 8, CB_MANY = 32;
uint32_t combine_rows(uint32_t n, uint32_t R) { return n < CB_MANY * 152u && R > 16u ? CB_FEW : CB_MANY; }

// a block's rows of the iterate, in shared memory, to the next sweep's right-hand sides in BF16 (c < R; the other rows of
// Bt stay zero): two neighbours of K a store (n is a multiple of 16)
template <uint32_t ROWS>
__device__ __forceinline__ void store_hi(const float (*tile)[65], uint32_t i0, uint32_t n, uint32_t R, uint16_t* __restrict__ Bt) {
  for (uint32_t q = threadIdx.x; q < R * (ROWS / 2u); q += CB_THREADS) {
    const uint32_t c = q / (ROWS / 2u), k = 2u * (q % (ROWS / 2u));
    if (i0 + k >= n) continue;
    float x0 = tile[k][c], x1 = tile[k + 1u][c];
    *reinterpret_cast<uint32_t*>(Bt + size_t(c) * n + i0 + k) = take_bf16x2(x0, x1);
  }
}

// Y = rhs + rho (sum of the row tile's partials, in CTA order), ROWS rows a block; Bt: also the next sweep's right-hand sides
// (null: none). Norms of Y - Xin and Y in FP32 per thread. W: columns a thread takes at a time, 4 where R is a multiple (n =
// 32768, 64 columns: 12 us, 20 a column at a time; with a pack launch of its own 35)
template <int W, uint32_t ROWS>
__global__ void __launch_bounds__(CB_THREADS) combine_sweep_kernel(const float* __restrict__ P, uint32_t ctas, uint32_t KT, uint32_t n, uint32_t R,
                                                                   const float* __restrict__ rho, const float* __restrict__ rhs,
                                                                   const float* __restrict__ Xin, float* __restrict__ Y,
                                                                   const float* __restrict__ rs, const float* __restrict__ cs,
                                                                   uint16_t* __restrict__ Bt, double* __restrict__ parts) {
  __shared__ float tile[ROWS][65];
  const uint32_t i0 = blockIdx.x * ROWS, rows = min(ROWS, n - i0), RW = R / W, segs = run_segments(i0 / 128u, KT, n, ctas);
  auto load = [](const float* p, float* v) {
    if (W == 4) {
      const float4 x = *reinterpret_cast<const float4*>(p);
      v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
    } else {
      v[0] = *p;
    }
  };
  float d2 = 0.0f, y2 = 0.0f;
#pragma unroll 2
  for (uint32_t q = threadIdx.x; q < rows * RW; q += CB_THREADS) {
    const uint32_t r = q / RW, c = W * (q % RW), i = i0 + r;
    const size_t idx = size_t(i) * R + c;
    float acc[W], v[W], e[W], x[W];
    load(rhs + idx, e);
    load(Xin + idx, x);
    load(P + size_t(i) * 64 + c, acc);
#pragma unroll 4
    for (uint32_t s = 1; s < segs; s++) {
      load(P + (size_t(s) * n + i) * 64 + c, v);
#pragma unroll
      for (int k = 0; k < W; k++) acc[k] += v[k];
    }
#pragma unroll
    for (int k = 0; k < W; k++) {
      if (rs) acc[k] *= rs[i] * cs[c + k];
      acc[k] = fmaf(rho[i], acc[k], e[k]);
      tile[r][c + k] = acc[k];
      const float dd = acc[k] - x[k];
      d2 = fmaf(dd, dd, d2);
      y2 = fmaf(acc[k], acc[k], y2);
    }
    if (W == 4) *reinterpret_cast<float4*>(Y + idx) = make_float4(acc[0], acc[1 % W], acc[2 % W], acc[3 % W]);
    else Y[idx] = acc[0];
  }
  __syncthreads();
  if (Bt) store_hi<ROWS>(tile, i0, n, R, Bt);
  block_sum2f(d2, y2, parts);
}

// r = E + rho (sum of the partials) - B in FP64, and r's BF16 columns (Bt, null: none)
template <uint32_t ROWS>
__global__ void __launch_bounds__(CB_THREADS) combine_residual_kernel(const float* __restrict__ P, uint32_t ctas, uint32_t KT, uint32_t n, uint32_t R,
                                                                      const float* __restrict__ rho, const float* __restrict__ E,
                                                                      const float* __restrict__ B, float* __restrict__ r, uint16_t* __restrict__ Bt,
                                                                      double* __restrict__ parts) {
  __shared__ float tile[ROWS][65];
  const uint32_t i0 = blockIdx.x * ROWS, rows = min(ROWS, n - i0), segs = run_segments(i0 / 128u, KT, n, ctas);
  double r2 = 0.0, b2 = 0.0;
#pragma unroll 4
  for (uint32_t q = threadIdx.x; q < rows * R; q += CB_THREADS) {
    const uint32_t k = q / R, c = q % R, i = i0 + k;
    const size_t idx = size_t(i0) * R + q;
    float acc = P[size_t(i) * 64 + c];
#pragma unroll 4
    for (uint32_t s = 1; s < segs; s++) acc += P[(size_t(s) * n + i) * 64 + c];
    const double b = double(B[idx]), rr = double(E[idx]) + double(rho[i]) * double(acc) - b;
    const float x = float(rr);
    r[idx] = x;
    tile[k][c] = x;
    r2 += rr * rr;
    b2 += b * b;
  }
  __syncthreads();
  if (Bt) store_hi<ROWS>(tile, i0, n, R, Bt);
  block_sum2(r2, b2, parts);
}

__global__ void axpy_kernel(float* __restrict__ B, const float* __restrict__ d, size_t count) {
  for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < count; i += size_t(gridDim.x) * blockDim.x) B[i] += d[i];
}

using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                              const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                              CUtensorMapFloatOOBfill);
EncodeFn encode_fn() {
  static EncodeFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeFn>(p);
  });
  return fn;
}

}  // namespace

static_assert(sizeof(CUtensorMap) == sizeof(TcMap), "tensor map size");

bool tc_encode(TcMap* map, const void* base, uint32_t inner, uint32_t rows, uint32_t elt_bytes, uint32_t box_rows, int* code, uint32_t pitch) {
  EncodeFn fn = encode_fn();
  if (!fn) { if (code) *code = -1; return false; }
  const cuuint64_t dims[2] = {inner, rows};
  const cuuint64_t strides[1] = {cuuint64_t(pitch ? pitch : inner) * elt_bytes};
  const cuuint32_t box[2] = {128u / elt_bytes, box_rows};
  const cuuint32_t estr[2] = {1, 1};
  const CUtensorMapDataType type = elt_bytes == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : elt_bytes == 2 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8;
  const CUresult r = fn(reinterpret_cast<CUtensorMap*>(map), type, 2,
                        const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (code) *code = int(r);
  return r == CUDA_SUCCESS;
}

// `ctas` CTAs at most for `total` stages
static uint32_t run_ctas(uint64_t ctas, uint64_t total) { return uint32_t(std::max<uint64_t>(1, std::min<uint64_t>(ctas, 0xffffffffu / total))); }
// One CTA per SM; runs of an eighth of a row tile at least, so that few of them meet a tile
uint32_t tc_ctas(int mode, uint32_t n, uint32_t sms) {
  const uint32_t ke = mode == TC_FP8 ? 128u : 64u, KT = (n + ke - 1u) / ke;
  const uint64_t total = uint64_t((n + 127u) / 128u) * KT;
  return run_ctas(std::min<uint64_t>(sms, total / ((KT + 7u) / 8u)), total);
}
uint32_t tc_segments(int mode, uint32_t n, uint32_t ctas) {
  const uint32_t ke = mode == TC_FP8 ? 128u : 64u, KT = (n + ke - 1u) / ke;
  return uint32_t(KT / std::max<uint64_t>(1, uint64_t((n + 127u) / 128u) * KT / ctas)) + 2u;
}

void tc_gemm(int mode, const TcMap* A, const TcMap* A2, const TcMap* B, const TcMap* B2, uint32_t n, uint32_t R, uint32_t ctas, float* partials,
             uint32_t* err, cudaStream_t st) {
  if (mode == TC_BF16) launch_gemm<TC_BF16, 6>(A, A2, B, B2, n, R, ctas, partials, err, st);
  else if (mode == TC_BF16X3) launch_gemm<TC_BF16X3, 4>(A, A2, B, B2, n, R, ctas, partials, err, st);
  else launch_gemm<TC_FP8, 6>(A, A2, B, B2, n, R, ctas, partials, err, st);
}

size_t tc_f32_parts_bytes(uint32_t n) { return size_t(192) * tc_f32_pad(n) * 2; }

// one CTA per SM, and the most CTAs whose runs meet one tile
uint32_t tc_f32_ctas(uint32_t n, uint32_t sms) {
  const uint64_t total = uint64_t((n + 127u) / 128u) * ((n + 63u) / 64u);
  return run_ctas(std::min<uint64_t>(sms, total), total);
}
uint32_t tc_f32_segments(uint32_t n, uint32_t ctas) {
  const uint32_t KT = (n + 63u) / 64u;
  const uint64_t run = uint64_t((n + 127u) / 128u) * KT / ctas;
  return uint32_t(KT / std::max<uint64_t>(1, run)) + 2u;
}

void tc_gemm_f32(const TcMap* F, const TcMap* B, uint32_t n, uint32_t R, uint32_t ctas, float* partials, uint32_t* err, cudaStream_t st) {
  static std::atomic<int> set[MAX_DEVICES];
  per_device_value(set, [](int) { cudaFuncSetAttribute(tc_gemm_f32_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(FX_SMEM)); return 1; });
  tc_gemm_f32_kernel<<<ctas, FX_THREADS, FX_SMEM, st>>>(*F, *B, n, R, partials, err);
}

void tc_pack_b_f32(const float* X, uint32_t n, uint32_t R, uint16_t* Bt, cudaStream_t st) {
  const uint32_t np = tc_f32_pad(n);
  pack_b_f32_kernel<<<np / 32, 256, 0, st>>>(X, n, R, np, Bt);
}

uint32_t tc_combine_f32(const float* part, uint32_t ctas, const float* rho, const float* E, const float* X, float* Y, uint32_t n, uint32_t R, uint16_t* Bt,
                        double* norms, cudaStream_t st) {
  const uint32_t np = tc_f32_pad(n);
  combine_f32_kernel<<<np / 32, 256, 0, st>>>(part, ctas, rho, E, X, Y, n, R, np, Bt, norms);
  return np / 32;
}

void tc_split_bf16(const float* F, uint16_t* hi, uint16_t* lo, size_t count, cudaStream_t st) {
  split_bf16_kernel<<<1216, 256, 0, st>>>(F, reinterpret_cast<__nv_bfloat16*>(hi), reinterpret_cast<__nv_bfloat16*>(lo), count);
}

void tc_quant_rows_fp8(const float* F, uint8_t* q, float* row_scale, uint32_t n, cudaStream_t st) {
  quant_rows_fp8_kernel<<<n, 256, 0, st>>>(F, q, row_scale, n);
}

void tc_pack_b(int mode, const float* X, uint32_t n, uint32_t R, uint16_t* hi, uint16_t* lo, uint8_t* q8, float* col_scale,
               uint32_t* col_max, cudaStream_t st) {
  const dim3 grid((n + 31) / 32, 2), block(32, 8);
  if (mode == TC_FP8) {
    cudaMemsetAsync(col_max, 0, 64 * sizeof(uint32_t), st);
    col_max_kernel<<<304, 256, 0, st>>>(X, n, R, col_max);
    pack_b_kernel<TC_FP8><<<grid, block, 0, st>>>(X, n, R, nullptr, nullptr, q8, col_max, col_scale);
  } else {
    pack_b_kernel<TC_BF16X3><<<grid, block, 0, st>>>(X, n, R, reinterpret_cast<__nv_bfloat16*>(hi), reinterpret_cast<__nv_bfloat16*>(lo),
                                                     nullptr, nullptr, nullptr);
  }
}

uint32_t tc_combine_sweep(int mode, const float* partials, uint32_t ctas, uint32_t n, uint32_t R, const float* rho, const float* rhs, const float* Xin,
                          float* Y, const float* row_scale, const float* col_scale, uint16_t* Bt, double* norm_partials, cudaStream_t st) {
  const uint32_t rows = combine_rows(n, R), blocks = (n + rows - 1u) / rows, ke = mode == TC_FP8 ? 128u : 64u;
  const auto kernel = rows == CB_FEW ? (R % 4u ? combine_sweep_kernel<1, CB_FEW> : combine_sweep_kernel<4, CB_FEW>)
                                     : (R % 4u ? combine_sweep_kernel<1, CB_MANY> : combine_sweep_kernel<4, CB_MANY>);
  kernel<<<blocks, CB_THREADS, 0, st>>>(partials, ctas, (n + ke - 1u) / ke, n, R, rho, rhs, Xin, Y, row_scale, col_scale, Bt, norm_partials);
  return blocks;
}

uint32_t tc_combine_residual(const float* partials, uint32_t ctas, uint32_t n, uint32_t R, const float* rho, const float* E, const float* B, float* r,
                             uint16_t* Bt, double* norm_partials, cudaStream_t st) {
  const uint32_t rows = combine_rows(n, R), blocks = (n + rows - 1u) / rows;
  const auto kernel = rows == CB_FEW ? combine_residual_kernel<CB_FEW> : combine_residual_kernel<CB_MANY>;
  kernel<<<blocks, CB_THREADS, 0, st>>>(partials, ctas, (n + 63u) / 64u, n, R, rho, E, B, r, Bt, norm_partials);
  return blocks;
}

void tc_axpy(float* B, const float* d, size_t count, cudaStream_t st) { axpy_kernel<<<1216, 256, 0, st>>>(B, d, count); }

}  // namespace vtk

// ------------------------------------------------------------------------------------------------ wait check
// The bounded-wait path of the pipelines above, exercised on purpose: one block waits on an mbarrier phase that
// completes only if `arrive` is set (one arrival of the barrier's count of 1). Without it the wait runs out after
// `cycles`, sets the error word and the kernel returns: the host sees a timeout and the context stays usable.
namespace vtk {
__global__ void wait_check_kernel(uint64_t cycles, uint32_t arrive, uint32_t* err) {
  __shared__ __align__(8) uint64_t bar;
  const uint32_t b = async::smem_u32(&bar);
  if (threadIdx.x == 0) {
    async::mbar_init(b, 1);
    async::mbar_fence_init();
  }
  __syncthreads();
  if (threadIdx.x == 0 && arrive) async::mbar_arrive(b);
  if (threadIdx.x == 0) async::mbar_wait(b, 0, err, cycles);
}
void launch_wait_check(uint64_t cycles, uint32_t arrive, uint32_t* err, cudaStream_t st) {
  wait_check_kernel<<<1, 32, 0, st>>>(cycles, arrive, err);
}
}  // namespace vtk
