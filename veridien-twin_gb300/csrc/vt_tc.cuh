// Tensor-core (tcgen05) Jacobi sweeps of the node radiosity with many right-hand sides (vt_tc.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace vtk {

enum TcMode { TC_BF16 = 0, TC_BF16X3 = 1, TC_FP8 = 2 };

// opaque tensor-map storage (CUtensorMap is 128 bytes, 64-byte aligned)
struct alignas(64) TcMap { unsigned char bytes[128]; };

// F (n x n, K contiguous) and the transposed right-hand sides Bt (r x n, K contiguous) as TMA tiles:
// mode BF16 / BF16X3: bf16 elements, boxes of 64 x 128 (F) and 64 x 64 (Bt); FP8: bytes, boxes of 128 x 128 / 128 x 64.
// Returns false (with the driver's error code in *code) when the map cannot be encoded.
// pitch: elements from row to row (0: inner).
bool tc_encode(TcMap* map, const void* base, uint32_t inner, uint32_t rows, uint32_t elt_bytes, uint32_t box_rows, int* code, uint32_t pitch = 0);

// A B by `ctas` CTAs, three products for BF16X3: partials[s][i][c], s < tc_segments, c < R (rows of 64), summed over the
// segments of row i's tile by the combine functions
uint32_t tc_ctas(int mode, uint32_t n, uint32_t sms);
uint32_t tc_segments(int mode, uint32_t n, uint32_t ctas);
void tc_gemm(int mode, const TcMap* A, const TcMap* A2, const TcMap* B, const TcMap* B2, uint32_t n, uint32_t R, uint32_t ctas, float* partials,
             uint32_t* err, cudaStream_t st);

// FP32 F (n x n, n % 4 == 0, 16-byte aligned rows) times the FP32 columns whose parts tc_pack_b_f32 laid out, by `ctas`
// CTAs: partials[s][i][c], s < tc_f32_segments, summed over the segments of row i's tile by tc_combine_f32; c < R
inline uint32_t tc_f32_pad(uint32_t n) { return (n + 63u) / 64u * 64u; }
size_t tc_f32_parts_bytes(uint32_t n);   // X's parts: 192 rows (h | m | l, 64 columns each) of tc_f32_pad(n) bf16
uint32_t tc_f32_ctas(uint32_t n, uint32_t sms);
uint32_t tc_f32_segments(uint32_t n, uint32_t ctas);
void tc_pack_b_f32(const float* X, uint32_t n, uint32_t R, uint16_t* Bt, cudaStream_t st);
void tc_gemm_f32(const TcMap* F, const TcMap* B, uint32_t n, uint32_t R, uint32_t ctas, float* partials, uint32_t* err, cudaStream_t st);
// Y = E + rho (sum of the partials), Y's parts into Bt, norms of Y - X and Y per block; returns the blocks
uint32_t tc_combine_f32(const float* part, uint32_t ctas, const float* rho, const float* E, const float* X, float* Y, uint32_t n, uint32_t R, uint16_t* Bt,
                        double* norms, cudaStream_t st);

// F (fp32) -> hi = bf16(F), lo = bf16(F - hi)
void tc_split_bf16(const float* F, uint16_t* hi, uint16_t* lo, size_t count, cudaStream_t st);
// F (fp32, n x n) -> q = e4m3(F / s_i), s_i = max_j |F_ij| / 448 (one scale per row)
void tc_quant_rows_fp8(const float* F, uint8_t* q, float* row_scale, uint32_t n, cudaStream_t st);
// X (n x R fp32, row-major) -> Bt (64 x n, transposed, rows >= R zero): bf16 hi and lo, or e4m3 with one scale per column
void tc_pack_b(int mode, const float* X, uint32_t n, uint32_t R, uint16_t* hi, uint16_t* lo, uint8_t* q8, float* col_scale,
               uint32_t* col_max, cudaStream_t st);
// Jacobi sweep epilogue: Y = rhs + rho * (sum of the partials) [* s_i t_c], norms of Y - Xin and Y per block; Bt: Y's
// columns < R in bf16 as tc_pack_b lays them out (null: none). Returns the blocks.
uint32_t tc_combine_sweep(int mode, const float* partials, uint32_t ctas, uint32_t n, uint32_t R, const float* rho, const float* rhs, const float* Xin,
                          float* Y, const float* row_scale, const float* col_scale, uint16_t* Bt, double* norm_partials, cudaStream_t st);
// accurate residual of a BF16X3 product: r = E + rho * acc - B in float64 (stored fp32), norms of r and B per block; Bt as above
uint32_t tc_combine_residual(const float* partials, uint32_t ctas, uint32_t n, uint32_t R, const float* rho, const float* E, const float* B, float* r,
                             uint16_t* Bt, double* norm_partials, cudaStream_t st);
// B += d
void tc_axpy(float* B, const float* d, size_t count, cudaStream_t st);

// one bounded mbarrier wait that completes only when `arrive` is set; *err is set when it runs out after `cycles`
void launch_wait_check(uint64_t cycles, uint32_t arrive, uint32_t* err, cudaStream_t st);

}  // namespace vtk
