// Grouped tensor-core GEMM for token counts above the streaming kernel's limit:
//     out[g][n][m] = sum_k W[g][m][k] * A[g][n][k]
// fp32 accumulation in TMEM, 16-bit output.  128 tokens are the rows of the tcgen05 tile, up to 256 weight rows its columns; an epilogue
// thread owns one token and writes runs of consecutive outputs.  (umma_wq.cu has the weights as the rows.)
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace blr {

struct alignas(64) GemmParams {
  CUtensorMap tmW;  // K-major: dims (K, M, G) box (64, row-tile, 1); M-major: dims (M, K, G) box (64, 64, 1)
                    // quantised weights (w_bits 8 | 4, K-major): bytes, dims (K*w_bits/8, M, G) box (8*w_bits, row-tile, 1), no swizzle
  CUtensorMap tmA;  // dims (K, N, G) box (64, token-tile, 1)
  int G, M, K, N;
  int kmajor;          // weight layout
  int w_odd;           // 16-bit weights whose rows start off 32 bytes: M-major ones, or K-major slices of a wider matrix
  int bn;              // weight rows of a tile; multiple of 16, <= 256 (of 64: weights M-major or quantised)
  int nstages;
  int is_bf16;
  int k_slices;     // > 0: the G groups are slices of one contraction of the whole matrices, K = their length (a multiple of 64; the
                    // copies pad the last one with zeros).  16-bit weights
  int out32;        // fp32 outputs (per >= M, os_lo = 1, rows of whole 16-byte pieces); k_slices, or up to 16 tokens (w_ints)
  int last;         // the last stage of a call: its weights do not come from the stages ahead of it
  int w_ahead;      // request weights before the kernel ahead has finished
  int round_out;    // round to nearest integer, clamp to [-128, 127] before storing
  int per;          // output offset = g*os_g + n*os_n + (m / per)*os_hi + (m % per)*os_lo
  long long os_g, os_n, os_hi, os_lo;
  void* out;
  unsigned* status;  // set to 1 when a device-side wait gave up; null where the call has no workspace
  // Optional additions in the epilogue, for outputs laid out [n][g * M + m] (per >= M, os_lo = 1): bias[g * M + m] and
  // residual[n * ldr + g * M + m], both of the 16-bit dtype.  extra_vec: both may be read in 16-byte pieces.
  const void* bias;
  const void* residual;
  long long ldr;
  int extra_vec;
  int act_out;  // applied after the bias, before the residual: 0 none, 1 GELU (erf), 2 GELU (tanh approximation)
  // Quantised weights: int8 or packed int4 (two per byte along k, even index in the low nibble, two's complement) with
  // fp16 scales [g][m][scales_per_row] (1: per weight row; K / 128: per 128 contraction indices).  Converter warps
  // widen every staged tile to the 16-bit dtype (q * scale, rounded once) in shared memory, or into TMEM, ahead of the MMA.
  int w_bits;  // 0 / 16: 16-bit weights
  int scales_per_row;
  int w_ints;  // up to 16 tokens (umma_wq.cu only): quantised weights, one scale per row, as integers with the scale on the sum in fp32; out32 possible
  const void* w_scale;
};

int launch_umma_gemm(const GemmParams& p, cudaStream_t stream);

// Sets the width of the tile and the depth of the ring.
void umma_gemm_tiling(GemmParams& p, int bn);

// Token rows that a stage copies.  (All 128 of them past the end of fewer tokens cost more than loads: 17 tokens, K = 1024 to 11008 outputs
// 9.3 us, 5.8 with a box of 32 rows.)
__host__ __device__ inline int umma_a_tile_rows(const GemmParams& p) { return p.N < 128 ? (p.N + 15) / 16 * 16 : 128; }

}  // namespace blr
