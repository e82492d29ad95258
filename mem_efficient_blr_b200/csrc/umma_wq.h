// Grouped tensor-core GEMM with 128 weight rows as the rows of a tcgen05 tile and up to 384 tokens as its columns (declared here, defined in umma_wq.cu):
//     out[g][n][m] = sum_k W[g][m][k] * A[g][n][k]
// 16-bit weights, or int8 / packed int4 ones, W = q * scale.
#pragma once
#include "umma_gemm.h"

namespace blr {

struct alignas(64) WqParams {
  CUtensorMap tmW;  // stored bytes: dims (K * bits / 8, M, G) box (64 k, 128, 1); 16 bits: K-major as these, M-major dims (M, K, G) box (64, 64, 1)
  CUtensorMap tmA;  // dims (K, N, G) box (64, tn, 1)
  CUtensorMap tmO;  // output: dims (per, N, M / per, G) box (128, tn, 1, 1)
  int G, M, K, N;
  int tn, tt;  // tokens of an MMA, MMAs side by side: a CTA's share is tn * tt tokens
  int nstages, kmajor, per;
  int ahead;  // a last stage: weights and scales are requested ahead of the wait for the kernel before
  int scales_per_row;
  const void* w_scale;
  unsigned* status;  // as in GemmParams
  const void* bias;  // the additions of GemmParams
  const void* residual;
  long long ldr;
  int act_out;
};

static constexpr int kWqMaxTokens = 384;  // of a CTA
// Tokens of an MMA (tn, a multiple of 16 up to 256) and MMAs (tt) of a CTA when N tokens are cut into c shares, none beyond kWqMaxTokens.
inline void umma_wq_share(int N, int c, int* tn, int* tt) {
  const int n = (N + c - 1) / c;
  *tt = (n + 255) / 256;
  *tn = ((n + *tt - 1) / *tt + 15) / 16 * 16;
}

// Whether the kernel can store this GEMM's outputs.
bool umma_wq_takes(const GemmParams& p);
// Into how many shares the tokens of quantised weights are cut: as many as cost the fewest cycles.
int umma_wq_shares(const GemmParams& p);
// W / A as in run_gemm, `p` with everything but the tensor maps and the tiling filled in.
int launch_umma_wq(const GemmParams& p, const void* W, int64_t w_row, int64_t w_grp, const void* A, int64_t ld_n, int64_t ld_g, int shares,
                   cudaStream_t stream);

}  // namespace blr
