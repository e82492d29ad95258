// Grouped tensor-core GEMM on int8 / packed int4 weights for more than 16 tokens (declared here, defined in umma_wq.cu):
//     out[g][n][m] = sum_k (q * scale)[g][m][k] * A[g][n][k]
// with 128 weight rows as the rows of a tcgen05 tile and up to 384 tokens as its columns.
#pragma once
#include "umma_gemm.h"

namespace blr {

struct alignas(64) WqParams {
  CUtensorMap tmW;  // stored bytes: dims (K * bits / 8, M, G) box (64 k, 128, 1)
  CUtensorMap tmA;  // dims (K, N, G) box (64, tn, 1)
  CUtensorMap tmO;  // output: dims (M, N, G) box (128, tn, 1)
  int G, M, K, N;
  int tn, tt;  // tokens of an MMA, MMAs side by side: a CTA's share is tn * tt tokens
  int nstages;
  int scales_per_row;
  const void* w_scale;
  const void* bias;  // the additions of GemmParams
  const void* residual;
  long long ldr;
  int act_out;
};

// Whether the kernel can store this GEMM's outputs.
bool umma_wq_takes(const GemmParams& p);
// W / A as in run_gemm, `p` with everything but the tensor maps and the tiling filled in.
int launch_umma_wq(const GemmParams& p, const void* W, const void* A, int64_t ld_n, int64_t ld_g, cudaStream_t stream);

}  // namespace blr
