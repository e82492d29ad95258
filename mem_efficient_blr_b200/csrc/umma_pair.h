// Grouped tensor-core GEMM with TMA stores, on single CTAs or CTA pairs (declared here, defined in umma_pair.cu):
//     out[g][n][m] = sum_k W[g][m][k] * A[g][n][k]
// with the tokens as the 128 or, over a pair, 256 rows of a tcgen05 tile and up to 256 weight rows as its columns.  16-bit
// weights.
#pragma once
#include "umma_gemm.h"

namespace blr {

struct alignas(64) PairParams {
  CUtensorMap tmW;  // K-major: dims (K, M, G) box (64, bn / CTAs, 1); M-major: dims (M, K, G) box (64, 64, 1)
  CUtensorMap tmA;  // dims (K, N, G) box (64, 128, 1)
  CUtensorMap tmO;  // output: dims (per, N, M / per, G) box (64, 32, 1, 1)
  int G, M, K, N;
  int kmajor, bn, nstages, per, last;
  const void* bias;      // the additions of GemmParams
  const void* residual;
  long long ldr;
  int extra_vec, act_out;
  unsigned* status;  // as in GemmParams
};

// Whether the kernel can store this GEMM's outputs (and is worth a look: more than one tile of tokens).
bool umma_pair_takes(const GemmParams& p);
// Launches it on cg = 1 or 2 CTAs per tile of bn weight rows; W / A as in run_gemm, `p` with everything but the tensor maps and the tiling
// filled in.  bn: a multiple of 64 where a block has several tiles (a store of 64 columns belongs to one of them), else of 32; weights
// M-major: of 64 cg.
int launch_umma_pair(const GemmParams& p, const void* W, int64_t w_row, int64_t w_grp, const void* A, int64_t ld_n, int64_t ld_g,
                     int cg, int bn, cudaStream_t stream);

}  // namespace blr
