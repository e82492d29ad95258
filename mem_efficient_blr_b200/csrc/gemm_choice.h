// Which tensor-core GEMM kernel runs a GEMM, on tiles of how many weight rows.
#pragma once
#include "umma_gemm.h"

namespace blr {

struct GemmChoice {
  int kernel;  // 0: umma_gemm.cu; umma_pair.cu on 1: single CTAs, 2: pairs
  int bn;      // weight rows of a tile
};
// Shape, weight layout and width, output layout and additions of `p` must be set.  row_shares: into how many shares the tokens are cut where the GEMM takes
// the weights as the rows (umma_wq.cu) instead; 0: it does not.
GemmChoice gemm_choice(const GemmParams& p, int* row_shares = nullptr);

}  // namespace blr
