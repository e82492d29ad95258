// BLAST coupling above 16 tokens: z[i][n][r] = sum_j S[i][j][r] y[j][n][r] on the tensor cores (declared here, defined in
// couple.cu).  y: b planes of (N, R) 16-bit values, z: b_out such planes.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace blr {

static constexpr int kCoupleMaxBlocks = 16;

// Whether launch_couple serves the shape: up to 16 blocks per side, rows of whole 16-byte pieces.
inline bool couple_supported(int b, int b_out, int R) { return b >= 2 && b <= kCoupleMaxBlocks && b_out <= kCoupleMaxBlocks && R % 8 == 0; }

// S with element strides (s_i, s_j, s_r).  round_z: round to the nearest integer in [-128, 127].  status: set to 1 when a wait gave up.
int launch_couple(const void* y, const void* S, int64_t s_i, int64_t s_j, int64_t s_r, void* z, int b, int b_out, int64_t N, int R,
                  int is_bf16, int round_z, unsigned* status, cudaStream_t stream);

// The same on fp32 y for up to 16 tokens; S with unit rank stride and 16-byte pieces.
int launch_couple_f32(const float* y, const void* S, int64_t s_i, int64_t s_j, void* z, int b, int b_out, int64_t N, int R, int is_bf16,
                      unsigned* status, cudaStream_t stream);

}  // namespace blr
