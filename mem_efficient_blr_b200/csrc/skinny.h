// 1..16 tokens on 16-bit factors in any layout, as two dependent launches (declared here, defined in skinny.cu):
//   first   y[plane][n][m] = sum_k V[block][m][k] x[n][k]: a CTA per 64 outputs of a plane; a plane is an in-block or, with long
//           in-blocks, a slice of its contraction
//   second  z_i = sum over planes of S_ij * y_j (or the sum alone, or Monarch's permutation) computed by the clusters of CTAs that then
//           multiply it with their rows of U_i
// Serves what the two-launch path of blast_split.cu does not take: factors with the output index contiguous, and long
// in-blocks whose front CTAs would not fit.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace blr {

enum SkinnyMode { kSkinnyCouple = 0, kSkinnySum = 1, kSkinnyMonarch = 2 };

static constexpr int kSkinnyMaxLayers = 3;  // of equal shape on one x (kSkinnyCouple)

struct alignas(64) SkinnyLayer {
  CUtensorMap tmV, tmU;
  const void* S;         // kSkinnyCouple
  const void* bias;      // (b_out * Q) or nullptr
  const void* residual;  // (N, b_out * Q), row stride ldr, or nullptr
  void* out;
  long long ldo, ldr;
};

struct alignas(64) SkinnyParams {
  SkinnyLayer layer[kSkinnyMaxLayers];
  const void* x;
  const void* x_mul;     // or nullptr: the input is silu(x) * x_mul (x_mul with x's row stride)
  void* y;               // layers x planes x N x R scratch, 16-bit or (y32) fp32
  unsigned* status;
  long long ldx, s_i, s_j, s_r;
  int layers, mode, N, R, Q, b_out;
  int b, split, Kp;      // in-blocks, slices of a block's contraction (planes = b * split), contraction indices of a slice
  int P;
  int per;               // kSkinnyMonarch: rank / b; z_l[k * per + jj] = y_k[l * per + jj]
  int round_y, round_z, interleaved;
  int y32;
  int nkb;               // first: 64-wide boxes of a slice
  int parts, cluster, tiles, nst, nstages;  // second: CTAs per out-block, of a cluster; 32-row tiles per CTA; 128-wide stages of the contraction; ring
};

// Planes of scratch y (each N x R) a call with these dimensions uses; 0: the path does not take them.
int skinny_split(int b, int P, int R);
// Fills the launch shape and the tensor maps and enqueues both kernels; V, U: one pointer per layer.  0: launched, 1: not applicable, < 0:
// error.
int launch_skinny(SkinnyParams& p, const void* const* V, int v_kmajor, const void* const* U, int u_kmajor, int is_bf16, size_t y_bytes, cudaStream_t stream);

}  // namespace blr
