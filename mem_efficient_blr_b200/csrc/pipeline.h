// Tensor-core pipeline for more than 16 tokens, and for layers on 4 or 9 to 16 where it is ahead (declared here, defined in pipeline.cu): grouped tcgen05 GEMMs, plus
// the BLAST coupling.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace blr {

// Quantised factors of a BLAST layer (bits 8 | 4 | 16 per factor; fp16 scales; group 0 | 128).
struct BlastQuant {
  int u_bits, v_bits, group;
  const void* u_scale;
  const void* v_scale;
};

// status: set to 1 when a wait of one of the call's kernels gave up (its output is not valid then).
int pipeline_blast(const void* x, int64_t ldx, int64_t N, int dtype, const void* U, int u_layout, const void* V,
                   int v_layout, const void* S, int64_t s_i, int64_t s_j, int64_t s_r, int b, int b_out, int P, int Q, int R,
                   int act_int8, void* out, int64_t ldo, void* y16, void* z16, void* e16, unsigned* status, cudaStream_t stream,
                   const void* e_ready = nullptr, const BlastQuant* quant = nullptr, const void* bias = nullptr,
                   const void* residual = nullptr, int64_t ldr = 0, int out_act = 0);
// The kernel of one GEMM of the pipelines with 16-bit, contraction-contiguous weights (gemm_choice): outputs [n][g * M + m], or in runs of `run` that lie a
// plane apart.
int pipeline_gemm_route(int G, int M, int K, int64_t N, int run, int additions, int layout, int bits, int* tile_rows);
// Into how many shares its tokens are cut where it takes the weights as the rows of its tiles instead; 0: it does not.
int pipeline_row_shares(int G, int M, int K, int64_t N, int run, int additions, int layout, int bits);

// Up to 16 tokens: y in fp32, z in 16 bits; quantised factors (K-major, one scale per row) as integers, scaled in fp32.  y32: 4, z16: 2 bytes for b
// (b_out) N R values.  quant: null for 16-bit factors.
bool pipeline_takes_small(int b, int b_out, int R, const void* S, int64_t s_i, int64_t s_j, int64_t s_r);
int pipeline_blast_small(const void* x, int64_t ldx, int64_t N, int dtype, const void* U, int u_layout, const void* V, int v_layout, const BlastQuant* quant,
                         const void* S, int64_t s_i, int64_t s_j, int b, int b_out, int P, int Q, int R, void* out, int64_t ldo, void* y32, void* z16,
                         unsigned* status, cudaStream_t stream, const void* bias, const void* residual, int64_t ldr);
// Expanded coupling factors of the prefill pipeline: size (0: shapes whose coupling does not use them) and construction.
size_t pipeline_coupling_bytes(int b, int b_out, int R);
int pipeline_expand_coupling(const void* S, int64_t s_i, int64_t s_j, int64_t s_r, int b, int b_out, int R, int dtype, void* E,
                             cudaStream_t stream);
int pipeline_monarch(const void* x, int64_t ldx, int64_t N, int dtype, const void* w1, int w1_layout, int grouped,
                     const void* w2, int w2_layout, int b, int P, int rank, int Qs, int interleaved, void* out,
                     int64_t ldo, void* z16, void* scratch, unsigned* status, cudaStream_t stream);
int pipeline_low_rank(const void* x, int64_t ldx, int64_t N, int dtype, const void* V, int v_layout, const void* U,
                      int u_layout, int I, int R, int O, void* out, int64_t ldo, void* z16, void* parts, size_t parts_bytes, void* planes, size_t planes_bytes,
                      unsigned* status, cudaStream_t stream);
int pipeline_dense(const void* x, int64_t ldx, int64_t N, int dtype, const void* W, int w_layout, int I, int O,
                   void* out, int64_t ldo, cudaStream_t stream);

}  // namespace blr
