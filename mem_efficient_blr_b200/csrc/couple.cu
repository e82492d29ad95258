// BLAST coupling above 16 tokens on mma.sync, one pass over y and z.
//
// For a fixed rank the coupling is a 16 x 16 product over the blocks.  Handing single ranks to the MMA would need the
// blocks of a token next to each other in memory; the first GEMM writes them a plane apart.  So the contraction index of
// an m16n8k16 step is (in-block j, rank r' of a pair of neighbouring ranks) and its output column (out-block i, r'), with
// the factors of the wrong rank zero: half of the products are with zeros, but a thread's A fragment is then a pair of
// ranks of one (block, token) and its accumulators a pair of ranks of one (out-block, token), both as they lie in
// memory.  A 16-byte piece of y is the A fragment of four such pairs, and four accumulator pairs are a 16-byte piece
// of z.  (A GEMM over factors expanded to groups of 16 ranks did 16 x the products on a layout that cost the first
// GEMM its wide stores, and had 8 MB of expanded factors to build: see launch_couple for the figures.)
//
// A CTA keeps one tile of 64 ranks and walks its share of the token tiles: warp w holds the factors of ranks
// 8 w .. 8 w + 7 in registers for the whole walk.  y comes in by TMA as [token][in-block][64 ranks] with 128-byte swizzle (in-blocks
// past b read as zeros), z leaves through a buffer of the same form.  Both are free of bank conflicts because the lanes
// of odd token rows take their two in-blocks (their two out-block tiles) in the opposite order.
// Bound: L2 / HBM traffic of y and z.
#include "couple.h"

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "ptx.cuh"
#include "stream_device.cuh"
#include "tmap.h"

namespace blr {

static constexpr int kCoupleWarps = 8;
static constexpr int kCoupleStages = 2;
static constexpr int kCoupleAlone = 120 * 1024;  // more shared memory than half of an SM's
static constexpr int kCoupleTileBytes = 32768;  // 64 ranks x 256 (token, block) rows

struct alignas(64) CoupleParams {
  CUtensorMap tmY;  // dims (R, b, N), box (64, blocks padded to 8 | 16, tokens per tile)
  CUtensorMap tmZ;  // the same over z
  CUtensorMap tmS;  // dims (R, b, b_out), box (64, padded, padded): S with unit rank stride (s_tma)
  const void* S;
  long long s_i, s_j, s_r;
  int b, b_out, N, R;
  int tok_groups;  // CTAs that share a rank tile
  int nstages;     // 1 when no CTA has a second tile, else kCoupleStages
  int s_tma;       // S has unit rank stride and 16-byte aligned rows
  unsigned* status;  // set to 1 when a wait gave up
};

// d = A B without a C operand (no registers to clear).
template <bool BF16>
__device__ __forceinline__ void mma_16816_first(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  if constexpr (BF16)
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
  else
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}

// The same over a contraction of 8 (half a step).
template <bool BF16>
__device__ __forceinline__ void mma_1688(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
  if constexpr (BF16)
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(b0));
  else
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(b0));
}

template <bool BF16, bool RND>
__device__ __forceinline__ uint32_t couple_pack(float a, float b) {
  if constexpr (RND) {
    a = fminf(fmaxf(rintf(a), -128.f), 127.f);
    b = fminf(fmaxf(rintf(b), -128.f), 127.f);
  }
  if constexpr (BF16) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
  } else {
    const __half2 v = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
  }
}

// KS: steps of 8 in-blocks, NT: tiles of 4 out-blocks per CTA (b <= 8: 1, 2; b <= 12: 2, 3; b <= 16: 2, 4; or 2, 2 with the out-blocks of a
// tile shared out over two CTAs).  HALF: the second half of the last step has no blocks (b <= 4; 9 .. 12).
template <bool BF16, int KS, int NT, bool RND, bool HALF>
__global__ void __launch_bounds__(kCoupleWarps * 32, 2) blast_couple_mma_kernel(const __grid_constant__ CoupleParams p) {
  extern __shared__ __align__(1024) uint8_t couple_raw[];
  constexpr int BP = 8 * KS, BO = NT == 3 ? 16 : 4 * NT;  // in-blocks / out-blocks per token row in shared memory
  constexpr int TN = kCoupleTileBytes / (128 * BP);       // tokens per tile
  constexpr int SUB = TN / 16;                            // MMA row tiles per tile
  const uint32_t base = (smem_u32(couple_raw) + 1023u) & ~1023u;
  const uint32_t outb = base + p.nstages * kCoupleTileBytes, bars = outb + kCoupleTileBytes;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(couple_raw + (bars - smem_u32(couple_raw)) + 8 * kCoupleStages + 8);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, tq = lane & 3;
  const int rt = blockIdx.x / p.tok_groups, tg = blockIdx.x - rt * p.tok_groups, r0 = rt * 64, i0 = blockIdx.y * BO;
  const int n_tiles = (p.N + TN - 1) / TN;

  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (tid == 0) {
    *abort_flag = 0;
    for (int s = 0; s <= kCoupleStages; ++s) mbar_init(bars + 8 * s, 1);
    mbar_init_fence();
    if (p.s_tma) {  // the tile's factors through the output buffer, which is free until the first tile is done
      mbar_arrive_expect_tx(bars + 8 * kCoupleStages, BO * BP * 128);
      tma_load_3d(outb, &p.tmS, r0, 0, i0, bars + 8 * kCoupleStages);
    }
    tma_prefetch_desc(&p.tmY);
    tma_prefetch_desc(&p.tmZ);
  }
  // factors of this warp's 8 ranks: sf[t][s][h] = the four of them that the lane's column keeps (rank 2 q + g % 2, q = 0 .. 3) of
  // (out-block 4 t + g / 2, in-block 8 s + 4 h + tq), two to a word; expanded to {value, 0} or {0, value} when used.
  uint32_t sf[NT][KS][2][2];
  __syncthreads();
  if (!p.s_tma) {
    // any strides (the factors of a rank next to each other in the reference's bmm layout): to the same place, neighbouring lanes on
    // neighbouring in-blocks (one or two lines per request where a lane per rank met 32: see launch_couple)
    const uint16_t* S = static_cast<const uint16_t*>(p.S);
    uint16_t* dst = reinterpret_cast<uint16_t*>(couple_raw + (outb - smem_u32(couple_raw)));
    constexpr int kRows = BO * BP, kStep = kCoupleWarps * 32 / kRows > 0 ? kCoupleWarps * 32 / kRows : 1;  // ranks per pass
    const int row = tid % kRows, j = row % BP, i = row / BP;
    const bool in = i0 + i < p.b_out && j < p.b;
    const uint16_t* src = S + (i0 + i) * p.s_i + j * p.s_j;
#pragma unroll 16
    for (int r = tid / kRows; r < 64; r += kStep) {
      const uint16_t f = in && r0 + r < p.R ? __ldg(src + (long long)(r0 + r) * p.s_r) : (uint16_t)0;
      dst[row * 64 + (((r >> 3) ^ (j & 7)) << 3) + (r & 7)] = f;
    }
  }
  const uint32_t sel0 = (g & 1) ? 0x1044u : 0x4410u, sel1 = (g & 1) ? 0x3244u : 0x4432u;
  asm volatile("griddepcontrol.wait;" ::: "memory");  // y comes from the kernel ahead; z may still be read by an earlier one
  if (tid == 0) {
    for (int s = 0; s < p.nstages; ++s) {
      const int nt = tg + s * p.tok_groups;
      if (nt < n_tiles) {
        mbar_arrive_expect_tx(bars + 8 * s, kCoupleTileBytes);
        tma_load_3d(base + s * kCoupleTileBytes, &p.tmY, r0, 0, nt * TN, bars + 8 * s);
      }
    }
  }
  bool ok = true;
  if (p.s_tma) ok = mbar_wait(bars + 8 * kCoupleStages, 0, abort_flag);
  else __syncthreads();
  {
    const uint32_t pick = (g & 1) ? 0x7632u : 0x5410u;
#pragma unroll
    for (int f = 0; f < NT * KS * 2; ++f) {
      const int t = f / (2 * KS), s = f / 2 % KS, h = f % 2;
      if (HALF && s == KS - 1 && h == 1) continue;
      const int i = 4 * t + (g >> 1), j = 8 * s + 4 * h + tq;
      uint32_t w[4];
      lds128(outb + (uint32_t)(i * BP + j) * 128 + (((uint32_t)warp ^ (j & 7u)) << 4), w[0], w[1], w[2], w[3]);
      sf[t][s][h][0] = prmt(w[0], w[1], pick);
      sf[t][s][h][1] = prmt(w[2], w[3], pick);
    }
  }
  const bool odd = (g & 1) != 0;
  int st = 0, parity = 0;
  for (int nt = tg; nt < n_tiles; nt += p.tok_groups) {
    ok = mbar_wait(bars + 8 * st, (uint32_t)parity, abort_flag) && ok;
    const uint32_t in = base + st * kCoupleTileBytes;
    uint32_t o[SUB][NT][2][4];  // [..][..][token g | g + 8][rank pair]
#pragma unroll
    for (int u = 0; u < SUB; ++u) {
      uint32_t a[KS][2][2][4];  // [s][in-block half][token g | g + 8][rank pair]
#pragma unroll
      for (int s = 0; s < KS; ++s)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint32_t row = (uint32_t)(u * 16 + h * 8 + g) * BP + 8 * s;
          if (HALF && s == KS - 1) {
            lds128(in + (row + tq) * 128 + (((uint32_t)warp ^ (uint32_t)tq) << 4), a[s][0][h][0], a[s][0][h][1], a[s][0][h][2], a[s][0][h][3]);
            continue;
          }
          const uint32_t ja = tq + (odd ? 4u : 0u), jb = ja ^ 4u;
          uint32_t va[4], vb[4];
          lds128(in + (row + ja) * 128 + (((uint32_t)warp ^ ja) << 4), va[0], va[1], va[2], va[3]);
          lds128(in + (row + jb) * 128 + (((uint32_t)warp ^ jb) << 4), vb[0], vb[1], vb[2], vb[3]);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            a[s][0][h][q] = odd ? vb[q] : va[q];
            a[s][1][h][q] = odd ? va[q] : vb[q];
          }
        }
#pragma unroll
      for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          float c[4];
#pragma unroll
          for (int s = 0; s < KS; ++s) {
            if (HALF && s == KS - 1) {
              if (s == 0) c[0] = c[1] = c[2] = c[3] = 0.f;
              mma_1688<BF16>(c, a[s][0][0][q], a[s][0][1][q], prmt(sf[t][s][0][q >> 1], 0u, q & 1 ? sel1 : sel0));
              continue;
            }
            const uint32_t b0 = prmt(sf[t][s][0][q >> 1], 0u, q & 1 ? sel1 : sel0), b1 = prmt(sf[t][s][1][q >> 1], 0u, q & 1 ? sel1 : sel0);
            if (s == 0) mma_16816_first<BF16>(c, a[s][0][0][q], a[s][0][1][q], a[s][1][0][q], a[s][1][1][q], b0, b1);
            else mma_16816<BF16>(c, a[s][0][0][q], a[s][0][1][q], a[s][1][0][q], a[s][1][1][q], b0, b1);
          }
          o[u][t][0][q] = couple_pack<BF16, RND>(c[0], c[1]);
          o[u][t][1][q] = couple_pack<BF16, RND>(c[2], c[3]);
        }
    }
    if (tid == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // the store before last has left the buffer
    __syncthreads();  // this tile is read, the output buffer is free
    if (*abort_flag) break;
    if (tid == 0) {
      const int nx = nt + p.nstages * p.tok_groups;
      if (nx < n_tiles) {
        mbar_arrive_expect_tx(bars + 8 * st, kCoupleTileBytes);
        tma_load_3d(in, &p.tmY, r0, 0, nx * TN, bars + 8 * st);
      }
    }
#pragma unroll
    for (int u = 0; u < SUB; ++u)
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int t = 0; t < NT; t += 2) {
          const uint32_t row = (uint32_t)(u * 16 + h * 8 + g) * BO;
          if (t + 1 == NT) {  // an odd tile out
            const uint32_t i = 4 * t + tq;
            asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(outb + (row + i) * 128 + (((uint32_t)warp ^ (i & 7u)) << 4)), "r"(o[u][t][h][0]), "r"(o[u][t][h][1]), "r"(o[u][t][h][2]), "r"(o[u][t][h][3]) : "memory");
            continue;
          }
          const uint32_t ia = 4 * t + tq + (odd ? 4u : 0u), ib = ia ^ 4u;
          uint32_t wa[4], wb[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            wa[q] = odd ? o[u][t + 1][h][q] : o[u][t][h][q];
            wb[q] = odd ? o[u][t][h][q] : o[u][t + 1][h][q];
          }
          asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(outb + (row + ia) * 128 + (((uint32_t)warp ^ (ia & 7u)) << 4)), "r"(wa[0]), "r"(wa[1]), "r"(wa[2]), "r"(wa[3]) : "memory");
          asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(outb + (row + ib) * 128 + (((uint32_t)warp ^ (ib & 7u)) << 4)), "r"(wb[0]), "r"(wb[1]), "r"(wb[2]), "r"(wb[3]) : "memory");
        }
    fence_proxy_async_smem();
    __syncthreads();
    if (tid == 0) {
      tma_store_3d(&p.tmZ, outb, r0, i0, nt * TN);
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    }
    if (++st == p.nstages) { st = 0; parity ^= 1; }
  }
  if (!ok) {
    atomicExch(p.status, 1u);
    for (int i = 0; i < 200; ++i) __nanosleep(1000);  // let loads in flight land before the CTA's memory is released
  }
  if (tid == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // (the end of the grid makes the stores visible)
}

template <bool BF16, int KS, int NT, bool RND, bool HALF>
static int launch_couple_impl(const CoupleParams& p, dim3 grid, int dev, cudaStream_t stream) {
  constexpr int smem_most = (kCoupleStages + 1) * kCoupleTileBytes + 64 + 1024, smem_max = smem_most > kCoupleAlone ? smem_most : kCoupleAlone;
  int smem = (p.nstages + 1) * kCoupleTileBytes + 64 + 1024;
  // No more CTAs than SMs: one to an SM, by room that it does not use.  They start while the GEMM ahead has most SMs, and up to three of them met on those that it
  // leaves free (us a call: 4096 -> 11008, R = 1024, 128 tokens 16.4 -> 15.7; 4096 -> 4096 17 / 128 tokens 11.8 / 14.7 -> 11.3 / 14.0; 768 -> 3072, R = 288,
  // 333 tokens 11.4 -> 10.8; the other way 4096 -> 11008, 17 tokens 12.4 -> 12.7).
  if ((long long)grid.x * grid.y <= sm_count() && smem < kCoupleAlone) smem = kCoupleAlone;
  static bool configured[64] = {};
  if (!configured[dev & 63]) {
    BLR_CUDA_OK(cudaFuncSetAttribute(blast_couple_mma_kernel<BF16, KS, NT, RND, HALF>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_max));
    configured[dev & 63] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(kCoupleWarps * 32);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  void* args[] = {const_cast<CoupleParams*>(&p)};
  BLR_CUDA_OK(cudaLaunchKernelExC(&cfg, (const void*)blast_couple_mma_kernel<BF16, KS, NT, RND, HALF>, args));
  return BLR_OK;
}

// ------------------------------------------------------------------------------------------ few tiles of up to 8 blocks
// The sums on the CUDA cores where latency is all there is: a thread owns 8 ranks of one token, holds the b vectors of y in registers and
// writes its share of the out-blocks; the factors of the CTA's 64 ranks lie in shared memory.  No copy engine on the way in (its boxes are
// padded to 8 blocks and walked row by row) or out.
struct CoupleFewParams {
  const void* y;
  const void* S;
  void* z;
  long long s_i, s_j, plane;  // plane = N R
  int b_out, N, R;
  int i_per;  // out-blocks per CTA
};

template <bool BF16, int B, bool RND>
__global__ void __launch_bounds__(256) blast_couple_few_kernel(const CoupleFewParams p) {
  extern __shared__ __align__(1024) uint8_t couple_raw[];
  uint4* sS = reinterpret_cast<uint4*>(couple_raw);  // [out-block of the CTA][in-block][64 ranks]
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int v = threadIdx.x & 7, r = blockIdx.x * 64 + v * 8, n = blockIdx.y * 32 + (threadIdx.x >> 3);
  const int i0 = blockIdx.z * p.i_per, i_n = min(p.i_per, p.b_out - i0);
  if (r < p.R) {
    for (int e = threadIdx.x >> 3; e < i_n * B; e += 32)
      sS[e * 8 + v] = __ldg(reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(p.S) + (i0 + e / B) * p.s_i + e % B * p.s_j + r));
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");  // y comes from the kernel ahead; z may still be read by an earlier one
  __syncthreads();
  if (r >= p.R || n >= p.N) return;
  const long long at = (long long)n * p.R + r;
  uint4 raw[B];
#pragma unroll
  for (int j = 0; j < B; ++j) raw[j] = __ldcg(reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(p.y) + j * p.plane + at));
  float yv[B][8];
#pragma unroll
  for (int j = 0; j < B; ++j) unpack8<BF16>(raw[j], yv[j]);
  for (int i = 0; i < i_n; ++i) {
    float acc[8] = {};
#pragma unroll
    for (int j = 0; j < B; ++j) {
      float f[8];
      unpack8<BF16>(sS[(i * B + j) * 8 + v], f);
#pragma unroll
      for (int k = 0; k < 8; ++k) acc[k] = fmaf(f[k], yv[j][k], acc[k]);
    }
    *reinterpret_cast<uint4*>(static_cast<uint16_t*>(p.z) + (i0 + i) * p.plane + at) =
        make_uint4(couple_pack<BF16, RND>(acc[0], acc[1]), couple_pack<BF16, RND>(acc[2], acc[3]), couple_pack<BF16, RND>(acc[4], acc[5]),
                   couple_pack<BF16, RND>(acc[6], acc[7]));
  }
}

template <bool BF16, bool RND>
static int launch_couple_few(const CoupleFewParams& p, int b, dim3 grid, cudaStream_t stream) {
  const void* kern = b == 2   ? (const void*)blast_couple_few_kernel<BF16, 2, RND>
                     : b == 3 ? (const void*)blast_couple_few_kernel<BF16, 3, RND>
                     : b == 4 ? (const void*)blast_couple_few_kernel<BF16, 4, RND>
                     : b == 6 ? (const void*)blast_couple_few_kernel<BF16, 6, RND>
                              : (const void*)blast_couple_few_kernel<BF16, 8, RND>;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(256);
  cfg.dynamicSmemBytes = (size_t)p.i_per * b * 128;
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  void* args[] = {const_cast<CoupleFewParams*>(&p)};
  BLR_CUDA_OK(cudaLaunchKernelExC(&cfg, kern, args));
  return BLR_OK;
}

// ------------------------------------------------------------------------------------------ up to 16 tokens, fp32 y
// A CTA owns 32 ranks of all tokens and four out-blocks; a thread 8 of the ranks, a token and an out-block, on the CUDA cores.  Latency is all there is: the
// factors are asked for ahead of the wait, all of the CTA's y by one copy behind it.
struct alignas(64) CoupleF32Params {
  CUtensorMap tmY;  // fp32, dims (R, N, b), box (32, N, b)
  CUtensorMap tmS;  // dims (R, b, b_out), box (32, b, 4)
  void* z;
  int b, b_out, N, R;
  unsigned* status;
};
static constexpr int kF32Threads = 256, kF32Outs = 4, kF32Tokens = 16;

template <bool BF16>
__global__ void __launch_bounds__(kF32Threads) blast_couple_f32_kernel(const __grid_constant__ CoupleF32Params p) {
  extern __shared__ __align__(1024) uint8_t couple_raw[];
  const uint32_t base = (smem_u32(couple_raw) + 1023u) & ~1023u, y_bytes = (uint32_t)p.b * p.N * 128, s_bytes = kF32Outs * p.b * 64;
  const uint32_t sS = base + y_bytes, bars = sS + s_bytes;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(couple_raw + (bars + 16 - smem_u32(couple_raw)));
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int tid = threadIdx.x, r0 = blockIdx.x * 32, i0 = blockIdx.y * kF32Outs;
  if (tid == 0) {
    *abort_flag = 0;
    mbar_init(bars, 1);
    mbar_init(bars + 8, 1);
    mbar_init_fence();
    mbar_arrive_expect_tx(bars, s_bytes);
    tma_load_3d(sS, &p.tmS, r0, 0, i0, bars);
    mbar_arrive_expect_tx(bars + 8, y_bytes);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    tma_load_3d(base, &p.tmY, r0, 0, 0, bars + 8);
  }
  __syncthreads();
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int v = tid & 3, n = (tid >> 2) & 15, i = tid >> 6, r = r0 + v * 8;
  const bool mine = r < p.R && n < p.N && i0 + i < p.b_out;
  const bool ok = mbar_wait(bars, 0, abort_flag) && mbar_wait(bars + 8, 0, abort_flag);
  if (!ok) {
    atomicExch(p.status, 1u);
    for (int k = 0; k < 200; ++k) __nanosleep(1000);  // let loads in flight land before the CTA's memory is released
    return;
  }
  if (!mine) return;
  float acc[8] = {};
#pragma unroll 4
  for (int j = 0; j < p.b; ++j) {
    const int row = j * p.N + n;
    uint32_t a[4], c[4], w[4];
    lds128(base + row * 128 + (((2 * v) ^ (row & 7)) << 4), a[0], a[1], a[2], a[3]);
    lds128(base + row * 128 + (((2 * v + 1) ^ (row & 7)) << 4), c[0], c[1], c[2], c[3]);
    lds128(sS + (i * p.b + j) * 64 + v * 16, w[0], w[1], w[2], w[3]);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float2 s = unpack16x2<BF16>(w[k]);
      acc[2 * k] = fmaf(s.x, __uint_as_float(k < 2 ? a[2 * k] : c[2 * k - 4]), acc[2 * k]);
      acc[2 * k + 1] = fmaf(s.y, __uint_as_float(k < 2 ? a[2 * k + 1] : c[2 * k - 3]), acc[2 * k + 1]);
    }
  }
  *reinterpret_cast<uint4*>(static_cast<uint16_t*>(p.z) + (i0 + i) * (long long)p.N * p.R + (long long)n * p.R + r) =
      make_uint4(couple_pack<BF16, false>(acc[0], acc[1]), couple_pack<BF16, false>(acc[2], acc[3]), couple_pack<BF16, false>(acc[4], acc[5]),
                 couple_pack<BF16, false>(acc[6], acc[7]));
}

int launch_couple_f32(const float* y, const void* S, int64_t s_i, int64_t s_j, void* z, int b, int b_out, int64_t N, int R, int is_bf16,
                      unsigned* status, cudaStream_t stream) {
  BLR_REQUIRE(N <= kF32Tokens && b <= kCoupleMaxBlocks && R % 8 == 0 && ((s_i | s_j) & 7) == 0 && (reinterpret_cast<uintptr_t>(S) & 15) == 0,
              BLR_ERR_ARG, "fp32 coupling: up to 16 tokens and blocks, factors in 16-byte pieces");
  CoupleF32Params p = {};
  p.z = z; p.b = b; p.b_out = b_out; p.N = (int)N; p.R = R; p.status = status;
  int rc;
  {
    const uint64_t dims[3] = {(uint64_t)R, (uint64_t)N, (uint64_t)b}, str[2] = {(uint64_t)R * 4, (uint64_t)N * R * 4};
    const uint32_t box[3] = {32, (uint32_t)N, (uint32_t)b};
    if ((rc = encode_tmap_3d(&p.tmY, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, y, dims, str, box, Swz::B128))) return rc;
  }
  {
    const uint64_t dims[3] = {(uint64_t)R, (uint64_t)b, (uint64_t)b_out}, str[2] = {(uint64_t)s_j * 2, (uint64_t)s_i * 2};
    const uint32_t box[3] = {32, (uint32_t)b, kF32Outs};
    if ((rc = encode_tmap_3d(&p.tmS, is_bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, S, dims, str, box, Swz::None))) return rc;
  }
  const void* kern = is_bf16 ? (const void*)blast_couple_f32_kernel<true> : (const void*)blast_couple_f32_kernel<false>;
  // More shared memory than it uses, so that its CTAs spread over the SMs: they start while the GEMM ahead has most SMs, and piled up, up to six to an SM, on
  // those that it leaves free (4096 -> 11008, R = 1024, int8, 16 tokens 15.5 us a call with what it needs, 12.7 with 80 KB, 12.4 with 120).
  static bool configured[2][64] = {};
  int dev = 0;
  BLR_CUDA_OK(cudaGetDevice(&dev));
  if (!configured[is_bf16 ? 1 : 0][dev & 63]) {
    BLR_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kCoupleAlone));
    configured[is_bf16 ? 1 : 0][dev & 63] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((R + 31) / 32), (unsigned)((b_out + kF32Outs - 1) / kF32Outs));
  cfg.blockDim = dim3(kF32Threads);
  cfg.dynamicSmemBytes = kCoupleAlone;
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  void* args[] = {&p};
  BLR_CUDA_OK(cudaLaunchKernelExC(&cfg, kern, args));
  return BLR_OK;
}

int launch_couple(const void* y, const void* S, int64_t s_i, int64_t s_j, int64_t s_r, void* z, int b, int b_out, int64_t N, int R,
                  int is_bf16, int round_z, unsigned* status, cudaStream_t stream) {
  const int ks = b <= 8 && b_out <= 8 ? 1 : 2, bp = 8 * ks, tn = kCoupleTileBytes / (128 * bp);
  const bool s_vec = s_r == 1 && (s_i & 7) == 0 && (s_j & 7) == 0 && (reinterpret_cast<uintptr_t>(S) & 15) == 0;
  // The CUDA cores for up to 8 blocks (counts with an instance) while the tiles are few: less so the more sums a tile has (us, mma | CUDA
  // cores: 8 blocks, R = 1136, 64 tokens, 36 tiles, 18.2 | 17.4; 8 blocks, 78 tiles 16.5 | 15.9, 105 tiles 19.0 | 19.5; 6 blocks, 95 tiles
  // 15.0 | 14.3; 4 blocks, 114 tiles 11.6 | 10.3, 207 tiles 13.9 | 13.8; 3 blocks, 104 tiles 13.1 | 12.2, 176 tiles 19.5 | 20.0; 2 blocks, 22
  // tiles 16.7 | 15.5, 286 tiles 14.4 | 13.7).
  const int64_t few = (int64_t)((R + 63) / 64) * ((N + 31) / 32);
  if (s_vec && (b <= 4 || b == 6 || b == 8) && b_out <= 8 && few * b <= 640) {
    int i_groups = (int)(sm_count() * 2 / few);  // two CTAs per SM, at least two out-blocks each
    if (i_groups > b_out / 2) i_groups = b_out / 2;
    if (i_groups < 1) i_groups = 1;
    const int i_per = (b_out + i_groups - 1) / i_groups;
    const CoupleFewParams q = {y, S, z, s_i, s_j, (long long)N * R, b_out, (int)N, R, i_per};
    const dim3 grid((unsigned)((R + 63) / 64), (unsigned)((N + 31) / 32), (unsigned)((b_out + i_per - 1) / i_per));
    if (round_z) return is_bf16 ? launch_couple_few<true, true>(q, b, grid, stream) : launch_couple_few<false, true>(q, b, grid, stream);
    return is_bf16 ? launch_couple_few<true, false>(q, b, grid, stream) : launch_couple_few<false, false>(q, b, grid, stream);
  }
  CoupleParams p = {};
  p.S = S;
  p.s_i = s_i; p.s_j = s_j; p.s_r = s_r;
  p.b = b; p.b_out = b_out; p.N = (int)N; p.R = R;
  p.s_tma = s_vec;
  p.status = status;
  const CUtensorMapDataType dt = is_bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  const uint64_t str[2] = {(uint64_t)N * R * 2, (uint64_t)R * 2};
  // Few tiles: the out-blocks of a tile shared out over two CTAs (half the factors to fetch and half the results to store per CTA,
  // where these latencies are all there is; longer so with factors that come 2 bytes at a time: 4096 -> 4096, R = 1024 in the bmm layout,
  // 87 tokens, 96 tiles, 20.7 -> 17.4 us).
  const int r_tiles = (R + 63) / 64, n_tiles = (int)((N + tn - 1) / tn);
  const bool halves = ks == 2 && b_out > 8 && r_tiles * n_tiles <= sm_count() / (s_vec ? 2 : 1);
  const int bo = halves ? 8 : bp;  // out-blocks per CTA
  const uint32_t box[3] = {64, (uint32_t)bp, (uint32_t)tn}, zbox[3] = {64, (uint32_t)bo, (uint32_t)tn};
  int rc;
  {
    const uint64_t dims[3] = {(uint64_t)R, (uint64_t)b, (uint64_t)N};
    if ((rc = encode_tmap_3d(&p.tmY, dt, y, dims, str, box, Swz::B128))) return rc;
  }
  {
    const uint64_t dims[3] = {(uint64_t)R, (uint64_t)b_out, (uint64_t)N};
    if ((rc = encode_tmap_3d(&p.tmZ, dt, z, dims, str, zbox, Swz::B128))) return rc;
  }
  if (p.s_tma) {
    const uint64_t dims[3] = {(uint64_t)R, (uint64_t)b, (uint64_t)b_out}, sstr[2] = {(uint64_t)s_j * 2, (uint64_t)s_i * 2};
    const uint32_t sbox[3] = {64, (uint32_t)bp, (uint32_t)bo};
    if ((rc = encode_tmap_3d(&p.tmS, dt, S, dims, sstr, sbox, Swz::B128))) return rc;
  }
  DeviceInfo di;
  if ((rc = device_info(&di))) return rc;
  int dev = 0;
  BLR_CUDA_OK(cudaGetDevice(&dev));
  // two CTAs per SM, shared out over the rank tiles; a CTA keeps its rank tile
  int groups = 2 * di.sm_count / r_tiles;
  if (groups > n_tiles) groups = n_tiles;
  if (groups < 1) groups = 1;
  p.tok_groups = groups;
  // (a smaller CTA of a small call may start beside the GEMM ahead of it and fetch its factors meanwhile)
  p.nstages = groups < n_tiles ? kCoupleStages : 1;
  const dim3 grid((unsigned)(r_tiles * groups), halves ? 2u : 1u);
  // Up to 12 (4) blocks: no products with the second half of the last step, and three tiles of out-blocks instead of four.  9 blocks, R = 384,
  // 2048 tokens 20.7 -> 19.5 us with both GEMMs, 4096 tokens 35.7 -> 33.5; 11 blocks, R = 328, 1024 tokens 16.5 -> 15.9; 4 blocks, R = 1024 1 %.  (Not
  // for out-blocks shared out over two CTAs, where latencies are all there is: 9 blocks, 333 tokens in the bmm layout 11.4 -> 12.1.)
  const bool half = b <= 8 * ks - 4 && b_out <= (ks == 1 ? 8 : 12);
#define BLR_COUPLE(BF, RND)                                                                                                                \
  (ks == 1  ? half ? launch_couple_impl<BF, 1, 2, RND, true>(p, grid, dev, stream) : launch_couple_impl<BF, 1, 2, RND, false>(p, grid, dev, stream) \
   : halves ? launch_couple_impl<BF, 2, 2, RND, false>(p, grid, dev, stream)                                                                \
   : half   ? launch_couple_impl<BF, 2, 3, RND, true>(p, grid, dev, stream) : launch_couple_impl<BF, 2, 4, RND, false>(p, grid, dev, stream))
  if (round_z) return is_bf16 ? BLR_COUPLE(true, true) : BLR_COUPLE(false, true);
  return is_bf16 ? BLR_COUPLE(true, false) : BLR_COUPLE(false, false);
#undef BLR_COUPLE
}

}  // namespace blr
