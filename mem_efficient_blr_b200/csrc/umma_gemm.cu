// tcgen05 / TMEM grouped GEMM (sm_100a).  Persistent, one CTA per SM, warp-specialised:
//   warp 0    TMA producer: per stage up to 128 token rows (16 KB) and one tile of up to 256 weight rows, both 64 k wide,
//             128-byte swizzled
//   warp 1    MMA issuer: one elected thread issues tcgen05.mma (M = 128, N = bn, K = 16) from shared-memory
//             descriptors; accumulators are double-buffered in TMEM (2 x bn columns of fp32)
//   warps 2-9 epilogue: tcgen05.ld the accumulator (one MMA row per thread, two warps per 32 rows taking
//             alternate 64-column chunks, loads of the next chunk in flight), convert, store
// Quantised weights (WQ = 8 | 4) add
//   warps 10-17 converter: the producer stages the stored bytes of the weight tile next to the operand tiles; these
//             warps widen them (q * scale, rounded once to the 16-bit dtype) into the swizzled weight tile of the
//             stage and release it to the MMA issuer, so the quantised factors are the only copy in global memory
// All waits are bounded; a time-out sets *status and the kernel drains and frees its TMEM.
#include <stdlib.h>

#include "ptx.cuh"
#include "tmap.h"
#include "umma_epilogue.cuh"
#include "umma_gemm.h"
#include "umma_widen.cuh"

namespace blr {

static constexpr int kGemmThreads = 320;
static constexpr int kBM = 128;  // rows of the MMA (TMEM lanes): tokens
static constexpr int kBK = 64;
static constexpr int kRowTileBytes = kBM * kBK * 2;
static constexpr int kMaxStages = 8;
static constexpr int kConvWarps = 8;  // converter warps of the quantised-weight variants

// MODE 3: fp32 outputs; 2: 32-byte stores (16 consecutive outputs contiguous and aligned, no ragged tile edge), 1: 16-byte stores,
// 0: element stores.  The mode is a template parameter so that a chunk executes only its own variant.
template <bool BF16, bool RND, int MODE, bool EX, bool LANES>
__device__ __forceinline__ void epilogue_store32(const EpiRow& e, int c0, uint32_t (&rr)[2][16], uint32_t bias2, int from) {
  int hi = (e.m0 + c0) / e.per, lo = (e.m0 + c0) - hi * e.per;  // (m / per, m % per), kept incrementally
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int c = c0 + 16 * u;
    if (c >= e.cend) break;
    uint32_t(&r)[16] = rr[u];
    tmem_regs_ready(r);
    if constexpr (EX) epilogue_extra16<BF16, LANES>(e, e.m0 + c, r, bias2, from + 8 * u);
    if constexpr (MODE == 3) {
      float* dst = static_cast<float*>(e.out) + e.nbase + e.m0 + c;
#pragma unroll
      for (int h = 0; h < 4; ++h)
        if (e.n_ok && e.m0 + c + 4 * h < e.M)
          *reinterpret_cast<uint4*>(dst + 4 * h) = make_uint4(r[4 * h], r[4 * h + 1], r[4 * h + 2], r[4 * h + 3]);
    } else if constexpr (MODE > 0) {
      uint32_t w[8];
#pragma unroll
      for (int k = 0; k < 8; ++k)
        w[k] = gemm_pack<BF16>(gemm_round<RND>(__uint_as_float(r[2 * k])), gemm_round<RND>(__uint_as_float(r[2 * k + 1])));
      uint16_t* o16 = reinterpret_cast<uint16_t*>(e.out);
      if constexpr (MODE == 2) {
        // one full 32-byte sector per thread
        uint16_t* dst = o16 + e.nbase + (long long)hi * e.os_hi + lo;
        if (e.n_ok)
          asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(dst), "r"(w[0]), "r"(w[1]), "r"(w[2]),
                       "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]) : "memory");
        lo += 16;
        if (lo >= e.per) { lo -= e.per; ++hi; }
      } else {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (e.n_ok && e.m0 + c + 8 * h < e.M)
            *reinterpret_cast<uint4*>(o16 + e.nbase + (long long)hi * e.os_hi + lo) = make_uint4(w[4 * h], w[4 * h + 1], w[4 * h + 2], w[4 * h + 3]);
          lo += 8;
          if (lo >= e.per) { lo -= e.per; ++hi; }
        }
      }
    } else {
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        if (e.n_ok && e.m0 + c + j < e.M)
          gemm_store<BF16>(e.out, e.nbase + (long long)hi * e.os_hi + (long long)lo * e.os_lo, gemm_round<RND>(__uint_as_float(r[j])));
        if (++lo == e.per) { lo = 0; ++hi; }
      }
    }
  }
}

__device__ __forceinline__ void epilogue_load32(uint32_t taddr, uint32_t (&rr)[2][16]) {
#pragma unroll
  for (int u = 0; u < 2; ++u) tmem_ld16(taddr + 16 * u, rr[u]);
}

// Columns c_first, c_first + 64, ... of the tile, 32 per round; the loads of the next round are in flight while
// this one is converted and stored.  (A round always loads 32 columns: the allocation has room behind the last
// tile column.)
template <bool BF16, bool RND, int MODE, bool EX, bool LANES>
__device__ __forceinline__ void epilogue_rows(const EpiRow& e, uint32_t taddr, int c_first, uint32_t bias_lo, uint32_t bias_hi) {
  uint32_t ra[2][16], rb[2][16];
  int c0 = c_first;
  // (bias of the rounds 0 and 1 in the halves of bias_lo's lanes, 2 and 3 in bias_hi's)
  auto bias2 = [&]() { return c0 < c_first + 128 ? bias_lo : bias_hi; };
  if (c0 < e.cend) epilogue_load32(taddr + c0, ra);
  while (c0 < e.cend) {
    tmem_ld_wait();
    if (c0 + 64 < e.cend) epilogue_load32(taddr + c0 + 64, rb);
    epilogue_store32<BF16, RND, MODE, EX, LANES>(e, c0, ra, bias2(), 0);
    c0 += 64;
    if (c0 >= e.cend) break;
    tmem_ld_wait();
    if (c0 + 64 < e.cend) epilogue_load32(taddr + c0 + 64, ra);
    epilogue_store32<BF16, RND, MODE, EX, LANES>(e, c0, rb, bias2(), 16);
    c0 += 64;
  }
}

// MODE = store width of the epilogue (see epilogue_store32), RND = round the outputs to int8 steps; both are
// chosen by the host from the parameters, so that the epilogue holds exactly one variant.
// WQ = 0: 16-bit weights; 8 | 4: quantised weights widened by converter warps (K-major only).
// EX: the epilogue adds a bias and / or a residual (an instance of its own: the additions cost registers).
template <bool BF16, int MODE, bool RND, int WQ, bool EX>
__global__ void __launch_bounds__(kGemmThreads + (WQ ? 32 * kConvWarps : 0), 1)
    blr_umma_gemm_kernel(const __grid_constant__ GemmParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t w_bytes = (uint32_t)p.bn * kBK * 2;
  const uint32_t tiles_bytes = kRowTileBytes + w_bytes;  // the two operand tiles of a stage
  // quantised weights: the stored bytes of the weight tile follow them (8 * WQ bytes per row)
  const uint32_t raw_bytes = WQ ? (uint32_t)p.bn * (8u * WQ) : 0u;
  const uint32_t stage_bytes = tiles_bytes + raw_bytes;
  const uint32_t NST = p.nstages;
  // (fewer tokens than rows: only their rows are copied; what lies in the others ends in rows of the accumulator that nobody reads)
  const uint32_t a_bytes = (uint32_t)umma_a_tile_rows(p) * kBK * 2;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + (size_t)NST * stage_bytes);
  // full[8], empty[8], tmem_full[2], tmem_empty[2], (slot, abort flag), raw_full[8]
  const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + kMaxStages);
  const uint32_t tfull0 = smem_u32(bars + 2 * kMaxStages), tempty0 = smem_u32(bars + 2 * kMaxStages + 2);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kMaxStages + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const uint32_t rfull0 = smem_u32(bars + 2 * kMaxStages + 5);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // m_tiles: tiles along the weight rows; n_tiles: tiles along the tokens
  const int m_tiles = (p.M + p.bn - 1) / p.bn, n_tiles = (p.N + kBM - 1) / kBM;
  const int tiles = p.G * m_tiles * n_tiles;
  const int kblocks = (p.K + kBK - 1) / kBK;

  if (p.last) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (uint32_t s = 0; s < NST; ++s) {
      mbar_init(full0 + 8 * s, WQ ? 1 + kConvWarps : 1);  // the producer's arrival (+ one per converter warp)
      mbar_init(empty0 + 8 * s, 1);
      if constexpr (WQ != 0) mbar_init(rfull0 + 8 * s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(tfull0 + 8 * b, 1);
      mbar_init(tempty0 + 8 * b, 8);  // one arrival per epilogue warp
    }
    mbar_init_fence();
  }
  if (warp == 1) tmem_alloc(smem_u32(tmem_slot), 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // The weights do not depend on the kernel ahead: a last stage requests its first two weight tiles before the wait.  Not the whole
  // ring: where the CTA starts late, the first tokens would queue behind it.  Last stages behind a coupling only: a first stage would take
  // the memory from the call ahead of it.
  uint32_t n_ahead = 0;
  if (WQ == 0 && p.w_ahead && warp == 0 && elect_one()) {
    const int mine = blockIdx.x < tiles ? (tiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;
    n_ahead = min(min(mine * kblocks, (int)NST), 2);
    int tile = blockIdx.x, kb = 0;
    for (uint32_t s = 0; s < n_ahead; ++s) {
      const int gm = tile / n_tiles, mt = gm % m_tiles, g = gm / m_tiles;
      const uint32_t dst = smem_base + s * stage_bytes + kRowTileBytes, bar = full0 + 8 * s;
      mbar_arrive_expect_tx(bar, a_bytes + w_bytes);
      if (p.kmajor) tma_load_3d(dst, &p.tmW, kb * kBK, mt * p.bn, g, bar);
      else
        for (int blk = 0; blk < p.bn / 64; ++blk) tma_load_3d(dst + blk * 8192, &p.tmW, mt * p.bn + blk * 64, kb * kBK, g, bar);
      if (++kb == kblocks) { kb = 0; tile += gridDim.x; }
    }
  }
  // Programmatic dependent launch: everything above overlaps the tail of the previous kernel in the stream; its
  // results (this kernel's activations) and the buffers it may still be reading (this kernel's output) are
  // touched only after it has completed.  Every thread waits, so this grid completes after its predecessor.
  asm volatile("griddepcontrol.wait;" ::: "memory");
  // (a first stage: what follows may request its weights ahead of its own wait, and they may come from the kernel that this one has waited for)
  if (!p.last) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  if (warp == 0) {
    // ------------------------------------------------ producer
    if (elect_one()) {
      tma_prefetch_desc(&p.tmW);
      tma_prefetch_desc(&p.tmA);
      uint32_t s = 0, parity = 0;
      bool first = true, ok = true;
      for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
        const int nt = tile % n_tiles, gm = tile / n_tiles, mt = gm % m_tiles, g = gm / m_tiles;
        const int k0 = WQ == 0 && MODE == 3 ? g * kblocks : 0, gw = WQ == 0 && MODE == 3 ? 0 : g;  // (slices of one contraction)
        for (int kb = 0; kb < kblocks; ++kb) {
          if (!first && !mbar_wait(empty0 + 8 * s, parity ^ 1u, abort_flag)) { ok = false; break; }
          const uint32_t dst = smem_base + s * stage_bytes, bar = full0 + 8 * s;
          if (n_ahead > 0) {
            --n_ahead;  // the stage's weights are on their way
          } else if constexpr (WQ != 0) {
            // stored bytes to the converter warps; only the token tile completes `bar` by bytes
            mbar_arrive_expect_tx(rfull0 + 8 * s, raw_bytes);
            tma_load_3d(dst + tiles_bytes, &p.tmW, kb * (8 * WQ), mt * p.bn, g, rfull0 + 8 * s);
            mbar_arrive_expect_tx(bar, a_bytes);
          } else if (p.kmajor) {
            mbar_arrive_expect_tx(bar, a_bytes + w_bytes);
            tma_load_3d(dst + kRowTileBytes, &p.tmW, (k0 + kb) * kBK, mt * p.bn, gw, bar);
          } else {
            mbar_arrive_expect_tx(bar, a_bytes + w_bytes);
            // output index contiguous: 64-wide column blocks of 64 k-rows, 8 KB each
            const uint32_t w = dst + kRowTileBytes;
            const int m = mt * p.bn, k = (k0 + kb) * kBK;
            tma_load_3d(w, &p.tmW, m, k, gw, bar);
            if (p.bn > 64) tma_load_3d(w + 8192, &p.tmW, m + 64, k, gw, bar);
            if (p.bn > 128) tma_load_3d(w + 16384, &p.tmW, m + 128, k, gw, bar);
            if (p.bn > 192) tma_load_3d(w + 24576, &p.tmW, m + 192, k, gw, bar);
          }
          tma_load_3d(dst, &p.tmA, (k0 + kb) * kBK, nt * kBM, gw, bar);
          if (++s == NST) { s = 0; parity ^= 1u; first = false; }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------ MMA issuer
    if (elect_one()) {
      // (the last tile of a block multiplies only the columns it has, to 16: 688 rows are 2.7 tiles of 256)
      const uint32_t idesc_full = umma_idesc(BF16, false, !p.kmajor, kBM, (uint32_t)p.bn);
      const uint32_t idesc_last = umma_idesc(BF16, false, !p.kmajor, kBM, (uint32_t)((p.M - (m_tiles - 1) * p.bn + 15) / 16 * 16));
      uint32_t s = 0, parity = 0;
      uint32_t it = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x, ++it) {
        const uint32_t buf = it & 1u, use = it >> 1;
        // wait until the epilogue has drained this accumulator buffer (first use of each buffer is free)
        if (use > 0 && !mbar_wait(tempty0 + 8 * buf, (use - 1) & 1u, abort_flag)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + buf * (uint32_t)p.bn;
        const uint32_t idesc = tile / n_tiles % m_tiles == m_tiles - 1 ? idesc_last : idesc_full;
        for (int kb = 0; kb < kblocks; ++kb) {
          if (!mbar_wait(full0 + 8 * s, parity, abort_flag)) { ok = false; break; }
          tc_fence_after();
          const uint32_t sA = smem_base + s * stage_bytes, sW = sA + kRowTileBytes;
#pragma unroll
          for (int kk = 0; kk < kBK / 16; ++kk) {
            // weights: K-major tile advances 32 B per k16 inside the swizzle atom; M-major tile advances 16 k-rows
            const uint64_t wdesc = p.kmajor ? umma_smem_desc(sW + kk * 32, 16, 1024) : umma_smem_desc(sW + kk * 2048, 8192, 1024);
            const uint64_t adesc = umma_smem_desc(sA + kk * 32, 16, 1024);
            umma_f16(d_tmem, adesc, wdesc, idesc, (kb | kk) != 0 ? 1u : 0u);
          }
          umma_commit(empty0 + 8 * s);  // frees the stage once these MMAs have read it
          if (++s == NST) { s = 0; parity ^= 1u; }
        }
        if (ok) umma_commit(tfull0 + 8 * buf);  // accumulator complete
      }
    }
  } else if (WQ != 0 && warp >= kGemmThreads / 32) {
    // ------------------------------------------------ converter: thread = (row of a band of rows, 16 weights of the
    // 64-wide k block); a warp reads 8 rows of stored bytes contiguously and writes their 16-byte pieces to the
    // places the 128-byte swizzle gives them (piece c of row r at c ^ (r & 7)): no bank conflicts either way
    if constexpr (WQ != 0) {
      const int ct = (int)threadIdx.x - kGemmThreads, j = ct & 3, r_in = ct >> 2;
      const __half* sc = static_cast<const __half*>(p.w_scale);
      constexpr int kBand = 8 * kConvWarps, kMaxBands = 256 / kBand;  // rows per pass of all converter threads
      const int bands = p.bn / kBand;
      const bool grouped = p.scales_per_row > 1;
      __half scale[kMaxBands];
      uint32_t s = 0, parity = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
        const int gm = tile / n_tiles, mt = gm % m_tiles, g = gm / m_tiles;
        const int row0 = mt * p.bn;
        for (int kb = 0; kb < kblocks; ++kb) {
          if (kb == 0 || (grouped && (kb & 1) == 0)) {
#pragma unroll
            for (int i = 0; i < kMaxBands; ++i) {
              const int m = row0 + r_in + kBand * i;
              scale[i] = i < bands && m < p.M ? sc[((long long)g * p.M + m) * p.scales_per_row + (grouped ? kb >> 1 : 0)]
                                              : __float2half(0.f);
            }
          }
          if (!mbar_wait(rfull0 + 8 * s, parity, abort_flag)) { ok = false; break; }
          const uint32_t st = smem_base + s * stage_bytes, raw = st + tiles_bytes, dstW = st + kRowTileBytes;
#pragma unroll
          for (int i = 0; i < kMaxBands; ++i) {
            if (i < bands) {
              const int row = r_in + kBand * i;
              uint32_t o[8];
              widen16<BF16, WQ>(raw + row * (8 * WQ) + j * (2 * WQ), scale[i], o);
              const uint32_t d = dstW + row * 128, x = (uint32_t)(row & 7);
              asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(d + (((2 * j) ^ x) << 4)), "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]) : "memory");
              asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(d + (((2 * j + 1) ^ x) << 4)), "r"(o[4]), "r"(o[5]), "r"(o[6]), "r"(o[7]) : "memory");
            }
          }
          fence_proxy_async_smem();  // the MMA reads the tile through the async proxy
          __syncwarp();
          if (lane == 0) mbar_arrive(full0 + 8 * s);
          if (++s == NST) { s = 0; parity ^= 1u; }
        }
      }
    }
  } else {
    // ------------------------------------------------ epilogue: warp w reads TMEM lanes 32*(w%4)..+31; the two
    // warps of a lane quarter take alternate column chunks of the accumulator
    const int q = warp & 3, half = (warp - 2) >> 2;
    uint32_t it = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++it) {
      const int nt = tile % n_tiles, gm = tile / n_tiles, mt = gm % m_tiles, g = gm / m_tiles;
      const uint32_t buf = it & 1u, use = it >> 1;
      // (not beside the converter warps, whose launch leaves 96 registers: 4096 -> 11008 int8 with a bias, 333 tokens 34.3 -> 36.1 us)
      constexpr bool kLanes = EX && WQ == 0;
      uint32_t bias2[2] = {0, 0};
      if constexpr (kLanes) {
        EpiRow e;
        e.extra_vec = p.extra_vec, e.M = p.M;
        e.bias = p.bias ? static_cast<const uint16_t*>(p.bias) + (long long)g * p.M : nullptr;
#pragma unroll
        for (int i = 0; i < 2; ++i) bias2[i] = epilogue_bias2(e, mt * p.bn + 32 * half + 64 * (2 * i + (lane >> 4)) + 2 * (lane & 15));
      }
      if (ok && !mbar_wait(tfull0 + 8 * buf, use & 1u, abort_flag)) ok = false;
      if (!ok) continue;
      tc_fence_after();
      const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + buf * (uint32_t)p.bn;
      EpiRow e;
      e.out = p.out;
      const int n = nt * kBM + q * 32 + lane;
      e.n_ok = n < p.N;
      e.extra_vec = p.extra_vec;
      e.act = p.act_out;
      e.bias = p.bias ? static_cast<const uint16_t*>(p.bias) + (long long)g * p.M : nullptr;
      e.res = p.residual && e.n_ok ? static_cast<const uint16_t*>(p.residual) + (long long)n * p.ldr + (long long)g * p.M : nullptr;
      e.nbase = (long long)g * p.os_g + (long long)n * p.os_n;
      e.os_hi = p.os_hi, e.os_lo = p.os_lo, e.per = p.per, e.M = p.M, e.m0 = mt * p.bn;
      e.cend = nt * kBM + q * 32 < p.N ? min(p.bn, p.M - e.m0) : 0;  // (a warp without a token has nothing to read)
      epilogue_rows<BF16, RND, MODE, EX, kLanes>(e, taddr, 32 * half, bias2[0], bias2[1]);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(tempty0 + 8 * buf);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    if (threadIdx.x == 0 && p.status) atomicExch(p.status, 1u);
    for (int i = 0; i < 200; ++i) __nanosleep(1000);  // let loads in flight land before the CTA's memory is released
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

static bool gemm_quantised(const GemmParams& p) { return p.w_bits == 8 || p.w_bits == 4; }
static int gemm_stage_bytes(const GemmParams& p) {
  return kRowTileBytes + p.bn * kBK * 2 + (gemm_quantised(p) ? p.bn * 8 * p.w_bits : 0);
}

void umma_gemm_tiling(GemmParams& p, int bn) {
  p.bn = bn;
  const int nst = (232448 - 1024 - 512) / gemm_stage_bytes(p);
  p.nstages = nst > kMaxStages ? kMaxStages : nst;
}

template <bool BF16, int MODE, bool RND, int WQ = 0, bool EX = false>
static int launch_variant(const GemmParams& p, int grid, size_t smem, int dev, int max_smem, cudaStream_t stream) {
  static bool configured[64] = {};
  if (!configured[dev & 63]) {
    BLR_CUDA_OK(cudaFuncSetAttribute(blr_umma_gemm_kernel<BF16, MODE, RND, WQ, EX>, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem));
    configured[dev & 63] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kGemmThreads + (WQ ? 32 * kConvWarps : 0));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  void* args[] = {const_cast<GemmParams*>(&p)};
  BLR_CUDA_OK(cudaLaunchKernelExC(&cfg, (const void*)blr_umma_gemm_kernel<BF16, MODE, RND, WQ, EX>, args));
  return BLR_OK;
}

// No rounding variant with quantised weights or with additions in the epilogue (the rounded intermediates exist for
// 16-bit factors only, and they are never a layer's final result).
template <bool BF16, int WQ, bool EX>
static int launch_plain(const GemmParams& p, int mode, int grid, size_t smem, int dev, int max_smem, cudaStream_t stream) {
  if (mode == 2) return launch_variant<BF16, 2, false, WQ, EX>(p, grid, smem, dev, max_smem, stream);
  if (mode == 1) return launch_variant<BF16, 1, false, WQ, EX>(p, grid, smem, dev, max_smem, stream);
  return launch_variant<BF16, 0, false, WQ, EX>(p, grid, smem, dev, max_smem, stream);
}
template <bool BF16, int WQ>
static int launch_quantised(const GemmParams& p, int mode, int grid, size_t smem, int dev, int max_smem, cudaStream_t stream) {
  return (p.bias || p.residual || p.act_out) ? launch_plain<BF16, WQ, true>(p, mode, grid, smem, dev, max_smem, stream)
                                : launch_plain<BF16, WQ, false>(p, mode, grid, smem, dev, max_smem, stream);
}

template <bool BF16>
static int launch_dtype(const GemmParams& p, int mode, int grid, size_t smem, int dev, int max_smem, cudaStream_t stream) {
  if (p.w_bits == 8) return launch_quantised<BF16, 8>(p, mode, grid, smem, dev, max_smem, stream);
  if (p.w_bits == 4) return launch_quantised<BF16, 4>(p, mode, grid, smem, dev, max_smem, stream);
  if (p.bias || p.residual || p.act_out) {
    BLR_REQUIRE(!p.round_out, BLR_ERR_ARG, "bias and residual are not combined with rounded outputs");
    return launch_plain<BF16, 0, true>(p, mode, grid, smem, dev, max_smem, stream);
  }
  if (p.round_out) {
    if (mode == 2) return launch_variant<BF16, 2, true>(p, grid, smem, dev, max_smem, stream);
    if (mode == 1) return launch_variant<BF16, 1, true>(p, grid, smem, dev, max_smem, stream);
    return launch_variant<BF16, 0, true>(p, grid, smem, dev, max_smem, stream);
  }
  if (mode == 3) return launch_variant<BF16, 3, false>(p, grid, smem, dev, max_smem, stream);
  if (mode == 2) return launch_variant<BF16, 2, false>(p, grid, smem, dev, max_smem, stream);
  if (mode == 1) return launch_variant<BF16, 1, false>(p, grid, smem, dev, max_smem, stream);
  return launch_variant<BF16, 0, false>(p, grid, smem, dev, max_smem, stream);
}

int launch_umma_gemm(const GemmParams& p_in, cudaStream_t stream) {
  GemmParams p = p_in;
  DeviceInfo di;
  int rc = device_info(&di);
  if (rc != BLR_OK) return rc;
  const size_t smem = (size_t)p.nstages * gemm_stage_bytes(p) + 512 + 1024;
  if (gemm_quantised(p)) {
    BLR_REQUIRE(p.kmajor && !p.round_out && p.w_scale != nullptr && p.scales_per_row >= 1, BLR_ERR_ARG,
                "quantised weights are contraction-contiguous, scaled and not combined with rounded outputs");
    BLR_REQUIRE(p.bn % (8 * kConvWarps) == 0, BLR_ERR_ARG, "bad tile configuration for quantised weights");
    BLR_REQUIRE(p.scales_per_row == 1 || p.scales_per_row * 128 == p.K, BLR_ERR_SHAPE,
                "scales per weight row: one, or one per 128 contraction indices");
  }
  BLR_REQUIRE((int)smem <= di.max_smem_optin, BLR_ERR_UNSUPPORTED, "needs %zu bytes of shared memory, device offers %d",
              smem, di.max_smem_optin);
  BLR_REQUIRE(p.bn % 16 == 0 && p.bn >= 16 && p.bn <= 256 && p.nstages >= 2, BLR_ERR_ARG, "bad tile configuration");
  BLR_REQUIRE(p.kmajor || p.bn % 64 == 0, BLR_ERR_ARG, "bad tile configuration for this weight layout");
  int dev;
  BLR_CUDA_OK(cudaGetDevice(&dev));
  const int m_tiles = (p.M + p.bn - 1) / p.bn, n_tiles = (p.N + kBM - 1) / kBM;
  const long long tiles = (long long)p.G * m_tiles * n_tiles;
  const int grid = (int)(tiles < di.sm_count ? tiles : di.sm_count);
  // store width of the epilogue: 16-byte stores need 8 consecutive outputs contiguous
  // and aligned in memory; 32-byte stores 16 of them, 32-byte aligned, and no ragged tile edge
  const bool vec_out = p.os_lo == 1 && (p.per & 7) == 0 && (p.M & 7) == 0 && (p.os_g & 7) == 0 && (p.os_n & 7) == 0 &&
                       (p.os_hi & 7) == 0 && (reinterpret_cast<uintptr_t>(p.out) & 15) == 0;
  const bool wide_out = vec_out && (p.per & 15) == 0 && (p.M & 15) == 0 && (p.os_g & 15) == 0 && (p.os_n & 15) == 0 &&
                        (p.os_hi & 15) == 0 && (p.bn & 15) == 0 && (reinterpret_cast<uintptr_t>(p.out) & 31) == 0;
  const int mode = p.out32 ? 3 : wide_out ? 2 : vec_out ? 1 : 0;
  BLR_REQUIRE((p.out32 != 0) == (p.k_slices != 0) && (!p.out32 || (!gemm_quantised(p) && !p.round_out && !p.bias && !p.residual &&
              !p.act_out && p.per >= p.M && ((p.M | p.os_g | p.os_n) & 3) == 0 && (reinterpret_cast<uintptr_t>(p.out) & 15) == 0)),
              BLR_ERR_ARG, "slices of a contraction are plain fp32 planes");
  return p.is_bf16 ? launch_dtype<true>(p, mode, grid, smem, dev, di.max_smem_optin, stream)
                   : launch_dtype<false>(p, mode, grid, smem, dev, di.max_smem_optin, stream);
}

}  // namespace blr
