// tcgen05 / TMEM grouped GEMM with TMA stores, on single CTAs or on pairs (CG = cta_group 1 | 2, sm_100a).  Persistent, one CTA
// per SM, warp-specialised:
//   warp 0     TMA producer: per stage this CTA's 128 token rows (16 KB) and its half of the weight rows (up to 16 KB), 64 k
//              wide, 128-byte swizzled; both CTAs' loads complete on the leader's barrier
//   warp 1     (leader only) one thread issues tcgen05.mma (M = 256 over the pair, N = bn, K = 16); accumulators double-buffered
//              in TMEM (2 x bn columns of fp32, 128 rows in each CTA)
//   warps 2-17 epilogue: 32 rows x 64 columns each from TMEM through a swizzled 4 KB buffer to a TMA store, which clips
//              ragged edges
// Why pairs: a 128 x 256 tile of one CTA takes 48 KB of operands per 512 cycles of MMA, 96 B per cycle and SM, where L2 delivers 50 (all of
// them distinct) to 75; the pair shares the weight tile, 32 KB per CTA and step.  Why TMA stores: with a token row per thread, 32-byte
// stores of a warp hit 32 lines.
// All waits are bounded; a time-out sets *status and the kernel drains and frees its TMEM.
#include "umma_pair.h"

#include "ptx.cuh"
#include "tmap.h"
#include "umma_epilogue.cuh"

namespace blr {

static constexpr int kPairEpiWarps = 16;
static constexpr int kPairThreads = 32 * (2 + kPairEpiWarps);
static constexpr int kPairRows = 128;  // token rows per CTA
static constexpr int kPairK = 64;
static constexpr int kPairTileA = kPairRows * kPairK * 2;
static constexpr int kPairMaxStages = 8;
static constexpr int kPairStoreBytes = 4096;  // 32 rows x 64 columns
static constexpr int kPairStaging = kPairEpiWarps * kPairStoreBytes;

__host__ __device__ static inline int pair_stage_bytes(int bn, int cg) { return kPairTileA + bn / cg * kPairK * 2; }

template <bool BF16, bool RND, bool EX, int CG>
__global__ void __launch_bounds__(kPairThreads, 1) blr_umma_pair_kernel(const __grid_constant__ PairParams p) {
  extern __shared__ __align__(1024) uint8_t pair_raw[];
  const uint32_t base = (smem_u32(pair_raw) + 1023u) & ~1023u;
  const uint32_t stage_bytes = (uint32_t)pair_stage_bytes(p.bn, CG), NST = p.nstages;
  const uint32_t staging = base + NST * stage_bytes, bars = staging + kPairStaging;
  // full[8], empty[8], tmem_full[2], tmem_empty[2], (slot, abort flag)
  const uint32_t full0 = bars, empty0 = bars + 8 * kPairMaxStages, tfull0 = bars + 16 * kPairMaxStages, tempty0 = tfull0 + 16;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(pair_raw + (tempty0 + 16 - smem_u32(pair_raw)));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = CG == 2 ? cluster_ctarank() : 0u;
  constexpr int kRows = CG * kPairRows;  // token rows of a tile
  const int m_tiles = (p.M + p.bn - 1) / p.bn, n_tiles = (p.N + kRows - 1) / kRows;
  const int tiles = p.G * m_tiles * n_tiles, kblocks = (p.K + kPairK - 1) / kPairK;
  const int first_tile = blockIdx.x / CG, step = gridDim.x / CG;

  if (p.last) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (uint32_t s = 0; s < NST; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(tfull0 + 8 * b, 1);
      mbar_init(tempty0 + 8 * b, CG * kPairEpiWarps);  // all epilogue warps (of a pair: the leader's barrier is the one in use)
    }
    mbar_init_fence();
    tma_prefetch_desc(&p.tmW);
    tma_prefetch_desc(&p.tmA);
    tma_prefetch_desc(&p.tmO);
  }
  if (warp == 1) {
    if constexpr (CG == 2) tmem_alloc_pair(smem_u32(tmem_slot), 512);
    else tmem_alloc(smem_u32(tmem_slot), 512);
  }
  tc_fence_before();
  if constexpr (CG == 2) cluster_sync_all();  // barriers of both CTAs are ready, both have their TMEM
  else __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // everything above overlaps the tail of the kernel ahead (see umma_gemm.cu)
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (!p.last) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");  // (see umma_gemm.cu)

  // columns of a tile's MMA: the last tile of a block may be narrower (a multiple of 16 CG); the CTAs of a pair hold half of them each
  auto tile_cols = [&](int mt) { return min(p.bn, (p.M - mt * p.bn + 16 * CG - 1) / (16 * CG) * (16 * CG)); };

  if (warp == 0) {
    if (elect_one()) {
      uint32_t s = 0, parity = 0;
      bool first = true, ok = true;
      for (int tile = first_tile; tile < tiles && ok; tile += step) {
        const int nt = tile % n_tiles, gm = tile / n_tiles, mt = gm % m_tiles, g = gm / m_tiles;
        const int w0 = mt * p.bn + (rank ? tile_cols(mt) / 2 : 0), n0 = nt * kRows + (int)rank * kPairRows;
        for (int kb = 0; kb < kblocks; ++kb) {
          if (!first && !mbar_wait(empty0 + 8 * s, parity ^ 1u, abort_flag)) { ok = false; break; }
          const uint32_t dst = base + s * stage_bytes, bar = CG == 2 ? mapa_shared(full0 + 8 * s, 0) : full0 + 8 * s;
          auto tma = [&](uint32_t to, const CUtensorMap* map, int c0, int c1) {
            if constexpr (CG == 2) tma_load_3d_pair(to, map, c0, c1, g, bar);
            else tma_load_3d(to, map, c0, c1, g, bar);
          };
          if (rank == 0) mbar_arrive_expect_tx(full0 + 8 * s, CG * stage_bytes);
          tma(dst, &p.tmA, kb * kPairK, n0);
          if (p.kmajor) {
            tma(dst + kPairTileA, &p.tmW, kb * kPairK, w0);
          } else {
            // 64-wide column blocks of 64 k-rows, 8 KB each (written out: see umma_wq.cu)
            const int blocks = p.bn / (64 * CG);
            tma(dst + kPairTileA, &p.tmW, w0, kb * kPairK);
            if (blocks > 1) tma(dst + kPairTileA + 8192, &p.tmW, w0 + 64, kb * kPairK);
            if (CG == 1 && blocks > 2) tma(dst + kPairTileA + 16384, &p.tmW, w0 + 128, kb * kPairK);
            if (CG == 1 && blocks > 3) tma(dst + kPairTileA + 24576, &p.tmW, w0 + 192, kb * kPairK);
          }
          if (++s == NST) { s = 0; parity ^= 1u; first = false; }
        }
      }
    }
  } else if (warp == 1) {
    if (rank == 0 && elect_one()) {
      uint32_t s = 0, parity = 0, it = 0;
      bool ok = true;
      for (int tile = first_tile; tile < tiles && ok; tile += step, ++it) {
        const int mt = tile / n_tiles % m_tiles;
        const uint32_t buf = it & 1u, use = it >> 1;
        if (use > 0 && !mbar_wait_cluster(tempty0 + 8 * buf, (use - 1) & 1u, abort_flag)) { ok = false; break; }
        tc_fence_after();
        const uint32_t idesc = umma_idesc(BF16, false, !p.kmajor, kRows, (uint32_t)tile_cols(mt));
        const uint32_t d_tmem = tmem_base + buf * (uint32_t)p.bn;
        for (int kb = 0; kb < kblocks; ++kb) {
          if (!mbar_wait(full0 + 8 * s, parity, abort_flag)) { ok = false; break; }
          tc_fence_after();
          const uint32_t sA = base + s * stage_bytes, sW = sA + kPairTileA;
#pragma unroll
          for (int kk = 0; kk < kPairK / 16; ++kk) {
            const uint64_t wdesc = p.kmajor ? umma_smem_desc(sW + kk * 32, 16, 1024) : umma_smem_desc(sW + kk * 2048, 8192, 1024);
            const uint64_t adesc = umma_smem_desc(sA + kk * 32, 16, 1024);
            if constexpr (CG == 2) umma_f16_pair(d_tmem, adesc, wdesc, idesc, (kb | kk) != 0 ? 1u : 0u);
            else umma_f16(d_tmem, adesc, wdesc, idesc, (kb | kk) != 0 ? 1u : 0u);
          }
          if constexpr (CG == 2) umma_commit_pair(empty0 + 8 * s);  // frees the stage (in both CTAs)
          else umma_commit(empty0 + 8 * s);
          if (++s == NST) { s = 0; parity ^= 1u; }
        }
        if (ok) {
          if constexpr (CG == 2) umma_commit_pair(tfull0 + 8 * buf);
          else umma_commit(tfull0 + 8 * buf);
        }
      }
    }
  } else {
    // A warp owns TMEM lanes 32 q .. 32 q + 31 and 64 columns of every tile: one chain of TMEM load, conversion, shared-memory
    // transposition and store per warp and tile.  (The chain is latency: with 8 warps and two of them per tile a tile of
    // a short contraction took 4000 cycles.)
    const int q = warp & 3, c0 = 64 * ((warp - 2) >> 2);
    const uint32_t sbuf = staging + (uint32_t)(warp - 2) * kPairStoreBytes;
    const uint32_t row = sbuf + (uint32_t)lane * 128u, x7 = (uint32_t)lane & 7u;
    uint32_t it = 0;
    bool ok = true;
    for (int tile = first_tile; tile < tiles; tile += step, ++it) {
      const int nt = tile % n_tiles, gm = tile / n_tiles, mt = gm % m_tiles, g = gm / m_tiles;
      const uint32_t buf = it & 1u, use = it >> 1;
      const int n_row = nt * kRows + (int)rank * kPairRows + q * 32, m = mt * p.bn + c0;
      EpiRow e;
      uint32_t bias2 = 0;
      if constexpr (EX) {
        const int n = n_row + lane;
        e.n_ok = n < p.N;
        e.extra_vec = p.extra_vec;
        e.act = p.act_out;
        e.M = p.M;
        e.bias = p.bias ? static_cast<const uint16_t*>(p.bias) + (long long)g * p.M : nullptr;
        e.res = p.residual && e.n_ok ? static_cast<const uint16_t*>(p.residual) + (long long)n * p.ldr + (long long)g * p.M : nullptr;
        bias2 = epilogue_bias2(e, m + 2 * lane);
      }
      if (ok && !mbar_wait(tfull0 + 8 * buf, use & 1u, abort_flag)) ok = false;
      if (!ok) continue;
      tc_fence_after();
      const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + buf * (uint32_t)p.bn + c0;
      const int cols = n_row < p.N ? min(64, min(p.bn - c0, p.M - m)) : 0;  // columns of this warp that exist (<= 0: none)
      auto release = [&]() {  // this warp has read the accumulator
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if constexpr (CG == 2) mbar_arrive_remote_relaxed(mapa_shared(tempty0 + 8 * buf, 0));
          else mbar_arrive(tempty0 + 8 * buf);
        }
      };
      auto buffer_free = [&]() {  // the store of the tile before has left the buffer
        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        __syncwarp();
      };
      auto put16 = [&](int u, uint32_t(&d)[16]) {
        uint32_t w[8];
#pragma unroll
        for (int k = 0; k < 8; ++k)
          w[k] = gemm_pack<BF16>(gemm_round<RND>(__uint_as_float(d[2 * k])), gemm_round<RND>(__uint_as_float(d[2 * k + 1])));
        asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(row + (((2u * u) ^ x7) << 4)), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]) : "memory");
        asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(row + (((2u * u + 1u) ^ x7) << 4)), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]) : "memory");
      };
      if constexpr (EX) {
        // 16 columns at a time in a rolled loop: the activations are long, and unrolled they outgrow the instruction cache
        buffer_free();
#pragma unroll 1
        for (int u = 0; 16 * u < cols; ++u) {
          uint32_t d[16];
          tmem_ld16(taddr + 16 * u, d);
          tmem_ld_wait();
          tmem_regs_ready(d);
          epilogue_extra16<BF16, true>(e, m + 16 * u, d, bias2, 8 * u);
          put16(u, d);
        }
        release();
        if (cols <= 0) continue;
      } else {
        uint32_t d[4][16];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (16 * u < cols) tmem_ld16(taddr + 16 * u, d[u]);
        tmem_ld_wait();
#pragma unroll
        for (int u = 0; u < 4; ++u) tmem_regs_ready(d[u]);
        release();
        if (cols <= 0) continue;
        buffer_free();
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (16 * u < cols) put16(u, d[u]);
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        const int hi = m / p.per;
        tma_store_4d(&p.tmO, sbuf, m - hi * p.per, n_row, hi, g);
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      }
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    for (int i = 0; i < 200; ++i) __nanosleep(1000);  // let loads in flight land before the CTA's memory is released
    // (behind the loop: ahead of it the compiler's registers for the rest of the kernel come out slower, an encoder pass 1600 us instead of 1596)
    if (threadIdx.x == 0 && p.status) atomicExch(p.status, 1u);
  }
  if constexpr (CG == 2) cluster_sync_all();  // neither CTA leaves while the other may still use its memory or barriers
  if (warp == 1) {
    tc_fence_after();
    if constexpr (CG == 2) tmem_dealloc_pair(tmem_base, 512);
    else tmem_dealloc(tmem_base, 512);
  }
}

template <bool BF16, bool RND, bool EX, int CG>
static int launch_pair_variant(const PairParams& p, int grid, int smem, const DeviceInfo& di, cudaStream_t stream) {
  static bool configured[64] = {};
  if (!configured[di.dev]) {
    BLR_CUDA_OK(cudaFuncSetAttribute(blr_umma_pair_kernel<BF16, RND, EX, CG>, cudaFuncAttributeMaxDynamicSharedMemorySize, di.max_smem_optin));
    configured[di.dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(kPairThreads);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = CG;
  at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = CG == 2 ? 2 : 1;
  void* args[] = {const_cast<PairParams*>(&p)};
  BLR_CUDA_OK(cudaLaunchKernelExC(&cfg, (const void*)blr_umma_pair_kernel<BF16, RND, EX, CG>, args));
  return BLR_OK;
}

bool umma_pair_takes(const GemmParams& p) {
  if (p.w_bits == 8 || p.w_bits == 4 || p.k_slices > 0 || p.N <= 128) return false;
  // one TMA store per 64 columns: they are consecutive in memory, every row of them 16-byte aligned
  const bool whole = p.per >= p.M;
  if (p.os_lo != 1 || (!whole && (p.per % 64 != 0 || p.M % p.per != 0))) return false;
  return ((p.os_n | p.os_g | (whole ? 0 : p.os_hi)) & 7) == 0 && (reinterpret_cast<uintptr_t>(p.out) & 15) == 0;
}

int launch_umma_pair(const GemmParams& g, const void* W, int64_t w_row, int64_t w_grp, const void* A, int64_t ld_n, int64_t ld_g,
                     int cg, int bn, cudaStream_t stream) {
  PairParams p = {};
  p.G = g.G; p.M = g.M; p.K = g.K; p.N = g.N;
  p.kmajor = g.kmajor;
  p.last = g.last; p.status = g.status;
  DeviceInfo di;
  int rc;
  if ((rc = device_info(&di))) return rc;
  p.bn = bn;
  p.bias = g.bias; p.residual = g.residual; p.ldr = g.ldr; p.extra_vec = g.extra_vec; p.act_out = g.act_out;
  const bool whole = g.per >= g.M;
  p.per = whole ? g.M : g.per;
  const CUtensorMapDataType dt = g.is_bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  if (p.kmajor) {
    BLR_REQUIRE(p.K % 8 == 0, BLR_ERR_SHAPE, "contraction length %d must be a multiple of 8", p.K);
    const uint64_t dims[3] = {(uint64_t)p.K, (uint64_t)p.M, (uint64_t)p.G};
    const uint64_t str[2] = {(uint64_t)(w_row ? w_row : p.K) * 2, (uint64_t)(w_grp ? w_grp : (int64_t)p.M * p.K) * 2};
    const uint32_t box[3] = {64, (uint32_t)(p.bn / cg), 1};
    rc = encode_tmap_3d(&p.tmW, dt, W, dims, str, box, Swz::B128);
  } else {
    BLR_REQUIRE(p.M % 8 == 0, BLR_ERR_SHAPE, "block output width %d must be a multiple of 8", p.M);
    const uint64_t dims[3] = {(uint64_t)p.M, (uint64_t)p.K, (uint64_t)p.G};
    const uint64_t str[2] = {(uint64_t)p.M * 2, (uint64_t)p.M * p.K * 2};
    const uint32_t box[3] = {64, 64, 1};
    rc = encode_tmap_3d(&p.tmW, dt, W, dims, str, box, Swz::B128);
  }
  if (rc) return rc;
  {
    const uint64_t dims[3] = {(uint64_t)p.K, (uint64_t)p.N, (uint64_t)p.G};
    const uint64_t str[2] = {(uint64_t)ld_n * 2, (uint64_t)(p.G > 1 ? ld_g : ld_n * p.N) * 2};
    const uint32_t box[3] = {64, kPairRows, 1};
    if ((rc = encode_tmap_3d(&p.tmA, dt, A, dims, str, box, Swz::B128))) return rc;
  }
  {
    const uint64_t dims[4] = {(uint64_t)p.per, (uint64_t)p.N, (uint64_t)(whole ? 1 : p.M / p.per), (uint64_t)p.G};
    const uint64_t row = (uint64_t)g.os_n * 2;
    const uint64_t str[3] = {row, whole ? row : (uint64_t)g.os_hi * 2, p.G > 1 ? (uint64_t)g.os_g * 2 : row};
    const uint32_t box[4] = {64, 32, 1, 1};
    if ((rc = encode_tmap_4d(&p.tmO, dt, g.out, dims, str, box, Swz::B128))) return rc;
  }
  const int stage = pair_stage_bytes(p.bn, cg), fixed = 1024 + kPairStaging + 512;
  int nst = (di.max_smem_optin - fixed) / stage;
  p.nstages = nst > kPairMaxStages ? kPairMaxStages : nst;
  BLR_REQUIRE(p.nstages >= 2, BLR_ERR_UNSUPPORTED, "device offers %d bytes of shared memory", di.max_smem_optin);
  const long long tiles = (long long)p.G * ((p.M + p.bn - 1) / p.bn) * ((p.N + cg * kPairRows - 1) / (cg * kPairRows));
  const int slots = di.sm_count / cg, grid = cg * (int)(tiles < slots ? tiles : slots), smem = fixed + p.nstages * stage;
  const bool ex = p.bias || p.residual || p.act_out;
#define BLR_PAIR(BF, CGV)                                                                                \
  (g.round_out ? launch_pair_variant<BF, true, false, CGV>(p, grid, smem, di, stream)                    \
   : ex        ? launch_pair_variant<BF, false, true, CGV>(p, grid, smem, di, stream)                    \
               : launch_pair_variant<BF, false, false, CGV>(p, grid, smem, di, stream))
  if (cg == 2) return g.is_bf16 ? BLR_PAIR(true, 2) : BLR_PAIR(false, 2);
  return g.is_bf16 ? BLR_PAIR(true, 1) : BLR_PAIR(false, 1);
#undef BLR_PAIR
}

}  // namespace blr
