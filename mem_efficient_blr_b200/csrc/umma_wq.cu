// tcgen05 / TMEM grouped GEMM with the weights as the rows (sm_100a), on int8 / packed int4 weights or 16-bit ones.  One tile per CTA, warp-specialised:
//   warps 0, 10  TMA producers: per stage 64 k of the CTA's tokens (128-byte swizzled) and of 128 weight rows as they are stored
//   warp 1     one elected thread issues tcgen05.mma (M = 128 weight rows, N = tn tokens from shared memory, K = 16)
//   warps 2-9  a thread owns a weight row.  Quantised weights: two sets of four warps take alternate stages, widen the row's 64 weights (q * scale, rounded once to the
//              16-bit dtype) and put them into the stage's TMEM columns, where the MMA reads them (16-bit weights: from shared memory).  Then the epilogue: accumulator -> additions -> shared memory [token][row] -> TMA store
// Why this orientation: fewer tokens than a tile has rows leave no row idle, and with the tokens as rows the widened weights are an operand in shared memory, which they cross three times (written, read
// by the MMA once per 128 tokens, and for every 128 tokens again): 1024 cycles a step of 256 rows x 128 tokens where its MMAs take 512.  Here they never do, and a
// weight is widened once for up to 384 tokens.
// What bounds it: with few tokens the chain of a step's waits, some 250 cycles (widening 64 weights a thread takes 500, of which two run at once); with
// many the MMAs (tn / 2 cycles each) and shared memory, a step of 352 tokens 830 cycles.  4096 -> 11008, R = 1024, int8: last GEMM alone 17.9 us before
// at 333 tokens, whole call 32.1 -> 25.0.
// All waits are bounded; a time-out sets *status and the kernel drains and frees its TMEM.
#include "umma_wq.h"

#include "ptx.cuh"
#include "tmap.h"
#include "umma_epilogue.cuh"
#include "umma_widen.cuh"

namespace blr {

static constexpr int kWqThreads = 352, kWqRows = 128, kWqK = 64, kWqMaxStages = 8, kWqSets = 2;

// (bits = 16: the weights as they are, an operand in shared memory)
__host__ __device__ static inline int wq_stage_bytes(int tokens, int bits) { return tokens * kWqK * 2 + kWqRows * kWqK * bits / 8; }

// MODE: kWqPlain, kWqExtra (additions in the epilogue), or, for up to 16 tokens, quantised weights as the integers they are and the scale on the sum, in
// fp32: kWqSums (fp32 outputs), kWqLast and kWqLastExtra (16-bit ones, these with bias and residual).
enum { kWqPlain, kWqExtra, kWqSums, kWqLast, kWqLastExtra };
template <bool BF16, int WQ, int MODE>
__global__ void __launch_bounds__(kWqThreads, 1) blr_umma_wq_kernel(const __grid_constant__ WqParams p) {
  extern __shared__ __align__(1024) uint8_t wq_raw[];
  const uint32_t base = (smem_u32(wq_raw) + 1023u) & ~1023u;
  const int share = p.tn * p.tt;
  const uint32_t tok_bytes = (uint32_t)share * kWqK * 2, raw_bytes = kWqRows * kWqK * WQ / 8, stage_bytes = tok_bytes + raw_bytes, NST = p.nstages;
  constexpr bool kWide = WQ == 16;
  // raw_full[8], tok_full[8], a_full[8], empty[8], done, (slot, abort flag)
  const uint32_t rawf = base + NST * stage_bytes, tokf = rawf + 64, af = rawf + 128, empty = rawf + 192, done = rawf + 256;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(wq_raw + (done + 8 - smem_u32(wq_raw)));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = blockIdx.x * kWqRows, n0 = blockIdx.y * share, g = blockIdx.z;
  const int steps = (p.K + kWqK - 1) / kWqK;
  constexpr bool EX = MODE == kWqExtra || MODE == kWqLastExtra, kInts = MODE >= kWqSums;

  if (p.ahead) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (uint32_t s = 0; s < NST; ++s) {
      mbar_init(rawf + 8 * s, 1);
      mbar_init(tokf + 8 * s, 1);
      mbar_init(af + 8 * s, 4);  // the warps of a set
      mbar_init(empty + 8 * s, 1);
    }
    mbar_init(done, 1);
    mbar_init_fence();
    tma_prefetch_desc(&p.tmW);
    tma_prefetch_desc(&p.tmA);
    tma_prefetch_desc(&p.tmO);
  }
  if (warp == 1) tmem_alloc(smem_u32(tmem_slot), 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot, a_cols = tmem_base + 512 - 32 * NST;

  // (Loops with a run-time count around a copy or an MMA cost the elected thread hundreds of cycles a step: 905 with the two MMA columns as a
  // loop, 440 written out, 64 tokens.)
  if (warp == 0 || warp == 10) {
    // A last stage's weights and scales do not depend on the stages ahead of it.  A first stage's may come from a kernel before it, and so may the factors of
    // the stages behind, which start once it has waited.
    if (warp == 0 || !p.ahead) asm volatile("griddepcontrol.wait;" ::: "memory");
    if (!p.ahead) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (elect_one()) {
      const bool two = p.tt > 1;
      const int n1 = n0 + p.tn;
      const uint32_t second = p.tn * 128;
      uint32_t s = 0, parity = 1;
#pragma unroll 1
      for (int k = 0; k < steps; ++k) {
        if (k >= (int)NST && !mbar_wait(empty + 8 * s, parity, abort_flag)) break;
        const uint32_t to = base + s * stage_bytes;
        if (warp == 0) {
          mbar_arrive_expect_tx(tokf + 8 * s, tok_bytes);
          tma_load_3d(to, &p.tmA, k * kWqK, n0, g, tokf + 8 * s);
          if (two) tma_load_3d(to + second, &p.tmA, k * kWqK, n1, g, tokf + 8 * s);
        } else {
          mbar_arrive_expect_tx(rawf + 8 * s, raw_bytes);
          if constexpr (!kWide) {
            tma_load_3d(to + tok_bytes, &p.tmW, k * (kWqK * WQ / 8), m0, g, rawf + 8 * s);
          } else if (p.kmajor) {
            tma_load_3d(to + tok_bytes, &p.tmW, k * kWqK, m0, g, rawf + 8 * s);
          } else {  // outputs contiguous: two blocks of 64 of them, 64 k-rows each
            tma_load_3d(to + tok_bytes, &p.tmW, m0, k * kWqK, g, rawf + 8 * s);
            tma_load_3d(to + tok_bytes + 8192, &p.tmW, m0 + 64, k * kWqK, g, rawf + 8 * s);
          }
        }
        if (++s == NST) { s = 0; parity ^= 1u; }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (elect_one()) {
      const bool a_mn = kWide && !p.kmajor;
      const uint32_t idesc = umma_idesc(BF16, a_mn, false, kWqRows, (uint32_t)p.tn), wf = kWide ? rawf : af;
      const uint64_t w_first = umma_smem_desc(base + tok_bytes, a_mn ? 8192 : 16, 1024);
      const uint32_t w_step = a_mn ? 128 : 2;  // a descriptor's address is in units of 16 bytes
      uint32_t s = 0, parity = 0;
      bool ok = true, ready = false;  // ready: the stage's operands were seen in the step before
#pragma unroll 1
      for (int k = 0; k < steps; ++k) {
        if (!ready && (!mbar_wait(tokf + 8 * s, parity, abort_flag) || !mbar_wait(wf + 8 * s, parity, abort_flag))) { ok = false; break; }
        tc_fence_after();
        const uint32_t next = s + 1 == NST ? 0 : s + 1, next_parity = next == 0 ? parity ^ 1u : parity;
        // (asked for here, so that the answers' latency passes under this step's MMAs)
        const bool tok_next = mbar_test_wait(tokf + 8 * next, next_parity), a_next = mbar_test_wait(wf + 8 * next, next_parity);
        const uint64_t b0 = umma_smem_desc(base + s * stage_bytes, 16, 1024);
        const uint32_t a0 = a_cols + 32 * s;
        const uint64_t w0 = w_first + (uint64_t)(s * (stage_bytes >> 4));
        auto mma = [&](uint32_t d, uint64_t bdesc, int kk) {
          if constexpr (kWide) umma_f16(d, w0 + kk * w_step, bdesc + 2 * kk, idesc, (k | kk) != 0 ? 1u : 0u);
          else umma_f16_ts(d, a0 + 8 * kk, bdesc + 2 * kk, idesc, (k | kk) != 0 ? 1u : 0u);
        };
#pragma unroll
        for (int kk = 0; kk < kWqK / 16; ++kk) mma(tmem_base, b0, kk);
        if (p.tt > 1) {
#pragma unroll
          for (int kk = 0; kk < kWqK / 16; ++kk) mma(tmem_base + p.tn, b0 + (uint64_t)(p.tn * 8), kk);
        }
        umma_commit(empty + 8 * s);  // frees the stage and its TMEM columns
        ready = tok_next && a_next;
        s = next, parity = next_parity;
      }
      if (ok) umma_commit(done);
    }
    __syncwarp();
  } else {
    const int set = (warp - 2) >> 2, q = warp & 3, row = 32 * q + lane, m = m0 + row;
    const uint32_t lanes = (uint32_t)(32 * q) << 16;
    bool ok = true;
    float row_scale = 1.f;
    if constexpr (!kWide) {
      const bool grouped = p.scales_per_row > 1, in = m < p.M;
      if (!p.ahead) asm volatile("griddepcontrol.wait;" ::: "memory");
      const __half* sc = static_cast<const __half*>(p.w_scale) + ((long long)g * p.M + m) * p.scales_per_row;
      __half scale = in ? sc[0] : __float2half(0.f);
      if constexpr (kInts) row_scale = __half2float(scale);
      // (NST is a multiple of the sets: a stage is always the same set's, which has then seen its last phase complete; a parity wait cannot tell that
      // from the one before)
      uint32_t s = set, parity = 0;
      for (int k = set; k < steps && ok; k += kWqSets) {
        const __half next = grouped && in && k + kWqSets < steps ? sc[(k + kWqSets) >> 1] : scale;  // (128 indices: two steps)
        if (!mbar_wait(rawf + 8 * s, parity, abort_flag)) { ok = false; break; }
        const uint32_t raw = base + s * stage_bytes + tok_bytes + row * (kWqK * WQ / 8);
#pragma unroll
        for (int c = 0; c < 4; ++c) {  // 16 weights each, where the swizzle of 64- or 32-byte rows put them
          uint32_t o[8];
          const uint32_t at = WQ == 8 ? raw + ((c ^ ((row >> 1) & 3)) << 4) : raw + (((c >> 1) ^ ((row >> 2) & 1)) << 4) + (c & 1) * 8;
          widen16<BF16, WQ, !kInts>(at, scale, o);
          tmem_st8(a_cols + lanes + 32 * s + 8 * c, o);
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(af + 8 * s);
        scale = next;
        if ((s += kWqSets) >= NST) s -= NST, parity ^= 1u;
      }
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");  // the additions, and the output that the kernel ahead may still read
    float bias = 0.f;
    if constexpr (EX) {
      if (p.bias != nullptr && m < p.M) bias = gemm_load<BF16>(static_cast<const uint16_t*>(p.bias) + (long long)g * p.M + m);
    }
    if (ok && !mbar_wait(done, 0, abort_flag)) ok = false;
    tc_fence_after();
    if (ok) {
      // every load of the ring has been used: it holds the tile now, [token][128 rows]
      const uint32_t to = base + row * 2;
      for (int c = 16 * set; c < share && n0 + c < p.N; c += 16 * kWqSets) {
        uint32_t d[16];
        tmem_ld16(tmem_base + lanes + c, d);
        uint16_t res[16];
        if constexpr (EX) {  // (plain loads: the kernel ahead may have written the residual while this one was already running)
#pragma unroll
          for (int j = 0; j < 16; ++j)
            res[j] = p.residual != nullptr && m < p.M && n0 + c + j < p.N
                         ? static_cast<const uint16_t*>(p.residual)[(long long)(n0 + c + j) * p.ldr + (long long)g * p.M + m] : (uint16_t)0;
        }
        tmem_ld_wait();
        tmem_regs_ready(d);
#pragma unroll
        for (int j = 0; j < 16; j += 2) {
          float a = __uint_as_float(d[j]), b = __uint_as_float(d[j + 1]);
          if constexpr (kInts && !kWide) a *= row_scale, b *= row_scale;
          if constexpr (EX) {
            a += bias, b += bias;
            if constexpr (MODE == kWqExtra) {
              if (p.act_out == 1) gelu_erf2(a, b);
              else if (p.act_out == 2) a = gelu_tanh(a), b = gelu_tanh(b);
            }
            if (p.residual != nullptr) a += gemm_load<BF16>(res + j), b += gemm_load<BF16>(res + j + 1);
          }
          if constexpr (MODE == kWqSums) {
            asm volatile("st.shared.f32 [%0], %1;" ::"r"(to + (c + j) * 512 + row * 2), "f"(a) : "memory");
            asm volatile("st.shared.f32 [%0], %1;" ::"r"(to + (c + j + 1) * 512 + row * 2), "f"(b) : "memory");
            continue;
          }
          const uint32_t v = gemm_pack<BF16>(a, b);
          asm volatile("st.shared.b16 [%0], %1;" ::"r"(to + (c + j) * 256), "h"((uint16_t)v) : "memory");
          asm volatile("st.shared.b16 [%0], %1;" ::"r"(to + (c + j + 1) * 256), "h"((uint16_t)(v >> 16)) : "memory");
        }
      }
    }
    fence_proxy_async_smem();
    asm volatile("bar.sync 1, %0;" ::"n"(256) : "memory");
    if (warp == 2 && ok && elect_one()) {
      const int hi = m0 / p.per;
      for (int t = 0; t < p.tt && n0 + t * p.tn < p.N; ++t) tma_store_4d(&p.tmO, base + t * p.tn * (MODE == kWqSums ? 512 : 256), m0 - hi * p.per, n0 + t * p.tn, hi, g);
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    }
    __syncwarp();
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");  // every thread: this grid completes after its predecessor
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

template <bool BF16, int WQ, int MODE>
static int launch_wq_variant(const WqParams& p, dim3 grid, int smem, const DeviceInfo& di, cudaStream_t stream) {
  static bool configured[64] = {};
  if (!configured[di.dev]) {
    BLR_CUDA_OK(cudaFuncSetAttribute(blr_umma_wq_kernel<BF16, WQ, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, di.max_smem_optin));
    configured[di.dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(kWqThreads);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  void* args[] = {const_cast<WqParams*>(&p)};
  BLR_CUDA_OK(cudaLaunchKernelExC(&cfg, (const void*)blr_umma_wq_kernel<BF16, WQ, MODE>, args));
  return BLR_OK;
}

bool umma_wq_takes(const GemmParams& p) {
  if (p.w_ints && p.act_out) return false;
  const bool quant = p.w_bits == 8 || p.w_bits == 4;
  if (p.round_out || p.k_slices > 0 || (p.out32 && !p.w_ints) || (p.w_ints && (p.N > 16 || (quant && p.scales_per_row != 1)))) return false;
  // TMA stores of 128 consecutive outputs, every row 16-byte aligned
  const bool whole = p.per >= p.M;
  if (!whole && (p.per % kWqRows != 0 || p.M % p.per != 0 || (p.os_hi & 7) != 0)) return false;
  return p.os_lo == 1 && ((p.os_n | p.os_g) & 7) == 0 && (reinterpret_cast<uintptr_t>(p.out) & 15) == 0;
}

// By estimate, nothing fitted: a step is the MMAs, or what shared memory takes, or the widening of 64 weights a thread (500 cycles, two at once) with its waits; a
// tile on top what fills and empties it.
int umma_wq_shares(const GemmParams& p) {
  const int sms = sm_count(), bits = p.w_bits, m_tiles = (p.M + kWqRows - 1) / kWqRows, steps = (p.K + kWqK - 1) / kWqK;
  int best = 0;
  double least = 0.;
  const int fewest = (p.N + kWqMaxTokens - 1) / kWqMaxTokens;
  for (int c = fewest; c <= fewest + 7 && c <= (p.N + 15) / 16; ++c) {
    int tn, tt;
    umma_wq_share(p.N, c, &tn, &tt);
    const long long waves = ((long long)p.G * m_tiles * c + sms - 1) / sms;
    const double mma = 2. * tt * tn, smem = (2. * tn * tt * 128. + 2. * kWqRows * kWqK * bits / 8) / 128.;
    double step = mma > smem ? mma : smem;
    if (step < 380.) step = 380.;
    const double t = waves * (steps * step + 4500. + 3. * tn * tt);
    if (best == 0 || t < least) least = t, best = c;
  }
  return best;
}

int launch_umma_wq(const GemmParams& g, const void* W, int64_t w_row, int64_t w_grp, const void* A, int64_t ld_n, int64_t ld_g, int shares,
                   cudaStream_t stream) {
  WqParams p = {};
  const int bits = g.w_bits == 8 || g.w_bits == 4 ? g.w_bits : 16;
  p.G = g.G; p.M = g.M; p.K = g.K; p.N = g.N;
  p.w_scale = g.w_scale; p.scales_per_row = g.scales_per_row; p.status = g.status;
  p.ahead = g.last;
  p.bias = g.bias; p.residual = g.residual; p.ldr = g.ldr; p.act_out = g.act_out;
  DeviceInfo di;
  int rc;
  if ((rc = device_info(&di))) return rc;
  const int m_tiles = (p.M + kWqRows - 1) / kWqRows, fixed = 1024 + 512;
  umma_wq_share(p.N, shares, &p.tn, &p.tt);
  const int parts = (p.N + p.tn * p.tt - 1) / (p.tn * p.tt);
  const int stage = wq_stage_bytes(p.tn * p.tt, bits);
  int nst = (di.max_smem_optin - fixed) / stage;
  if (nst > kWqMaxStages) nst = kWqMaxStages;
  if (bits != 16 && nst > (512 - p.tn * p.tt) / 32) nst = (512 - p.tn * p.tt) / 32;
  p.nstages = bits == 16 ? nst : nst / kWqSets * kWqSets;
  BLR_REQUIRE(p.nstages >= kWqSets && p.nstages * stage >= p.tn * p.tt * kWqRows * (g.out32 ? 4 : 2) && p.tn <= 256, BLR_ERR_UNSUPPORTED,
              "device offers %d bytes of shared memory", di.max_smem_optin);
  const CUtensorMapDataType dt = g.is_bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  p.kmajor = g.kmajor;
  p.per = g.per >= g.M ? g.M : g.per;
  if (bits != 16) {
    const uint64_t row = (uint64_t)p.K * bits / 8;
    const uint64_t dims[3] = {row, (uint64_t)p.M, (uint64_t)p.G}, str[2] = {row, (uint64_t)p.M * row};
    const uint32_t box[3] = {(uint32_t)(kWqK * bits / 8), kWqRows, 1};
    rc = encode_tmap_3d(&p.tmW, CU_TENSOR_MAP_DATA_TYPE_UINT8, W, dims, str, box, bits == 8 ? Swz::B64 : Swz::B32);
  } else if (p.kmajor) {
    BLR_REQUIRE(p.K % 8 == 0, BLR_ERR_SHAPE, "contraction length %d must be a multiple of 8", p.K);
    const uint64_t dims[3] = {(uint64_t)p.K, (uint64_t)p.M, (uint64_t)p.G};
    const uint64_t str[2] = {(uint64_t)(w_row ? w_row : p.K) * 2, (uint64_t)(w_grp ? w_grp : (int64_t)p.M * p.K) * 2};
    const uint32_t box[3] = {kWqK, kWqRows, 1};
    rc = encode_tmap_3d(&p.tmW, dt, W, dims, str, box, Swz::B128);
  } else {
    BLR_REQUIRE(p.M % 8 == 0, BLR_ERR_SHAPE, "block output width %d must be a multiple of 8", p.M);
    const uint64_t dims[3] = {(uint64_t)p.M, (uint64_t)p.K, (uint64_t)p.G}, str[2] = {(uint64_t)p.M * 2, (uint64_t)p.M * p.K * 2};
    const uint32_t box[3] = {64, kWqK, 1};
    rc = encode_tmap_3d(&p.tmW, dt, W, dims, str, box, Swz::B128);
  }
  if (rc) return rc;
  {
    const uint64_t dims[3] = {(uint64_t)p.K, (uint64_t)p.N, (uint64_t)p.G};
    const uint64_t str[2] = {(uint64_t)ld_n * 2, (uint64_t)(p.G > 1 ? ld_g : ld_n * p.N) * 2};
    const uint32_t box[3] = {kWqK, (uint32_t)p.tn, 1};
    if ((rc = encode_tmap_3d(&p.tmA, dt, A, dims, str, box, Swz::B128))) return rc;
  }
  {
    const uint64_t size = g.out32 ? 4 : 2, row = (uint64_t)g.os_n * size;
    const uint64_t dims[4] = {(uint64_t)p.per, (uint64_t)p.N, (uint64_t)(p.M / p.per), (uint64_t)p.G};
    const uint64_t str[3] = {row, p.per < p.M ? (uint64_t)g.os_hi * size : row, p.G > 1 ? (uint64_t)g.os_g * size : row};
    const uint32_t box[4] = {kWqRows, (uint32_t)p.tn, 1, 1};
    if ((rc = encode_tmap_4d(&p.tmO, g.out32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : dt, g.out, dims, str, box, Swz::None))) return rc;
  }
  const dim3 grid((unsigned)m_tiles, (unsigned)parts, (unsigned)p.G);
  int smem = fixed + p.nstages * stage;
  if (smem < 120 * 1024) smem = 120 * 1024;  // one CTA per SM: a second one would only wait for TMEM, while other SMs idle
  const bool ex = p.bias || p.residual || p.act_out;
#define BLR_WQ(BF, BITS)                                                                      \
  (g.w_ints ? g.out32 ? launch_wq_variant<BF, BITS, kWqSums>(p, grid, smem, di, stream)       \
              : ex    ? launch_wq_variant<BF, BITS, kWqLastExtra>(p, grid, smem, di, stream)  \
                      : launch_wq_variant<BF, BITS, kWqLast>(p, grid, smem, di, stream)       \
   : ex     ? launch_wq_variant<BF, BITS, kWqExtra>(p, grid, smem, di, stream)                \
            : launch_wq_variant<BF, BITS, kWqPlain>(p, grid, smem, di, stream))
  if (bits == 16) {
    if (g.out32) return g.is_bf16 ? launch_wq_variant<true, 16, kWqSums>(p, grid, smem, di, stream) : launch_wq_variant<false, 16, kWqSums>(p, grid, smem, di, stream);
    if (ex && g.w_ints)
      return g.is_bf16 ? launch_wq_variant<true, 16, kWqLastExtra>(p, grid, smem, di, stream) : launch_wq_variant<false, 16, kWqLastExtra>(p, grid, smem, di, stream);
    if (ex) return g.is_bf16 ? launch_wq_variant<true, 16, kWqExtra>(p, grid, smem, di, stream) : launch_wq_variant<false, 16, kWqExtra>(p, grid, smem, di, stream);
    return g.is_bf16 ? launch_wq_variant<true, 16, kWqPlain>(p, grid, smem, di, stream) : launch_wq_variant<false, 16, kWqPlain>(p, grid, smem, di, stream);
  }
  if (g.w_bits == 8) return g.is_bf16 ? BLR_WQ(true, 8) : BLR_WQ(false, 8);
  return g.is_bf16 ? BLR_WQ(true, 4) : BLR_WQ(false, 4);
#undef BLR_WQ
}

}  // namespace blr
