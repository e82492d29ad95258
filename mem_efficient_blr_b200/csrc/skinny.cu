// 1..16 tokens on 16-bit factors in any layout as two dependent launches (see skinny.h).
//
// Both kernels request their weights before they wait for the kernel ahead (programmatic dependent launch): the first holds its whole
// share in shared memory, the second a ring.  After the wait only activations move: x slices of a plane (not all of x), 16-bit y planes
// through L2, z through distributed shared memory inside a cluster.  Every sum has a fixed order.
// Bound: HBM for the weights; below that the chain wait -> x -> products -> y -> wait -> z -> products -> out.
#include "skinny.h"

#include <atomic>

#include "ptx.cuh"
#include "stream_device.cuh"
#include "tmap.h"

namespace blr {

static constexpr int kSkWarps = 16, kSkThreads = kSkWarps * 32, kSkBackThreads = kSkThreads + 32;  // second (+ its producer)
static constexpr int kSkFrontWarps = 8, kSkFrontThreads = kSkFrontWarps * 32, kSkSlices = kSkFrontWarps / 4, kSkIssuers = 4;
static constexpr int kSkBox = 8192;        // first: 64 outputs x 64 k; second: 32 outputs x 128 k
static constexpr int kSkMaxBoxes = 12;     // boxes of a slice: 96 KB, two CTAs per SM
static constexpr int kSkRowPad1 = 68, kSkRowPad2 = 36;  // floats per token of a partial-sum slot (64 | 32 rows, padded against conflicts)

__device__ __forceinline__ void sk_cp_async_zfill(uint32_t dst, const void* src, uint32_t bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void sk_bar(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
__device__ __forceinline__ uint4 sk_ldcg(const void* p) {
  uint4 v;
  asm volatile("ld.global.cg.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}

// Eight consecutive values of y.
template <bool BF16, bool Y32>
__device__ __forceinline__ void sk_load8(const SkinnyParams& p, long long o, float (&f)[8]) {
  if constexpr (Y32) {
    const float4 a = __ldcg(reinterpret_cast<const float4*>(static_cast<const float*>(p.y) + o)), b = __ldcg(reinterpret_cast<const float4*>(static_cast<const float*>(p.y) + o) + 1);
    f[0] = a.x, f[1] = a.y, f[2] = a.z, f[3] = a.w, f[4] = b.x, f[5] = b.y, f[6] = b.z, f[7] = b.w;
  } else {
    unpack8<BF16>(sk_ldcg(static_cast<const uint16_t*>(p.y) + o), f);
  }
}

// Shared memory of the first kernel: boxes, x [box][token][128 B] + slack for token rows past N, barriers; the partial sums overlay the
// boxes once these are read.  (With a place of their own, 11 boxes and 10 to 16 tokens left one CTA per SM: low rank 11008 -> 4096,
// R = 1488, 12 tokens 22.2 -> 19.8 us.)
struct SkFront {
  uint32_t xs, part, bars, total;
};
__host__ __device__ static inline SkFront sk_front(int N, int nkb) {
  SkFront L;
  const uint32_t np = N <= 8 ? 8 : 16;
  uint32_t o = (uint32_t)nkb * kSkBox;
  L.xs = o; o += (uint32_t)nkb * N * 128 + (np - N) * 128;
  L.part = 0;  // (at most 8704 bytes; one box and 16 tokens of x are 10240)
  L.bars = o; o += 8 * kSkMaxBoxes + 16;
  L.total = o + 1024;
  return L;
}
// ... of the second: ring, z [64-wide box][token][128 B] + slack, factors of the CTA's ranks, partial sums, barriers.
struct SkBack {
  uint32_t zs, ss, part, bars, total;
};
__host__ __device__ static inline SkBack sk_back(int N, int R, int b, int cluster, int mode, int tiles, int nst, int nstages) {
  SkBack L;
  const uint32_t np = N <= 8 ? 8 : 16, nvs = ((uint32_t)R / 8 + cluster - 1) / cluster;
  uint32_t o = (uint32_t)nstages * kSkBox;
  L.zs = o; o += (uint32_t)nst * 2 * N * 128 + 2048;
  L.ss = o; o += mode == kSkinnyCouple ? (uint32_t)b * nvs * 16 : 0u;
  L.part = o; o += (uint32_t)tiles * 8 * np * kSkRowPad2 * 4;
  L.bars = o; o += 16u * nstages + 16;
  L.total = o + 1024;
  return L;
}

template <bool BF16>
__device__ __forceinline__ void sk_mma_acc(float (&acc)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  mma_16816<BF16>(acc, a[0], a[1], a[2], a[3], b[0], b[1]);
}

// ---------------------------------------------------------------------------------------------------- first stage
template <bool BF16, int NT, bool KM>
__global__ void __launch_bounds__(kSkFrontThreads, 4) skinny_first_kernel(const __grid_constant__ SkinnyParams p) {
  extern __shared__ __align__(1024) uint8_t sk_raw[];
  const uint32_t base = (smem_u32(sk_raw) + 1023u) & ~1023u;
  uint8_t* smem = sk_raw + (base - smem_u32(sk_raw));
  constexpr int NP = NT * 8;
  const SkFront L = sk_front(p.N, p.nkb);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, N = p.N, nkb = p.nkb;
  const SkinnyLayer& ly = p.layer[blockIdx.z];
  const int plane = blockIdx.y, m0 = blockIdx.x * 64, jb = plane / p.split, koff = (plane - jb * p.split) * p.Kp;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L.bars + 8 * kSkMaxBoxes);
  const uint32_t bars = base + L.bars;
  // (four warps ask for the boxes: one thread takes some 300 cycles for each, 11008 -> 4096, R = 1488, 1 / 8 tokens 14.4 / 17.4 -> 14.1 / 17.1 us)
  if (warp < kSkIssuers && elect_one()) {
    if (warp == 0) *abort_flag = 0;
#pragma unroll 1
    for (int kb = warp; kb < nkb; kb += kSkIssuers) {
      mbar_init(bars + 8 * kb, 1);
      mbar_init_fence();
      mbar_arrive_expect_tx(bars + 8 * kb, kSkBox);
      if constexpr (KM) tma_load_3d(base + kb * kSkBox, &ly.tmV, koff + kb * 64, m0, jb, bars + 8 * kb);
      else tma_load_3d(base + kb * kSkBox, &ly.tmV, m0, koff + kb * 64, jb, bars + 8 * kb);
    }
  }
  __syncwarp();
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (warp == 0) asm volatile("griddepcontrol.wait;" ::: "memory");
  __syncthreads();
  // x of this slice: [64-wide box][token][128 B], zero past the slice (a box may reach into the next slice's weights)
  {
    const uint16_t* x = static_cast<const uint16_t*>(p.x) + (long long)jb * p.P + koff;
    const int cpr = nkb * 8;
    if (p.x_mul != nullptr) {
      const uint16_t* xm = static_cast<const uint16_t*>(p.x_mul) + (long long)jb * p.P + koff;
#pragma unroll 1
      for (int n = warp; n < N; n += kSkFrontWarps)
#pragma unroll 1
        for (int ch = lane; ch < cpr; ch += 32) {
          uint4 v = make_uint4(0, 0, 0, 0);
          if (ch * 8 < p.Kp) {
            v = sk_ldcg(x + (long long)n * p.ldx + ch * 8);
            silu_mul8<BF16>(v, sk_ldcg(xm + (long long)n * p.ldx + ch * 8));
          }
          const uint32_t d = base + L.xs + (uint32_t)((ch >> 3) * N + n) * 128u + (uint32_t)(((ch & 7) ^ (n & 7)) << 4);
          asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(d), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
        }
    } else
    for (int n = warp; n < N; n += kSkFrontWarps)
      for (int ch = lane; ch < cpr; ch += 32) {
        const bool in = ch * 8 < p.Kp;
        sk_cp_async_zfill(base + L.xs + (uint32_t)((ch >> 3) * N + n) * 128u + (uint32_t)(((ch & 7) ^ (n & 7)) << 4),
                          x + (long long)n * p.ldx + (in ? ch * 8 : 0), in ? 16u : 0u);
      }
  }
  cp_async_wait_all();
  __syncthreads();
  const int rg = warp & 3, slice = warp >> 2;  // 16 outputs; boxes slice, slice + 2, ...
  const uint32_t jm = lane >> 3, l7 = lane & 7;
  float acc[4][NT][4];
#pragma unroll
  for (int s = 0; s < 4; ++s)
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[s][n][e] = 0.f;
  bool ok = true;
#pragma unroll 1
  for (int kb = slice; kb < nkb && ok; kb += kSkSlices) {
    ok = mbar_wait(bars + 8 * kb, 0, abort_flag);
    const uint32_t box = base + kb * kSkBox, xb = base + L.xs + (uint32_t)kb * N * 128u;
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      uint32_t bf[NT][2], a[4];
      load_bfrag<NT>(xb, ks, lane, bf);
      if constexpr (KM) ldsm_x4(box + sw128(rg * 16 + l7 + (jm & 1) * 8, ks * 2 + (jm >> 1)), a[0], a[1], a[2], a[3]);
      else ldsm_x4_t(box + sw128(ks * 16 + l7 + (jm >> 1) * 8, rg * 2 + (jm & 1)), a[0], a[1], a[2], a[3]);
#pragma unroll
      for (int n = 0; n < NT; ++n) sk_mma_acc<BF16>(acc[ks][n], a, bf[n]);
    }
  }
  float* part = reinterpret_cast<float*>(smem + L.part);
  __syncthreads();  // every box is read
  {
    const int gq = lane >> 2, tq = lane & 3;
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        part[(slice * NP + n * 8 + tq * 2 + (e & 1)) * kSkRowPad1 + rg * 16 + gq + (e >> 1) * 8] = acc[0][n][e] + acc[1][n][e] + acc[2][n][e] + acc[3][n][e];
  }
  if (__syncthreads_or(ok ? 0 : 1)) {
    if (tid == 0) atomicExch(p.status, 1u);
    return;
  }
  const long long y0 = (long long)(blockIdx.z * gridDim.y + plane) * N * p.R;
#pragma unroll 1
  for (int e = tid; e < N * 32; e += kSkFrontThreads) {
    const int n = e >> 5, r = (e & 31) * 2;
    if (m0 + r >= p.R) continue;
    float s0 = 0.f, s1 = 0.f;
#pragma unroll
    for (int s = 0; s < kSkSlices; ++s) {
      const float2 v = *reinterpret_cast<const float2*>(part + (s * NP + n) * kSkRowPad1 + r);
      s0 += v.x, s1 += v.y;
    }
    if (p.round_y) s0 = round_clamp_i8(s0), s1 = round_clamp_i8(s1);
    const long long o = y0 + (long long)n * p.R + m0 + r;
    if (p.y32) *reinterpret_cast<float2*>(static_cast<float*>(p.y) + o) = make_float2(s0, s1);
    else *reinterpret_cast<uint32_t*>(static_cast<uint16_t*>(p.y) + o) = pack16x2<BF16>(s0, s1);
  }
}

// ---------------------------------------------------------------------------------------------------- second stage
template <bool BF16, int NT, bool KM, bool Y32>
__global__ void __launch_bounds__(kSkBackThreads, 1) skinny_second_kernel(const __grid_constant__ SkinnyParams p) {
  extern __shared__ __align__(1024) uint8_t sk_raw[];
  const uint32_t base = (smem_u32(sk_raw) + 1023u) & ~1023u;
  uint8_t* smem = sk_raw + (base - smem_u32(sk_raw));
  constexpr int NP = NT * 8;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, N = p.N, R = p.R, NST = p.nstages, nst = p.nst, C = p.cluster;
  const SkBack L = sk_back(N, R, p.b, C, p.mode, p.tiles, nst, NST);
  const SkinnyLayer& ly = p.layer[blockIdx.z];
  const int blk = blockIdx.y, q0 = blockIdx.x * p.tiles * 32;
  const int ntile = min(p.tiles, (p.Q - q0 + 31) / 32), total = ntile > 0 ? ntile * nst : 0;
  const uint32_t full0 = base + L.bars, empty0 = full0 + 8u * NST;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L.bars + 16 * NST);
  if (tid == 0) {
    *abort_flag = 0;
    for (int s = 0; s < NST; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 4);  // the four warps that share a stage
    }
    mbar_init_fence();
  }
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  __syncthreads();
  cluster_arrive();  // (the peers' shared memory may be written once all of them have got here)

  if (warp == kSkWarps) {
    // producer: stages of 32 outputs x 128 k, a tile's stages in order.  (Tile and stage are counted along: behind the division that took them from the stage's
    // number the refills, not HBM, bounded layers that outgrow the ring: two of 4096 -> 11008, R = 1488, 4 / 8 tokens 27.7 / 30.2 -> 24.1 / 26.6 us.  Its
    // first turn shared out over more warps delays the first kernel's weights: 4096 -> 11008, R = 1024, 1 token 11.6 -> 12.2.)
    int t = 0, c = 0;
    auto issue = [&](uint32_t s) {
      const int m = q0 + t * 32;
      const uint32_t dst = base + s * kSkBox, bar = full0 + 8 * s;
      mbar_arrive_expect_tx(bar, kSkBox);
      if constexpr (KM) {
        tma_load_3d(dst, &ly.tmU, c * 128, m, blk, bar);
        tma_load_3d(dst + 4096, &ly.tmU, c * 128 + 64, m, blk, bar);
      } else {
        tma_load_3d(dst, &ly.tmU, m, c * 128, blk, bar);
      }
      if (++c == nst) c = 0, ++t;
    };
    const int first = total < NST ? total : NST;
    if (elect_one()) {
#pragma unroll 1
      for (int q = 0; q < first; ++q) issue((uint32_t)q);
    }
    __syncwarp();
    cluster_wait();
    cluster_arrive();
    cluster_wait();
    t = first / nst, c = first - t * nst;  // (for whichever lane is elected)
    if (elect_one()) {
      RingPos rp;
      rp.first_pass = false;
#pragma unroll 1
      for (int q = first; q < total; ++q) {
        if (!mbar_wait(empty0 + 8 * rp.s, rp.use_parity, abort_flag)) break;
        issue(rp.s);
        rp.advance(NST);
      }
    }
    return;
  }
  // ---- consumers
  const uint32_t rank = cluster_ctarank();
  const int nv = R / 8, nvs = (nv + C - 1) / C, v_lo = (int)rank * nvs, v_n = max(0, min(nvs, nv - v_lo));  // this CTA's pieces of 8 ranks
  if (p.mode == kSkinnyCouple) {
    // the factors of this out-block and these ranks: [in-block][piece][8]
    const uint16_t* S = static_cast<const uint16_t*>(ly.S) + blk * p.s_i;
    const bool vec = p.s_r == 1 && ((p.s_i | p.s_j) & 7) == 0 && (reinterpret_cast<uintptr_t>(ly.S) & 15) == 0;
    for (int e = tid; e < p.b * v_n; e += kSkThreads) {
      const int j = e / v_n, v = e - j * v_n;
      const uint32_t dst = base + L.ss + (uint32_t)(j * nvs + v) * 16u;
      const uint16_t* src = S + j * p.s_j + (long long)(v_lo + v) * 8 * p.s_r;
      if (vec) {
        cp_async16(dst, src);
      } else {
        uint16_t h[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) h[k] = __ldg(src + k * p.s_r);
#pragma unroll
        for (int k = 0; k < 8; ++k) asm volatile("st.shared.u16 [%0], %1;" ::"r"(dst + 2 * k), "h"(h[k]) : "memory");
      }
    }
  }
  // z past the rank meets zero weights: it must not hold NaNs
  for (int e = tid; e < N * (nst * 16 - nv); e += kSkThreads) {
    const int n = e / (nst * 16 - nv), v = nv + e - n * (nst * 16 - nv);
    asm volatile("st.shared.v4.b32 [%0], {%1,%1,%1,%1};" ::"r"(base + L.zs + (uint32_t)((v >> 3) * N + n) * 128u + (uint32_t)(((v & 7) ^ (n & 7)) << 4)), "r"(0) : "memory");
  }
  cp_async_wait_all();
  if (warp == 0) asm volatile("griddepcontrol.wait;" ::: "memory");
  sk_bar(1, kSkThreads);
  cluster_wait();
  // ---- z of this CTA's ranks into every CTA of the cluster.  With few tokens G lanes share a piece, each a part of the planes.
  {
    const int planes = p.mode == kSkinnyMonarch ? p.split : p.b * p.split, items = N * v_n;
    int G = 1;
    while (G < 16 && items * G * 2 <= kSkThreads && G * 2 <= planes) G *= 2;
    const long long plane_sz = (long long)N * R, layer0 = (long long)blockIdx.z * planes * plane_sz;  // (several layers: coupled ones only)
    for (int e0 = 0; e0 < items * G; e0 += kSkThreads) {
      const int e = e0 + tid, it = e / G, g = e - it * G;
      const bool live = it < items;
      const int n = live ? it / v_n : 0, v = live ? v_lo + it - n * v_n : 0;
      float z[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      if (live) {
        if (p.mode == kSkinnyMonarch) {
          // position t = k * per + jj of z_l comes from row l * per + jj of block k
#pragma unroll 1
          for (int s = g; s < planes; s += G) {
            if (p.per % 8 == 0) {
              const int t = v * 8, k = t / p.per, m = blk * p.per + t - k * p.per;
              float f[8];
              sk_load8<BF16, Y32>(p, (k * p.split + s) * plane_sz + (long long)n * R + m, f);
#pragma unroll
              for (int i = 0; i < 8; ++i) z[i] += f[i];
            } else {
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                const int t = v * 8 + i, k = t / p.per, m = blk * p.per + t - k * p.per;
                const long long o = (k * p.split + s) * plane_sz + (long long)n * R + m;
                z[i] += Y32 ? __ldcg(static_cast<const float*>(p.y) + o) : load16<BF16>(p.y, o);
              }
            }
          }
        } else {
          const long long src = (long long)n * R + v * 8;
          const bool couple = p.mode == kSkinnyCouple;
          auto add = [&](int pl, const float(&f)[8]) {
            uint32_t sw[4] = {0, 0, 0, 0};
            if (couple) {
              const int j = p.split == 1 ? pl : pl / p.split;
              lds128(base + L.ss + (uint32_t)(j * nvs + v - v_lo) * 16u, sw[0], sw[1], sw[2], sw[3]);
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const float2 c = couple ? unpack16x2<BF16>(sw[k]) : make_float2(1.f, 1.f);
              z[2 * k] = fmaf(c.x, f[2 * k], z[2 * k]);
              z[2 * k + 1] = fmaf(c.y, f[2 * k + 1], z[2 * k + 1]);
            }
          };
          if constexpr (Y32) {
            const float* y = static_cast<const float*>(p.y) + layer0 + src;
#pragma unroll 1
            for (int p0 = g; p0 < planes; p0 += 4 * G) {  // four planes requested before the first is used
              float4 w[4][2];
#pragma unroll
              for (int i = 0; i < 4; ++i)
                if (p0 + i * G < planes) {
                  w[i][0] = __ldcg(reinterpret_cast<const float4*>(y + (p0 + i * G) * plane_sz));
                  w[i][1] = __ldcg(reinterpret_cast<const float4*>(y + (p0 + i * G) * plane_sz) + 1);
                }
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                if (p0 + i * G >= planes) break;
                const float f[8] = {w[i][0].x, w[i][0].y, w[i][0].z, w[i][0].w, w[i][1].x, w[i][1].y, w[i][1].z, w[i][1].w};
                add(p0 + i * G, f);
              }
            }
          } else {
            const uint16_t* y = static_cast<const uint16_t*>(p.y) + layer0 + src;
#pragma unroll 1
            for (int p0 = g; p0 < planes; p0 += 8 * G) {  // eight planes
              uint4 w[8];
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                w[i] = make_uint4(0, 0, 0, 0);
                if (p0 + i * G < planes) w[i] = sk_ldcg(y + (p0 + i * G) * plane_sz);
              }
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                if (p0 + i * G >= planes) break;
                float f[8];
                unpack8<BF16>(w[i], f);
                add(p0 + i * G, f);
              }
            }
          }
        }
      }
      for (int o = G >> 1; o > 0; o >>= 1)  // (uniform over the CTA)
#pragma unroll
        for (int i = 0; i < 8; ++i) z[i] += __shfl_xor_sync(0xffffffffu, z[i], o);
      if (live) {
        if (p.round_z) {
#pragma unroll
          for (int i = 0; i < 8; ++i) z[i] = round_clamp_i8(z[i]);
        }
        const uint4 o4 = make_uint4(pack16x2<BF16>(z[0], z[1]), pack16x2<BF16>(z[2], z[3]), pack16x2<BF16>(z[4], z[5]), pack16x2<BF16>(z[6], z[7]));
        const uint32_t dst = base + L.zs + (uint32_t)((v >> 3) * N + n) * 128u + (uint32_t)(((v & 7) ^ (n & 7)) << 4);
        for (int d = g; d < C; d += G) st_shared_cluster_v4(mapa_shared(dst, (uint32_t)d), o4);
      }
    }
  }
  cluster_arrive();
  cluster_wait();
  // ---- products: stage q belongs to warps 4 (q % 4) .. + 3, which take its two row groups and two halves of its k
  const int set = warp >> 2, rg = warp & 1, kh = (warp >> 1) & 1;
  const uint32_t jm = lane >> 3, l7 = lane & 7;
  float* part = reinterpret_cast<float*>(smem + L.part);
  bool ok = true;
  {
    const int gq = lane >> 2, tq = lane & 3;
    float acc[4][NT][4];
    int q = set;
    uint32_t s = (uint32_t)set % (uint32_t)NST, parity = ((uint32_t)set / (uint32_t)NST) & 1u;
#pragma unroll 1
    for (int t = 0; t < ntile; ++t) {
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[a][n][e] = 0.f;
#pragma unroll 1
      for (; q < (t + 1) * nst && ok; q += 4) {
        if (!mbar_wait(full0 + 8 * s, parity, abort_flag)) { ok = false; break; }
        const int c = q - t * nst;
        const uint32_t box = base + s * kSkBox, zb = base + L.zs + (uint32_t)((2 * c + kh) * N) * 128u;
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
          uint32_t bf[NT][2], a[4];
          load_bfrag<NT>(zb, ks, lane, bf);
          if constexpr (KM) ldsm_x4(box + kh * 4096 + sw128(rg * 16 + l7 + (jm & 1) * 8, ks * 2 + (jm >> 1)), a[0], a[1], a[2], a[3]);
          else ldsm_x4_t(box + sw64(kh * 64 + ks * 16 + l7 + (jm >> 1) * 8, rg * 2 + (jm & 1)), a[0], a[1], a[2], a[3]);
#pragma unroll
          for (int n = 0; n < NT; ++n) sk_mma_acc<BF16>(acc[ks][n], a, bf[n]);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(empty0 + 8 * s);
        s += 4;
        while (s >= (uint32_t)NST) s -= (uint32_t)NST, parity ^= 1u;
      }
      float* slot = part + (size_t)(t * 8 + set * 2 + kh) * NP * kSkRowPad2;
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          slot[(n * 8 + tq * 2 + (e & 1)) * kSkRowPad2 + rg * 16 + gq + (e >> 1) * 8] = acc[0][n][e] + acc[1][n][e] + acc[2][n][e] + acc[3][n][e];
    }
  }
  if (!ok) *abort_flag = 1;
  sk_bar(1, kSkThreads);
  if (*abort_flag) {
    if (tid == 0) atomicExch(p.status, 1u);
    return;
  }
  uint16_t* outp = static_cast<uint16_t*>(ly.out);
  const int pairs = ntile * 16;
#pragma unroll 1
  for (int e = tid; e < N * pairs; e += kSkThreads) {
    const int n = e / pairs, lr = (e - n * pairs) * 2, t = lr >> 5, row = lr & 31, qq = q0 + lr;
    if (qq >= p.Q) continue;
    float s0 = 0.f, s1 = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float2 v = *reinterpret_cast<const float2*>(part + ((size_t)(t * 8 + k) * NP + n) * kSkRowPad2 + row);
      s0 += v.x, s1 += v.y;
    }
    const bool two = qq + 1 < p.Q;
    if (p.interleaved) {
      const long long o = (long long)n * ly.ldo + (long long)qq * p.b_out + blk;
      store16<BF16>(ly.out, o, s0);
      if (two) store16<BF16>(ly.out, o + p.b_out, s1);
      continue;
    }
    const long long col = (long long)blk * p.Q + qq, o = (long long)n * ly.ldo + col;
    if (ly.bias != nullptr) {
      s0 += load16<BF16>(ly.bias, col);
      if (two) s1 += load16<BF16>(ly.bias, col + 1);
    }
    if (ly.residual != nullptr) {
      s0 += load16<BF16>(ly.residual, (long long)n * ly.ldr + col);
      if (two) s1 += load16<BF16>(ly.residual, (long long)n * ly.ldr + col + 1);
    }
    if (two && (o & 1) == 0) {
      *reinterpret_cast<uint32_t*>(outp + o) = pack16x2<BF16>(s0, s1);
    } else {
      store16<BF16>(ly.out, o, s0);
      if (two) store16<BF16>(ly.out, o + 1, s1);
    }
  }
}

// ---------------------------------------------------------------------------------------------------- host side
int skinny_split(int b, int P, int R) {
  const int m_tiles = (R + 63) / 64, sms = sm_count();
  int best = 0;
  for (int s = 1; s <= 64; ++s) {
    if (P % s != 0 || (P / s) % 8 != 0) continue;
    const int Kp = P / s;
    if (Kp > kSkMaxBoxes * 64) continue;
    if (best != 0 && Kp < 128) break;
    best = s;
    // enough CTAs to fill the GPU: shorter slices only add planes for the second kernel to read
    if ((long long)m_tiles * b * s >= sms) break;
  }
  return best;
}

template <bool BF16, int NT>
static int launch_skinny_impl(const SkinnyParams& p, int v_kmajor, int u_kmajor, int planes, size_t fs, size_t bs, const DeviceInfo& di, cudaStream_t stream) {
  auto first = v_kmajor ? skinny_first_kernel<BF16, NT, true> : skinny_first_kernel<BF16, NT, false>;
  auto second = u_kmajor ? (p.y32 ? skinny_second_kernel<BF16, NT, true, true> : skinny_second_kernel<BF16, NT, true, false>)
                         : (p.y32 ? skinny_second_kernel<BF16, NT, false, true> : skinny_second_kernel<BF16, NT, false, false>);
  static bool configured[8][64] = {};
  bool& done = configured[(v_kmajor ? 4 : 0) + (u_kmajor ? 2 : 0) + (p.y32 ? 1 : 0)][di.dev];
  if (!done) {
    BLR_CUDA_OK(cudaFuncSetAttribute(first, cudaFuncAttributeMaxDynamicSharedMemorySize, di.max_smem_optin));
    BLR_CUDA_OK(cudaFuncSetAttribute(second, cudaFuncAttributeMaxDynamicSharedMemorySize, di.max_smem_optin));
    done = true;
  }
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = (unsigned)p.cluster;
  at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.stream = stream;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  void* args[] = {const_cast<SkinnyParams*>(&p)};
  cfg.gridDim = dim3((unsigned)((p.R + 63) / 64), (unsigned)planes, (unsigned)p.layers);
  cfg.blockDim = dim3(kSkFrontThreads);
  cfg.dynamicSmemBytes = fs;
  BLR_CUDA_OK(cudaLaunchKernelExC(&cfg, (const void*)first, args));
  cfg.numAttrs = 2;
  cfg.gridDim = dim3((unsigned)p.parts, (unsigned)p.b_out, (unsigned)p.layers);
  cfg.blockDim = dim3(kSkBackThreads);
  cfg.dynamicSmemBytes = bs;
  BLR_CUDA_OK(cudaLaunchKernelExC(&cfg, (const void*)second, args));
  return BLR_OK;
}

// Clusters of the second kernel that are resident at once, with one CTA per SM (its launch bounds allow no second one).
static int skinny_resident(int cluster, const DeviceInfo& di) {
  if (cluster == 1) return di.sm_count;
  static std::atomic<int> cache[64][3];  // 0: not asked yet
  std::atomic<int>& slot = cache[di.dev][cluster >> 1];
  int n = slot.load(std::memory_order_relaxed);
  if (n != 0) return n;
  auto kern = skinny_second_kernel<false, 1, true, true>;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)cluster);
  cfg.blockDim = dim3(kSkBackThreads);
  cfg.dynamicSmemBytes = (size_t)di.max_smem_optin;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)cluster;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, di.max_smem_optin) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, (const void*)kern, &cfg) != cudaSuccess || n < 1) {
    (void)cudaGetLastError();
    n = di.sm_count / cluster;
  }
  slot.store(n, std::memory_order_relaxed);
  return n;
}

int launch_skinny(SkinnyParams& p, const void* const* V, int v_kmajor, const void* const* U, int u_kmajor, int is_bf16, size_t y_bytes, cudaStream_t stream) {
  if (p.layers < 1 || p.layers > kSkinnyMaxLayers || (p.layers > 1 && p.mode != kSkinnyCouple)) return 1;
  if (p.N < 1 || p.N > kStreamMaxTokens || p.R % 8 != 0 || p.P % 8 != 0 || (!u_kmajor && p.Q % 8 != 0)) return 1;
  if (((reinterpret_cast<uintptr_t>(p.x) | reinterpret_cast<uintptr_t>(p.x_mul)) & 15) != 0 || p.ldx % 8 != 0) return 1;
  p.split = skinny_split(p.b, p.P, p.R);
  if (p.split == 0) return 1;
  p.Kp = p.P / p.split;
  p.nkb = (p.Kp + 63) / 64;
  const int planes = p.b * p.split;
  if (p.mode == kSkinnyMonarch && p.split > 1) p.y32 = 1;  // (z is rounded once)
  if ((size_t)p.layers * planes * p.N * p.R * (p.y32 ? 4 : 2) > y_bytes || planes > 65535) return 1;
  DeviceInfo di;
  int rc;
  if ((rc = device_info(&di))) return rc;
  // Second kernel: clusters of 4, 2 or 1 CTAs of an out-block, all resident at once with one CTA per SM (a cluster in a second wave doubles
  // the kernel: 36 clusters of 4 where 33 fit, 1152 -> 4608, b = 9, R = 256, 4 tokens 9.8 us, 18 of them with two tiles per CTA 5.6; clusters
  // of 8, of which 15 fit, 18.2 instead of 13.4 on 11008 -> 4096).  A larger cluster shares the reading of the planes of y among more CTAs
  // but fits fewer of them, which then have more tiles: the us of a stage of weights and of a MB of planes, as measured over 260 shapes, and
  // one for smaller clusters, which fill the GPU to the last SM.  (2880 -> 4224, b = 8, R = 352, 8 tokens: two tiles and clusters of 4 6.4,
  // one and clusters of 2 8.5; 288 -> 3360, b = 12, R = 1840, 1 token: 11.2 | 9.1; three layers 4096 -> 4096, R = 1024, 16 tokens: four
  // tiles and clusters of 2 27.4, three and single CTAs 35.5.)
  const int t_all = (p.Q + 31) / 32;
  p.nst = (p.R + 127) / 128;
  // stages of weights that an SM holds beside the rest
  auto room = [&](int c, int tiles) {
    return (di.max_smem_optin - (int)sk_back(p.N, p.R, p.b, c, p.mode, tiles, p.nst, 0).total - 16 * tiles * p.nst) / kSkBox;
  };
  const double planes_mb = 1e-6 * (p.mode == kSkinnyMonarch ? p.split : planes) * p.N * p.R * (p.y32 ? 4 : 2);
  double best = -1.;
  for (int c = 4; c >= 1; c /= 2) {
    int most = skinny_resident(c, di) / (p.b_out * p.layers) * c;  // CTAs of an out-block
    if (most == 0 && c > 1) continue;
    if (most == 0) most = 1;
    const int tiles = (t_all + most - 1) / most;
    const double us = 0.2 * tiles * p.nst + (p.N > 8 ? 22. : 16.) * planes_mb / c + (c < 4 ? 1. : 0.);
    if (room(c, tiles) < 4 || (best >= 0. && us >= best)) continue;
    best = us;
    p.tiles = tiles;
    p.cluster = c;
    p.parts = ((t_all + tiles - 1) / tiles + c - 1) / c * c;
  }
  const size_t fs = sk_front(p.N, p.nkb).total;
  if (best < 0. || (int)fs > di.max_smem_optin) return 1;
  // ring: the CTA's whole share, or what an SM holds (leaving room for a first-kernel CTA of the next call instead measured 13.6 -> 14.8 us
  // on Monarch 4096 -> 11008, 10.1 -> 10.5 on BLAST 4096 -> 11008 with R = 1024, 1 token)
  const int total = p.tiles * p.nst;
  int ring = room(p.cluster, p.tiles);
  if (ring > total) ring = total < 4 ? 4 : total;
  // A ring that is used again has whole turns of the four sets of warps, so that a stage always belongs to the same set: a set that comes to
  // a stage for the first time in its second turn could take the parity of a load still on its way for that of a finished one.
  if (ring < total) ring &= ~3;
  p.nstages = ring;
  const size_t bs = sk_back(p.N, p.R, p.b, p.cluster, p.mode, p.tiles, p.nst, ring).total;
  if ((int)bs > di.max_smem_optin) return 1;
  const CUtensorMapDataType dt = is_bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  auto map = [&](CUtensorMap* m, const void* W, int kmajor, int M, int K, int G, uint32_t bm, uint32_t bk) {
    const uint64_t dims[3] = {(uint64_t)(kmajor ? K : M), (uint64_t)(kmajor ? M : K), (uint64_t)G};
    const uint64_t str[2] = {dims[0] * 2, (uint64_t)M * K * 2};
    const uint32_t box[3] = {kmajor ? 64u : bm, kmajor ? bm : bk, 1};
    return encode_tmap_3d(m, dt, W, dims, str, box, kmajor || bm == 64 ? Swz::B128 : Swz::B64);
  };
  for (int i = 0; i < p.layers; ++i) {
    if ((rc = map(&p.layer[i].tmV, V[i], v_kmajor, p.R, p.P, p.b, 64, 64))) return rc;
    if ((rc = map(&p.layer[i].tmU, U[i], u_kmajor, p.Q, p.R, p.b_out, 32, 128))) return rc;
  }
  if (is_bf16) return p.N <= 8 ? launch_skinny_impl<true, 1>(p, v_kmajor, u_kmajor, planes, fs, bs, di, stream) : launch_skinny_impl<true, 2>(p, v_kmajor, u_kmajor, planes, fs, bs, di, stream);
  return p.N <= 8 ? launch_skinny_impl<false, 1>(p, v_kmajor, u_kmajor, planes, fs, bs, di, stream) : launch_skinny_impl<false, 2>(p, v_kmajor, u_kmajor, planes, fs, bs, di, stream);
}

}  // namespace blr
