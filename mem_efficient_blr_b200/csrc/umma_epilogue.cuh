// Epilogue arithmetic shared by the tensor-core GEMM kernels.
#pragma once
#include "ptx.cuh"

namespace blr {

template <bool BF16>
__device__ __forceinline__ void gemm_store(void* base, long long off, float v) {
  if constexpr (BF16) reinterpret_cast<__nv_bfloat16*>(base)[off] = __float2bfloat16_rn(v);
  else reinterpret_cast<__half*>(base)[off] = __float2half_rn(v);
}
template <bool BF16>
__device__ __forceinline__ uint32_t gemm_pack(float a, float b) {
  if constexpr (BF16) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
  } else {
    const __half2 v = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
  }
}
template <bool RND>
__device__ __forceinline__ float gemm_round(float v) {
  if constexpr (RND) return fminf(fmaxf(rintf(v), -128.f), 127.f);
  else return v;
}

template <bool BF16>
__device__ __forceinline__ float2 gemm_unpack(uint32_t w) {
  if constexpr (BF16) return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w));
  else return __half22float2(*reinterpret_cast<const __half2*>(&w));
}
template <bool BF16>
__device__ __forceinline__ float gemm_load(const uint16_t* p) {
  if constexpr (BF16) return __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(p));
  else return __half2float(*reinterpret_cast<const __half*>(p));
}

// x Phi(x), Phi the normal distribution.  Both forms below are fitted here.
//   |x| < 1.1: x / 2 + x^2 R(x^2), R of six terms for (Phi(x) - 1/2) / x (2.5e-10 off in x^2 R): one rounding of the result's size, and the
//     approximate instructions' errors stay out of the range in which they would be the largest of all.
//   else: max(x, 0) - |x| Phi(-|x|), and Phi(-|x|) = exp(-x^2 / 2) P(t) with t = 1 / (1 + p |x|) and P of five terms without a constant one (the
//     form of Hastings' approximations, 9.4e-10 off in |x| Phi(-|x|)): no cancellation for negative x.
// Root mean square of the error in single precision over normal x of deviation 0.1 / 0.3 / 0.5 / 1 / 2: 1.3e-9 / 4.6e-9 / 8.6e-9 / 1.8e-8 / 3.5e-8,
// with erff 1.9e-9 / 6.4e-9 / 1.1e-8 / 2.4e-8 / 4.9e-8; the second form alone is worse than that up to a deviation of some 0.8 (5.7e-9 / 1.2e-8 /
// 1.6e-8).  Two values at a time, their products and sums in packed instructions: 15 instructions a value where erff took some 40 and bound the last GEMM
// of 768 -> 3072, R = 288 on 3152 tokens (one value at a time, 24 instructions, that layer takes 39.5 us, with these 37.5, without an activation 30.9).
struct F2 {
  unsigned long long v;
};
__device__ __forceinline__ F2 f2(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void f2_split(F2 x, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(x.v)); }
__device__ __forceinline__ F2 f2_mul(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, float c) { return f2_fma(a, b, f2(c, c)); }

__device__ __forceinline__ void gelu_erf2(float& x, float& y) {
  const float ax = fabsf(x), ay = fabsf(y);
  const F2 v = f2(x, y), a = f2(ax, ay), u = f2_mul(v, v), h = f2_mul(v, f2(0.5f, 0.5f));
  F2 r = f2_fma(u, f2(-7.059720701363403e-06f, -7.059720701363403e-06f), 0.00011174543033121154f);
  r = f2_fma(r, u, -0.0011844459222629666f);
  r = f2_fma(r, u, 0.009972406551241875f);
  r = f2_fma(r, u, -0.06649016588926315f);
  r = f2_fma(r, u, 0.3989422619342804f);
  float tx, ty, ex, ey;
  f2_split(f2_fma(a, f2(0.3642290234565735f, 0.3642290234565735f), 1.f), tx, ty);
  f2_split(f2_mul(u, f2(-0.72134752f, -0.72134752f)), ex, ey);
  asm("rcp.approx.ftz.f32 %0, %0;" : "+f"(tx));
  asm("rcp.approx.ftz.f32 %0, %0;" : "+f"(ty));
  asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(ex));
  asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(ey));
  const F2 t = f2(tx, ty);
  F2 s = f2_fma(t, f2(-0.1040828600525856f, -0.1040828600525856f), 0.2556341886520386f);
  s = f2_fma(s, t, 0.03702527657151222f);
  s = f2_fma(s, t, 0.16834469139575958f);
  s = f2_fma(s, t, 0.1429252326488495f);
  // (|x| bounded in the last term, which is 0 there: an infinite x stays what it was; 0.5 |x| + 0.5 x is max(x, 0))
  float sx, sy, lx, ly;
  f2_split(f2_fma(u, r, h), sx, sy);
  f2_split(f2_fma(f2(-fminf(ax, 64.f), -fminf(ay, 64.f)), f2_mul(f2_mul(s, t), f2(ex, ey)), f2_fma(a, f2(0.5f, 0.5f), h)), lx, ly);
  // (said in PTX because the compiler made it a branch around either form, which a warp walks both of: 46.8 us for that layer)
  asm("{\n\t.reg .pred p;\n\tsetp.lt.f32 p, %1, 0f3F8CCCCD;\n\tselp.f32 %0, %2, %3, p;\n\t}" : "=f"(x) : "f"(ax), "f"(sx), "f"(lx));
  asm("{\n\t.reg .pred p;\n\tsetp.lt.f32 p, %1, 0f3F8CCCCD;\n\tselp.f32 %0, %2, %3, p;\n\t}" : "=f"(y) : "f"(ay), "f"(sy), "f"(ly));
}

__device__ __forceinline__ float gelu_tanh(float v) {
  float t;
  asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(0.7978845608028654f * fmaf(0.044715f * v, v * v, v)));
  return 0.5f * v * (1.f + t);
}

// Epilogue of one tile when tokens are the MMA rows: this thread's token, its columns = consecutive weight rows.
struct EpiRow {
  int act;
  const uint16_t* bias;  // at the group's first feature, or null
  const uint16_t* res;   // the token's residual row at the group's first feature, or null
  int extra_vec;
  void* out;
  long long nbase, os_hi, os_lo;  // element offset of the token; strides of (m / per) and (m % per)
  int per, M, m0, cend;           // first weight row of the tile, columns of the tile that exist
  bool n_ok;                      // token exists
};

// Two neighbouring features' bias, for the warp's lanes to pass on: requested ahead of the wait for the accumulator, whose epilogue otherwise
// ran into the latency of its loads once per 16 columns.  (A plain load, as the residual's: the kernel ahead may have written either while this one was
// already running.)
__device__ __forceinline__ uint32_t epilogue_bias2(const EpiRow& e, int m) {
  return e.bias != nullptr && e.extra_vec && m < e.M ? *reinterpret_cast<const uint32_t*>(e.bias + m) : 0u;
}

// Adds bias and residual of features m .. m + 15 to 16 accumulator columns, the activation in between (16-byte pieces where
// the host found them aligned; with LANES the bias then in lanes from .. from + 7 of `bias2`).  The whole warp.
template <bool BF16, bool LANES>
__device__ __forceinline__ void epilogue_extra16(const EpiRow& e, int m, uint32_t (&r)[16], uint32_t bias2, int from) {
#pragma unroll
  for (int part = 0; part < 2; ++part) {
    if (LANES && part == 0 && e.extra_vec) {
      if (e.bias == nullptr) continue;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float2 f = gemm_unpack<BF16>(__shfl_sync(0xffffffffu, bias2, from + k));
        r[2 * k] = __float_as_uint(__uint_as_float(r[2 * k]) + f.x);
        r[2 * k + 1] = __float_as_uint(__uint_as_float(r[2 * k + 1]) + f.y);
      }
      continue;
    }
    const uint16_t* src = part == 0 ? e.bias : e.res;
    if (part == 1 && e.act == 1) {
#pragma unroll
      for (int j = 0; j < 16; j += 2) {
        float x = __uint_as_float(r[j]), y = __uint_as_float(r[j + 1]);
        gelu_erf2(x, y);
        r[j] = __float_as_uint(x);
        r[j + 1] = __float_as_uint(y);
      }
    } else if (part == 1 && e.act == 2) {
#pragma unroll
      for (int j = 0; j < 16; ++j) r[j] = __float_as_uint(gelu_tanh(__uint_as_float(r[j])));
    }
    if (src == nullptr || (part == 1 && !e.n_ok)) continue;
    if (e.extra_vec && m + 16 <= e.M) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint4 v = *reinterpret_cast<const uint4*>(src + m + 8 * h);
        const uint32_t ws[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float2 f = gemm_unpack<BF16>(ws[k]);
          r[8 * h + 2 * k] = __float_as_uint(__uint_as_float(r[8 * h + 2 * k]) + f.x);
          r[8 * h + 2 * k + 1] = __float_as_uint(__uint_as_float(r[8 * h + 2 * k + 1]) + f.y);
        }
      }
    } else {
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (m + j < e.M) r[j] = __float_as_uint(__uint_as_float(r[j]) + gemm_load<BF16>(src + m + j));
    }
  }
}

}  // namespace blr
