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

// x Phi(x), Phi the normal distribution: max(x, 0) - |x| Phi(-|x|), and Phi(-|x|) = exp(-x^2 / 2) P(t) with t = 1 / (1 + p |x|) and P of six terms
// without a constant one (the form of Hastings' approximations; p and P fitted here to the least largest error of |x| Phi(-|x|), 2.8e-9).
// In single precision at most 2.4e-7 off, 3.8e-8 in the root mean square over normal x of deviation 2, where 0.5 x (1 + erff(x / sqrt 2)) is 4.5e-7 and 5.0e-8 off; no
// cancellation for negative x.  17 instructions against some 40: the last GEMM of 768 -> 3072, R = 288 on 3152 tokens was bound by them.
__device__ __forceinline__ float gelu_erf(float v) {
  const float a = fabsf(v);
  float t, e;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(t) : "f"(fmaf(0.280859027f, a, 1.f)));
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(v * -0.72134752f * v));
  float s = fmaf(-0.10660312324762344f, t, 0.3891717791557312f);
  s = fmaf(s, t, -0.2372603714466095f);
  s = fmaf(s, t, 0.2709754407405853f);
  s = fmaf(s, t, 0.06658425182104111f);
  s = fmaf(s, t, 0.11713188141584396f);
  // (|x| bounded in the second term, which is 0 there: an infinite x stays what it was; 0.5 |x| + 0.5 x is max(x, 0))
  return fmaf(-fminf(a, 64.f), s * t * e, fmaf(0.5f, a, 0.5f * v));
}

__device__ __forceinline__ float gemm_act(float v, int act) {
  if (act == 1) return gelu_erf(v);
  if (act == 2) {
    float t;
    asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(0.7978845608028654f * fmaf(0.044715f * v, v * v, v)));
    return 0.5f * v * (1.f + t);
  }
  return v;
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
// ran into the latency of its loads once per 16 columns.
__device__ __forceinline__ uint32_t epilogue_bias2(const EpiRow& e, int m) {
  return e.bias != nullptr && e.extra_vec && m < e.M ? __ldg(reinterpret_cast<const uint32_t*>(e.bias + m)) : 0u;
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
    if (part == 1 && e.act != 0) {
#pragma unroll
      for (int j = 0; j < 16; ++j) r[j] = __float_as_uint(gemm_act(__uint_as_float(r[j]), e.act));
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
