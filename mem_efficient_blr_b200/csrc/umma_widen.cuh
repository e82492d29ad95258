// Widening of stored int8 / packed int4 weights to the 16-bit dtype, shared by the GEMM kernels that stage them as they are.
#pragma once
#include "ptx.cuh"

namespace blr {

// Bytes k0 and k0 + 1 of `w` hold u = q + OFF: returns (q * s) for both as two values of the 16-bit dtype, the
// product rounded once (q and the fp16 scale are exact in either arithmetic: the result equals rn(float(q) * float(s))); q alone, which is exact, where
// not SCALED.
template <bool BF16, int OFF, int K0, bool SCALED>
__device__ __forceinline__ uint32_t widen2(uint32_t w, float sf, __half2 sh) {
  if constexpr (BF16) {
    // 0x4B0000uu = 2^23 + u as a float
    const float a = __uint_as_float(prmt(w, 0x4B000000u, 0x7650u | K0)) - (8388608.f + OFF);
    const float b = __uint_as_float(prmt(w, 0x4B000000u, 0x7650u | (K0 + 1))) - (8388608.f + OFF);
    const __nv_bfloat162 v = SCALED ? __floats2bfloat162_rn(a * sf, b * sf) : __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
  } else {
    // 0x64uu = 1024 + u as a half
    const uint32_t m = prmt(w, 0x64646464u, K0 == 0 ? 0x4140u : 0x4342u);
    const __half2 off = __floats2half2_rn(1024.f + OFF, 1024.f + OFF);
    __half2 v = __hsub2(*reinterpret_cast<const __half2*>(&m), off);
    if constexpr (SCALED) v = __hmul2(v, sh);
    return *reinterpret_cast<const uint32_t*>(&v);
  }
}

// 16 consecutive quantised weights at `raw` (shared memory) -> 32 bytes of the 16-bit dtype in o[0..7]
template <bool BF16, int WQ, bool SCALED = true>
__device__ __forceinline__ void widen16(uint32_t raw, __half scale, uint32_t (&o)[8]) {
  uint32_t bw[4];
  constexpr int OFF = WQ == 8 ? 128 : 8;
  if constexpr (WQ == 8) {
    asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(bw[0]), "=r"(bw[1]), "=r"(bw[2]), "=r"(bw[3]) : "r"(raw));
#pragma unroll
    for (int i = 0; i < 4; ++i) bw[i] ^= 0x80808080u;
  } else {
    uint32_t w[2];
    asm volatile("ld.shared.v2.b32 {%0,%1}, [%2];" : "=r"(w[0]), "=r"(w[1]) : "r"(raw));
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const uint32_t lo = (w[i] & 0x0F0F0F0Fu) ^ 0x08080808u, hi = ((w[i] >> 4) & 0x0F0F0F0Fu) ^ 0x08080808u;
      bw[2 * i] = prmt(lo, hi, 0x5140u);      // weights 0..3 of the word: (low, high) nibbles of bytes 0, 1
      bw[2 * i + 1] = prmt(lo, hi, 0x7362u);  // weights 4..7
    }
  }
  const float sf = __half2float(scale);
  const __half2 sh = __half2half2(scale);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    o[2 * i] = widen2<BF16, OFF, 0, SCALED>(bw[i], sf, sh);
    o[2 * i + 1] = widen2<BF16, OFF, 2, SCALED>(bw[i], sf, sh);
  }
}

}  // namespace blr
