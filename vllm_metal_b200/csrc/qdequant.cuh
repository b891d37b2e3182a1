// Unpacking of affine-quantized words to 16-bit operands of the tensor cores (qgemm_tc.cu, qexperts.cu).
#pragma once

#include "common.cuh"

namespace b200 {
namespace qtc {

// ------------------------------------------------------------- dequant traits ----
template <typename T>
struct Cvt;
template <>
struct Cvt<__nv_bfloat16> {
  using T2 = __nv_bfloat162;
  static constexpr int kFmt = 1;
  static constexpr uint32_t kMagic = 0x43004300u;  // bf16 128.0: 128 + q exact for q < 128
  __device__ static __forceinline__ T2 magic_off() { return __float2bfloat162_rn(-128.f); }
  __device__ static __forceinline__ T2 pair(float v) { return __float2bfloat162_rn(v); }
  __device__ static __forceinline__ T2 bcast(uint16_t raw) {
    __nv_bfloat16_raw r;
    r.x = raw;
    return __bfloat162bfloat162(__nv_bfloat16(r));
  }
  __device__ static __forceinline__ uint32_t f2(float lo, float hi) {
    T2 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  }
  __device__ static __forceinline__ float to_f(uint16_t raw) {
    return __uint_as_float((uint32_t)raw << 16);
  }
};
template <>
struct Cvt<__half> {
  using T2 = __half2;
  static constexpr int kFmt = 0;
  static constexpr uint32_t kMagic = 0x64006400u;  // fp16 1024.0: 1024 + q exact
  __device__ static __forceinline__ T2 magic_off() { return __float2half2_rn(-1024.f); }
  __device__ static __forceinline__ T2 pair(float v) { return __float2half2_rn(v); }
  __device__ static __forceinline__ T2 bcast(uint16_t raw) {
    __half_raw r;
    r.x = raw;
    return __half2half2(__half(r));
  }
  __device__ static __forceinline__ uint32_t f2(float lo, float hi) {
    T2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  }
  __device__ static __forceinline__ float to_f(uint16_t raw) {
    __half_raw r;
    r.x = raw;
    return __half2float(__half(r));
  }
};

// By mask and magic number: an integer's bits under a chosen exponent read as that power of two plus the integer, which one exact
// operation takes off again (the method of Kim, Henry, Fahim, Awadalla, "Who Says Elephants Can't Run", 2022, for fp16).
// 8 nibbles of one packed word -> 8 values s*q+b in memory order (k0..k7), as 4 packed pairs.
// PRE: the word was nibble-permuted at load time (b200_qlinear_prepack) so that nibbles
// (i, i+4) hold (k_{2i}, k_{2i+1}); the extraction then yields the pairs in memory order
// and the four PRMTs disappear.
template <typename T, bool PRE>
__device__ __forceinline__ uint4 dequant_word4(uint32_t w, typename Cvt<T>::T2 s2,
                                               typename Cvt<T>::T2 b2) {
  using C = Cvt<T>;
  using T2 = typename C::T2;
  uint32_t a[4];
  const uint32_t mask = 0x000F000Fu, magic = C::kMagic;
  // (nibble i, nibble i+4) as the low/high halves: one LOP3 ((x & mask) | magic) each (the constants live in registers so
  // that ptxas keeps it a single instruction).  Nibbles 1 and 3 stay four bits up, where fp16 reads 1024 + 16 q: an exact
  // FMA brings them down, which saves their shifts.
  const T2 sixteenth = Cvt<T>::pair(0.0625f), m64 = Cvt<T>::pair(-64.f);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    uint32_t v;
    T2 q;
    if constexpr (C::kFmt == 0) {
      const uint32_t half_word = i < 2 ? w : w >> 8;
      asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(v) : "r"(half_word), "r"(i & 1 ? mask << 4 : mask), "r"(magic));
      q = i & 1 ? __hfma2(*reinterpret_cast<T2*>(&v), sixteenth, m64) : __hadd2(*reinterpret_cast<T2*>(&v), C::magic_off());
    } else {
      asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(v) : "r"(w >> (4 * i)), "r"(mask), "r"(magic));
      q = __hadd2(*reinterpret_cast<T2*>(&v), C::magic_off());  // exact: q in [0, 15]
    }
    T2 r = __hfma2(s2, q, b2);  // s*q+b, one rounding
    a[i] = *reinterpret_cast<uint32_t*>(&r);
  }
  uint4 o;
  if constexpr (PRE) {
    o.x = a[0]; o.y = a[1]; o.z = a[2]; o.w = a[3];
  } else {
    o.x = __byte_perm(a[0], a[1], 0x5410);  // (k0, k1)
    o.y = __byte_perm(a[2], a[3], 0x5410);  // (k2, k3)
    o.z = __byte_perm(a[0], a[1], 0x7632);  // (k4, k5)
    o.w = __byte_perm(a[2], a[3], 0x7632);  // (k6, k7)
  }
  return o;
}
// 4 bytes of one packed word -> 4 fp16 values s*q+b: a byte under the exponent byte 0x64 reads 1024 + q exactly
// (q < 1024), the subtraction is exact and the FMA rounds once -- the same single rounding as an fp32 fma followed
// by a conversion, in six packed operations instead of ten scalar ones per word (the int8 GEMM at
// M >= 256 was dequant-bound on the conversions: 0.28-0.47 of the bf16 peak, profiles/r02_gemm_bigm.txt).
template <typename T>
__device__ __forceinline__ uint2 dequant_word8(uint32_t w, float s, float b) {
  const __half2 s2 = __float2half2_rn(s), b2 = __float2half2_rn(b), off = __float2half2_rn(-1024.f);
  const uint32_t lo = __byte_perm(w, 0x64646464u, 0x5140), hi = __byte_perm(w, 0x64646464u, 0x7362);
  const __half2 q0 = __hadd2(*reinterpret_cast<const __half2*>(&lo), off);
  const __half2 q1 = __hadd2(*reinterpret_cast<const __half2*>(&hi), off);
  const __half2 r0 = __hfma2(s2, q0, b2), r1 = __hfma2(s2, q1, b2);
  uint2 o;
  o.x = *reinterpret_cast<const uint32_t*>(&r0);
  o.y = *reinterpret_cast<const uint32_t*>(&r1);
  return o;
}

}  // namespace qtc
}  // namespace b200
