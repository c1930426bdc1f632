// int4 and int8 weights to bf16 / f16 pairs, for the kernels that multiply in 16-bit floats.
#pragma once

#include <cuda_fp16.h>
#include <stdint.h>
#include <type_traits>

namespace qmm {

// a * m + c on pairs
template <typename XT>
__device__ __forceinline__ uint32_t pair_fma(uint32_t a, uint32_t m, uint32_t c) {
  uint32_t r;
  if constexpr (std::is_same<XT, __half>::value) asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(m), "r"(c));
  else asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(m), "r"(c));
  return r;
}

// Byte permutation with the selectors' sign bit: 8 + i is the sign of byte i, eight times
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
  return r;
}

// Integers to 16-bit floats.  A 16-bit float with a zero in its upper byte is its lower byte u times the type's smallest
// subnormal, 2^-133 (bf16) or 2^-24 (f16), for every u: subnormals and the first normal numbers are evenly spaced.  So the
// offset-binary value only has to be put beside a zero byte, wherever it lies in the byte, and one multiply-add takes the
// offset off and brings the value to 2^-6 (bf16) or 2^-9 (f16) of itself; all of it is exact.  The factor is the most that the
// types' largest power of two leaves, and comes back in at the end (Unit).  (Integer instructions run at half rate and bound the
// kernels that convert: nine for eight nibbles and six for four bytes when the bytes go under an exponent, six and
// three this way.)
template <typename XT>
struct Unit {
  static constexpr bool kHalf = std::is_same<XT, __half>::value;
  static constexpr float kBack = kHalf ? 512.f : 64.f;
  static constexpr uint32_t kLow = kHalf ? 0x7800u : 0x7F00u, kHigh = kHalf ? 0x6800u : 0x7D00u;  // 2^15, 2^11; 2^127, 2^123
  static constexpr uint32_t kEight = kHalf ? 0xA400u : 0xBE00u, k128 = kHalf ? 0xB400u : 0xC000u;  // -8 and -128 of these units
};

// Eight nibbles -> four pairs in k order: the low nibble of a byte, then the high one (sixteen times itself in its byte).
template <typename XT>
__device__ __forceinline__ void cvt_s4x8(uint32_t w, uint32_t* p) {
  using U = Unit<XT>;
  const uint32_t lo = (w & 0x0F0F0F0Fu) ^ 0x08080808u, hi = (w & 0xF0F0F0F0u) ^ 0x80808080u;
  // selector 8 + i: the sign of byte i of `lo`, a zero
  p[0] = pair_fma<XT>(prmt(lo, hi, 0x8480), U::kHigh << 16 | U::kLow, U::kEight * 0x10001u);
  p[1] = pair_fma<XT>(prmt(lo, hi, 0x8581), U::kHigh << 16 | U::kLow, U::kEight * 0x10001u);
  p[2] = pair_fma<XT>(prmt(lo, hi, 0x8682), U::kHigh << 16 | U::kLow, U::kEight * 0x10001u);
  p[3] = pair_fma<XT>(prmt(lo, hi, 0x8783), U::kHigh << 16 | U::kLow, U::kEight * 0x10001u);
}

// Four bytes -> two pairs in k order
template <typename XT>
__device__ __forceinline__ void cvt_s8x4(uint32_t w, uint32_t* p) {
  using U = Unit<XT>;
  const uint32_t u = w ^ 0x80808080u;
  p[0] = pair_fma<XT>(__byte_perm(u, 0u, 0x4140), U::kLow * 0x10001u, U::k128 * 0x10001u);
  p[1] = pair_fma<XT>(__byte_perm(u, 0u, 0x4342), U::kLow * 0x10001u, U::k128 * 0x10001u);
}

}  // namespace qmm
