// Activations as int8 limbs: x = X * 2^(e - q) with an integer X relative to the row's largest exponent e, and the
// balanced base-256 digits of X.  Shared by the kernels that multiply unconverted integer weights.
#pragma once

#include "common.cuh"

namespace qmm {

template <typename XT>
__device__ __forceinline__ void load8(const XT* p, float* v);
template <>
__device__ __forceinline__ void load8<float>(const float* p, float* v) {
  const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
template <>
__device__ __forceinline__ void load8<__nv_bfloat16>(const __nv_bfloat16* p, float* v) {
  const uint4 a = *reinterpret_cast<const uint4*>(p);
  const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[2 * i] = __uint_as_float(w[i] << 16);
    v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}
template <>
__device__ __forceinline__ void load8<__half>(const __half* p, float* v) {
  const uint4 a = *reinterpret_cast<const uint4*>(p);
  const __half2* h = reinterpret_cast<const __half2*>(&a);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = __half22float2(h[i]);
    v[2 * i] = f.x;
    v[2 * i + 1] = f.y;
  }
}

// 2^(q-e) and 2^(e-q) * pw_mul for a row whose largest |x| has the float bits `mx`; a row with a non-finite entry
// gets (0, NaN), an all-zero or denormal row any small exponent.  Three limbs: q = 21 (|X| < 2^22 of the 2^23 that
// balanced limbs hold).  Two limbs: balanced limbs hold -32896..32639, so q = 14 unless the row's largest value
// would round above 32639 (mantissa beyond 32639 / 16384), which takes q = 13.
template <int NL>
__device__ __forceinline__ void row_factors(uint32_t mx, float pw_mul, float& mult, float& pw) {
  int e = (int)(mx >> 23) - 127;
  const bool finite = e < 128;
  if (e < -100) e = -100;
  const int q = NL == 3 ? 21 : ((mx & 0x7fffffu) > 0x7EFE00u ? 13 : 14);
  mult = finite ? __uint_as_float((uint32_t)(q - e + 127) << 23) : 0.f;
  pw = finite ? __uint_as_float((uint32_t)(e - q + 127) << 23) * pw_mul : __uint_as_float(0x7fc00000u);
}

// Eight values -> the bytes of their three limbs, packed in k order (two words per limb).
// X = rint(v * mult) comes out of one FMA against 1.5 * 2^23 (the sum lands where fp32 spacing is 1, so the FMA's
// round-to-nearest-even IS the rint, and X sits in the low mantissa bits).  Balanced limbs l_i in [-128,127] with
// X = l0 + 256 l1 + 65536 l2 are the base-256 digits of X + 0x808080, each minus 128: one integer add puts the digits
// into bytes 0..2, one XOR with 0x808080 turns digit into limb.  Three instructions per value, then byte gathers.
// With two limbs the same holds for X + 0x8080 and bytes 0..1 (l2 is not written).
template <int NL>
__device__ __forceinline__ void split8(const float* v, float mult, uint32_t* l0, uint32_t* l1, uint32_t* l2) {
  constexpr uint32_t kBias = NL == 3 ? 0x808080u : 0x8080u;
  uint32_t z[8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
    z[i] = (__float_as_uint(fmaf(v[i], mult, 12582912.f)) + (kBias - 0x4B400000u)) ^ kBias;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint32_t a = z[4 * h], b = z[4 * h + 1], c = z[4 * h + 2], d = z[4 * h + 3];
    // byte j of a/b in the low half, of c/d in the high half
    const uint32_t ab0 = __byte_perm(a, b, 0x0040), cd0 = __byte_perm(c, d, 0x0040);
    const uint32_t ab1 = __byte_perm(a, b, 0x0051), cd1 = __byte_perm(c, d, 0x0051);
    l0[h] = __byte_perm(ab0, cd0, 0x5410);
    l1[h] = __byte_perm(ab1, cd1, 0x5410);
    if constexpr (NL == 3) {
      const uint32_t ab2 = __byte_perm(a, b, 0x0062), cd2 = __byte_perm(c, d, 0x0062);
      l2[h] = __byte_perm(ab2, cd2, 0x5410);
    }
  }
}

}  // namespace qmm
