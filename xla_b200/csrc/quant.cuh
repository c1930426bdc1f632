// The per-token activation quantizer's scalar steps, shared by the stand-alone kernel and the decode kernel that
// quantizes its activations itself.  Bit for bit the reference's (torch_xla/experimental/xla_quantized_matmul.py:56-73):
// scale = amax / 127 and q = x / scale, each rounded to the activations' type, then rint.
#pragma once

#include "common.cuh"

namespace qmm {

template <typename T>
__device__ __forceinline__ float round_to(float v) {
  return to_f32(from_f32<T>(v));
}

__device__ __forceinline__ int8_t to_int8(float r, bool saturate) {
  if (r != r) return 0;
  if (saturate) {
    r = fminf(fmaxf(r, -128.f), 127.f);
    return (int8_t)(int)r;
  }
  // wrap like a float -> int32 -> int8 conversion chain does for values in int32 range
  if (r > 2147483520.f || r < -2147483648.f) return 0;
  return (int8_t)(uint8_t)(((int)r) & 0xff);
}

template <typename T>
__device__ __forceinline__ float quant_scale(float amax) {
  return round_to<T>(__fdiv_rn(amax, 127.0f));
}

template <typename T>
__device__ __forceinline__ int8_t quantize_value(float xv, float scale, bool saturate) {
  return to_int8(rintf(round_to<T>(__fdiv_rn(xv, scale))), saturate);
}

// bf16 activations with a regular scale.  The quotient x / scale must be the correctly rounded fp32 quotient (it is
// rounded to bf16 next and ties decide).  One Newton step on q0 = x * (1/scale) gives it: both operands have 8-bit
// significands, so the exact quotient is either a tie (exactly representable: the step lands on it) or at least 2^-17
// away from any bf16 rounding boundary, far more than the error of q0.
// Everything after the quotient stays on the FMA and integer pipes (no conversion-unit instruction):
//   bf16 rounding   Veltkamp split with 2^16 + 1: g = q * 65537, qb = g + (q - g) is q rounded to 8 significant bits,
//                   ties to even (each step is one correctly rounded operation; the explicit _rn intrinsics keep the
//                   compiler from fusing them)
//   rint -> int     qb + 1.5 * 2^23 leaves the integer, rounded ties-to-even, in the low mantissa bits
// The int8 conversion is a clamp in integers, or the low byte.
__device__ __forceinline__ bool quant_regular(float scale) { return scale > 1e-30f && scale < 1e30f; }

__device__ __forceinline__ int quantize_bf16_regular(float xv, float scale, float rcp, bool saturate) {
  const float q0 = xv * rcp;
  const float r = fmaf(-q0, scale, xv);
  const float q = fmaf(r, rcp, q0);
  const float g = __fmul_rn(q, 65537.f);
  const float qb = __fadd_rn(g, __fsub_rn(q, g));
  const int t = __float_as_int(__fadd_rn(qb, 12582912.f)) - 0x4B400000;
  return saturate ? max(-128, min(127, t)) : t;
}

// low bytes of four ints
__device__ __forceinline__ uint32_t pack_bytes(const int* q) {
  return __byte_perm(__byte_perm((uint32_t)q[0], (uint32_t)q[1], 0x0040), __byte_perm((uint32_t)q[2], (uint32_t)q[3], 0x0040), 0x5410);
}

}  // namespace qmm
