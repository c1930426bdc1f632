// Shared host/device helpers for the quantized-linear kernels.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <type_traits>

#include "../../include/qmm_b200.h"

namespace qmm {

// ---- error reporting (host) ---------------------------------------------------------------
int fail(int status, const char* fmt, ...);  // records the message for qmm_last_error_string
int check_launch(const char* what);          // cudaPeekAtLastError -> status

inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

// Word that kernels with bounded waits set when a wait gives up (0 = healthy).
uint32_t* device_error_word();  // device address of the flag for the current device, or nullptr

// How long a kernel waits for another GPU before it gives up, in SM clock cycles (qmm_set_peer_wait_limit).
long long peer_wait_cycles();

inline int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

inline bool aligned(const void* p, size_t a) { return (reinterpret_cast<uintptr_t>(p) % a) == 0; }

inline bool valid_float_dtype(int dt) { return dt == QMM_F32 || dt == QMM_BF16 || dt == QMM_F16; }

inline size_t dtype_size(int dt) { return dt == QMM_F32 ? 4 : 2; }

int sm_count();
bool device_is_sm100();

// ---- element access (device) --------------------------------------------------------------
template <int DT>
struct ElemOf;
template <>
struct ElemOf<QMM_F32> {
  using type = float;
};
template <>
struct ElemOf<QMM_BF16> {
  using type = __nv_bfloat16;
};
template <>
struct ElemOf<QMM_F16> {
  using type = __half;
};

__device__ __forceinline__ float to_f32(float v) { return v; }
__device__ __forceinline__ float to_f32(__nv_bfloat16 v) { return __bfloat162float(v); }
__device__ __forceinline__ float to_f32(__half v) { return __half2float(v); }

template <typename T>
__device__ __forceinline__ T from_f32(float v);
template <>
__device__ __forceinline__ float from_f32<float>(float v) {
  return v;
}
template <>
__device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float v) {
  return __float2bfloat16_rn(v);
}
template <>
__device__ __forceinline__ __half from_f32<__half>(float v) {
  return __float2half_rn(v);
}

// Runtime-typed scalar load/store for the kernels that are not specialised per dtype.
__device__ __forceinline__ float load_as_f32(const void* p, int64_t i, int dt) {
  if (dt == QMM_F32) return reinterpret_cast<const float*>(p)[i];
  if (dt == QMM_BF16) return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p)[i]);
  return __half2float(reinterpret_cast<const __half*>(p)[i]);
}

__device__ __forceinline__ void store_from_f32(void* p, int64_t i, int dt, float v) {
  if (dt == QMM_F32)
    reinterpret_cast<float*>(p)[i] = v;
  else if (dt == QMM_BF16)
    reinterpret_cast<__nv_bfloat16*>(p)[i] = __float2bfloat16_rn(v);
  else
    reinterpret_cast<__half*>(p)[i] = __float2half_rn(v);
}

// ---- data of earlier kernels (device) --------------------------------------------------------
// A kernel launched with programmatic stream serialization starts while the kernel before it still runs.  Only the raw
// weights, which no kernel directly in front may write, are read before griddepcontrol.wait; activations, scratch, scales
// and zero points come after it, and with ordinary loads: __ldg and const __restrict__ stand for data that nobody writes
// while the kernel runs, so such a load may be moved ahead of the wait or served from a stale cache line.
template <typename T>
__device__ __forceinline__ T ld_ordered(const T* p) {
  return *p;
}

// Brings a line into L2, where all SMs see the same data: allowed ahead of the wait for data that is loaded after it.
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// ---- weight scales and zero points ---------------------------------------------------------
// In fp32 or in a 16-bit type (the buffers of a quantized 16-bit model), both in the same one.
struct Scales {
  const void* scale;
  const void* zp;  // or null
  int dt;
};

inline const void* elements_from(const void* p, int64_t n, int dt) {
  return p ? static_cast<const uint8_t*>(p) + n * (int64_t)dtype_size(dt) : nullptr;
}

// Kernels that stream block scales copy them in 32-bit words: one fp32 value, or the pair of 16-bit values that holds the
// wanted one.  For that a 16-bit tensor has to start on a word.  (Per channel the scales are read one by one.)
inline bool scale_words_ok(const Scales& s, int64_t block_size) {
  return s.dt == QMM_F32 || block_size <= 0 || (aligned(s.scale, 4) && aligned(s.zp, 4));
}
// An odd number of 16-bit scales: the last one's word would reach beyond the tensor, so it is copied by itself.
inline int scale_tail(const Scales& s, int64_t blocks, int64_t N) { return s.dt != QMM_F32 && blocks * N % 2 != 0; }

// Copies the word that holds the scale at `src` to shared memory.  W16: 16-bit scales; a template parameter of the kernels,
// because their loops have no register to spare for the conversion (decided at run time it cost fp32 scales 2 to 25 %: int4
// block 128, [57344,8192] and [8192,28672] at 64 tokens 182 us, up to 228).
template <bool W16>
__device__ __forceinline__ void copy_scale_word(uint32_t dst, const uint8_t* src) {
  const uintptr_t at = reinterpret_cast<uintptr_t>(src);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(W16 ? at & ~(uintptr_t)3 : at) : "memory");
}

__device__ __forceinline__ void copy_last_scale(uint32_t dst, const uint8_t* src) {
  asm volatile("st.shared.u16 [%0], %1;" ::"r"(dst), "h"(ld_ordered(reinterpret_cast<const unsigned short*>(src))) : "memory");
}

// The scale in a copied word: of row n (counted from an even one) and block b of a weight with N rows; T: its type, if known.
// The odd rows, and with an odd N those of the other parity in every second block, are the second value of a pair.
template <bool W16, typename T = void>
__device__ __forceinline__ float scale_in(const uint32_t* word, int n, int b, int N, int dt) {
  if (!W16) return __uint_as_float(*word);
  const uint32_t at = ((uint32_t)n & 1u) ^ ((uint32_t)b & (uint32_t)N & 1u);
  const unsigned short h = reinterpret_cast<const unsigned short*>(word)[at];
  if (std::is_same<T, __half>::value || (std::is_void<T>::value && dt == QMM_F16)) return __half2float(__ushort_as_half(h));
  return __uint_as_float((uint32_t)h << 16);
}

// The same for a word in a register; T: the type of 16-bit scales.
template <bool W16, typename T>
__device__ __forceinline__ float scale_of_word(uint32_t word, int n, int b, int N) {
  if (!W16) return __uint_as_float(word);
  const uint32_t at = ((uint32_t)n & 1u) ^ ((uint32_t)b & (uint32_t)N & 1u);
  const uint32_t h = __byte_perm(word, 0u, at ? 0x3244u : 0x1044u);  // the value in the upper half
  return std::is_same<T, __half>::value ? __half2float(__ushort_as_half((unsigned short)(h >> 16))) : __uint_as_float(h);
}

// A single scale as its bits, and their value: apart, because the conversion waits for the load
__device__ __forceinline__ uint32_t load_scale_bits(const void* p, int64_t n, int dt) {
  return dt == QMM_F32 ? ld_ordered(static_cast<const uint32_t*>(p) + n) : (uint32_t)ld_ordered(static_cast<const unsigned short*>(p) + n);
}
__device__ __forceinline__ float scale_value(uint32_t bits, int dt) {
  return dt == QMM_F32 ? __uint_as_float(bits) : dt == QMM_BF16 ? __uint_as_float(bits << 16) : __half2float(__ushort_as_half((unsigned short)bits));
}

// 128-bit streaming load that does not pollute L1 (weights are read exactly once).
__device__ __forceinline__ uint4 ld_stream_u4(const void* p) {
  uint4 r;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
               : "l"(p));
  return r;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Dispatch a runtime dtype to a compile-time one.
#define QMM_DISPATCH_DTYPE(dt, NAME, ...)          \
  switch (dt) {                                    \
    case QMM_F32: {                                \
      using NAME = float;                          \
      __VA_ARGS__;                                 \
    } break;                                       \
    case QMM_BF16: {                               \
      using NAME = __nv_bfloat16;                  \
      __VA_ARGS__;                                 \
    } break;                                       \
    default: {                                     \
      using NAME = __half;                         \
      __VA_ARGS__;                                 \
    } break;                                       \
  }

}  // namespace qmm
