// extern "C" entry points of libqmm_b200 (declared in include/qmm_b200.h): argument checks,
// kernel-family selection, and the host-side helpers the kernels share.
#include <cuda.h>
#include <algorithm>
#include <atomic>
#include <stdarg.h>
#include <stdio.h>
#include <string.h>

#include "common.cuh"
#include "kernels.h"
#include "ptx_sm100.cuh"

namespace qmm {

// ---- error reporting ----------------------------------------------------------------------
static thread_local char g_last_error[512] = "";

int fail(int status, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_last_error, sizeof(g_last_error), fmt, ap);
  va_end(ap);
  return status;
}

int check_launch(const char* what) {
  cudaError_t e = cudaPeekAtLastError();
  if (e != cudaSuccess) {
    cudaGetLastError();  // clear the sticky-less launch error so later calls start clean
    return fail(QMM_ERR_LAUNCH, "%s: %s", what, cudaGetErrorString(e));
  }
  return QMM_OK;
}

// ---- device queries -----------------------------------------------------------------------
struct DeviceInfo {
  bool known = false;
  int sms = 0;
  int cc_major = 0;
};
static DeviceInfo g_dev[64];

static DeviceInfo* device_info() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  DeviceInfo* d = &g_dev[dev];
  if (!d->known) {
    cudaDeviceProp prop;
    if (cudaGetDeviceProperties(&prop, dev) != cudaSuccess) return nullptr;
    d->sms = prop.multiProcessorCount;
    d->cc_major = prop.major;
    d->known = true;
  }
  return d;
}

int sm_count() {
  DeviceInfo* d = device_info();
  return d ? d->sms : 1;
}

bool device_is_sm100() {
  DeviceInfo* d = device_info();
  return d && d->cc_major == 10;
}

// One error word per device, living in the library's own device image.
__device__ uint32_t g_qmm_error_word;

uint32_t* device_error_word() {
  static uint32_t* cached[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  if (!cached[dev]) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_qmm_error_word) != cudaSuccess) {
      cudaGetLastError();
      return nullptr;
    }
    cached[dev] = reinterpret_cast<uint32_t*>(p);
  }
  return cached[dev];
}

static std::atomic<long long> g_peer_wait_cycles{2000000000ll};  // about a second of SM clock
long long peer_wait_cycles() { return g_peer_wait_cycles.load(std::memory_order_relaxed); }


// ---- tensor maps --------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) != cudaSuccess ||
        qres != cudaDriverEntryPointSuccess) {
      cudaGetLastError();
      return nullptr;
    }
    fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

int encode_tmap_2d(CUtensorMap* map, const void* base, int elem_bytes, bool is_float16_family,
                   uint64_t rows, uint64_t cols, uint32_t box_rows, uint32_t box_cols) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return fail(QMM_ERR_DEVICE, "driver does not provide cuTensorMapEncodeTiled");
  CUtensorMapDataType dt = CU_TENSOR_MAP_DATA_TYPE_UINT8;
  if (elem_bytes == 2) dt = is_float16_family ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_UINT16;
  if (elem_bytes == 4) dt = CU_TENSOR_MAP_DATA_TYPE_UINT32;
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {cols * (uint64_t)elem_bytes};
  cuuint32_t box[2] = {box_cols, box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(map, dt, 2, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    return fail(QMM_ERR_LAUNCH,
                "cuTensorMapEncodeTiled failed (%d) for [%llu x %llu] elem %d box [%u x %u]", (int)r,
                (unsigned long long)rows, (unsigned long long)cols, elem_bytes, box_rows, box_cols);
  return QMM_OK;
}

// ---- argument checks ----------------------------------------------------------------------
static int check_common(const void* x, int x_dt, const void* w, const void* scale, void* out,
                        int out_dt, int64_t M, int64_t N, int64_t K) {
  if (M < 0 || N < 0 || K < 0) return fail(QMM_ERR_BAD_SHAPE, "negative dimension (M=%lld N=%lld K=%lld)",
                                           (long long)M, (long long)N, (long long)K);
  if (!valid_float_dtype(x_dt) || !valid_float_dtype(out_dt))
    return fail(QMM_ERR_UNSUPPORTED, "dtype must be QMM_F32, QMM_BF16 or QMM_F16 (x=%d out=%d)", x_dt, out_dt);
  if (M * N == 0) return QMM_OK;
  if (!out) return fail(QMM_ERR_NULL, "out is NULL");
  if (K > 0 && (!x || !w)) return fail(QMM_ERR_NULL, "x or w is NULL");
  if (!scale) return fail(QMM_ERR_NULL, "scale is NULL");
  return QMM_OK;
}

static bool env_flag(const char* name) {
  const char* v = getenv(name);
  return v && v[0] && v[0] != '0';
}

static void log_choice(const char* op, const char* variant, int64_t M, int64_t N, int64_t K) {
  static int on = -1;
  if (on < 0) on = env_flag("QMM_B200_LOG") ? 1 : 0;
  if (on) fprintf(stderr, "[qmm_b200] %s M=%lld N=%lld K=%lld -> %s\n", op, (long long)M, (long long)N,
                  (long long)K, variant);
}

}  // namespace qmm

using namespace qmm;

extern "C" {

int qmm_abi_version(void) { return QMM_ABI_VERSION; }

const char* qmm_status_string(int status) {
  switch (status) {
    case QMM_OK: return "ok";
    case QMM_ERR_BAD_SHAPE: return "bad shape";
    case QMM_ERR_UNSUPPORTED: return "unsupported";
    case QMM_ERR_MISALIGNED: return "misaligned";
    case QMM_ERR_LAUNCH: return "launch failure";
    case QMM_ERR_WORKSPACE: return "workspace too small";
    case QMM_ERR_NULL: return "null pointer";
    case QMM_ERR_DEVICE: return "device not supported";
    case QMM_ERR_TIMEOUT: return "device-side wait timed out";
    default: return "unknown status";
  }
}

const char* qmm_last_error_string(void) { return g_last_error; }

// AUTO choice for the weight-only ops on K-minor weights: the register-dequant MMA kernel for decode
// batches, the tcgen05 kernel above that, the CUDA-core GEMV where those cannot go (zero points, f32
// activations), the any-shape kernel for everything else.
static int pick_weight_only(int wbits, int64_t M, int64_t N, int64_t K, int64_t bs, const void* x, int x_dt,
                            const void* w, bool has_zp, bool sm100) {
  if (decode_mma_supported(wbits, M, N, K, bs, x, x_dt, w, has_zp)) return QMM_VARIANT_MMA;
  if (sm100 && mixed_tc_shape_ok(wbits, M, N, K, bs, x_dt, has_zp) && aligned(x, 16) && aligned(w, 16)) return QMM_VARIANT_TCGEN05;
  if (gemv_nk_supported(wbits, M, N, K, bs, x, x_dt, w)) return QMM_VARIANT_GEMV;
  return QMM_VARIANT_GENERIC;
}

// AUTO's choice between the two warp-level decode kernels (where the tensor-core kernels below were not taken).  The integer
// one streams weights 1.5 times faster, but every
// CTA of it first splits all activations into limbs, about 0.6 us per token at K = 4096, in proportion to M * K; the
// gain is proportional to the weight bytes.  K cancels: it wins at one token, and up to one token per 1850 bytes of
// weight column (14336 int8 outputs: 7 tokens; measured 15.1 against 16.7 us at 4, equal at 8; 4096 outputs: 2).
// Zero points, scale blocks of 64 and ragged K are beyond the other kernel.
static bool use_decode_i8(int wbits, int64_t M, int64_t N, int64_t K, int64_t bs, const void* x, int x_dt, const void* w, bool has_zp) {
  if (!decode_i8_supported(wbits, M, N, K, bs, x, x_dt, w, has_zp)) return false;
  return M == 1 || M * 1850 <= N * wbits / 8 || !decode_mma_supported(wbits, M, N, K, bs, x, x_dt, w, has_zp);
}

// Batches of two tokens and more of which a tensor-core kernel (tmem or i8tc: both take about as long for one token as for
// 32) beats the decode kernels, whose time grows with the tokens.  `decode`: the integer decode kernel takes the call.
//   zero points  The other decode kernel is the GEMV, four tokens at a time: int4 block 128 [8192,28672] 70 us at two tokens and
//                188 at eight, 49 on tmem; int8 per channel [4096,4096] 8 at two, 13 at four, 18 at five, 14 on i8tc, [5120,6912]
//                14 at two and 22 at three, 17 there; [28672,8192] 31 at two, 43 at five on the integer kernel, 49 on tmem, 185 on the GEMV
//                from six on.  int8: [14336,4096] 15 us at two and 18 at four, 16 on i8tc.
//                Where the integer kernel goes, not with scale blocks of 64 ([25292,2688] int4 at seven 22.9 us, 30.1 on tmem; int8
//                [28672,8192] at four 61.5, 70.6), and with other blocks later where there are more weight tiles than SMs (int4 block 128
//                [25292,2688] at eight 19.4, 22.1 on tmem, [14336,4096] 18.8, 16.1; int8 [28672,2048] at three 16.8, 18.9, at six 19.7, 19.3).
static bool zp_decode_on_tc(int wbits, int64_t M, int64_t N, int64_t K, int64_t bs, bool decode) {
  const int64_t E = N * K;
  if (M < 2) return false;
  if (M > 8) return true;
  if (!decode) return E >= (M == 2 ? 50000000 : M <= 4 ? 1 << 25 : 1 << 24);
  if (E < 1 << 25 || bs == 64) return false;
  const bool rounds = bs > 0 && ceil_div(N, 128) > sm_count();
  return wbits == 8 ? M * E >= (rounds ? 350000000 : 175000000) : M >= 6 && !rounds;
}

// Batches of nine to sixteen tokens, int4 with scale blocks, that the split-activation kernel has ahead of the tensor-memory one (figures
// there, under 9..32 tokens).
static bool int4_blocks_on_limbs(int wbits, int64_t M, int64_t N, int64_t K, int64_t bs, int x_dt) {
  const int64_t E = N * K;
  if (M <= 8 || M > 16 || wbits != 4 || bs <= 64 || E < 1 << 26 || !limb_tc_shape_ok(wbits, M, N, K, bs, x_dt, false)) return false;
  const bool rounds = ceil_div(N, 128) > sm_count();
  return M <= 10 ? E >= 80000000 || rounds : bs >= 256 && rounds && E < 1 << 27;
}

// Where AUTO takes the tensor-memory kernel (16-bit activations).
//   zero points    with scale blocks wherever a tensor-core kernel is taken: it applies them in the drain it runs anyway (int4
//                  block 128 [37888,3584] at 29 tokens 32 us against 59 on the split-activation kernel, [14336,4096] at 512: 106
//                  against 211).  Per channel the other kernel hands over once per tile, and the products are exact here but fp32
//                  sums of int8 ones are a little further off (2.5e-7 of the results against 1.2e-7; int4 8e-8 and 1.2e-7).  So
//                  2..8     here, but int8 with fp32 results and int4 from 2^27 values there: int4 [21601,2208] at eight tokens 14.8 us,
//                           18.4 there and 15.2 on the integer decode kernel, [8192,8192] at six 14.5, 18.9 there; [28672,8192] 33.6, 29.4
//                  9..32    here, but int4 from 2^25 values (to 42 tokens, a tile there: [28672,8192] at 16 37 us, 31 there)
//                  33..64   int4 here; int8 from 12288 outputs ([14336,4096] at 64 16 us, 18 there; [2970,1792] 10.4, 9.9 there)
//                  above    from 64 items of 128 rows and 192 tokens on, int8 only with long rows or narrow beyond one launch there
//                           ([8192,2048] at 445 36 us, 25 there, [28672,2048] 81, 62; [4096,14336] 62, 73; [2970,1792] at 1024 24, 31).  Fewer
//                           items: int4 with long rows, more items than SMs there (of 42 tokens), or more than one launch: [4096,14336] at
//                           128 32 us, 38 there, [8064,7168] 28, 38, [7168,2048] at 100 16, 19, [1024,512] at 1024 15, 21; else there where
//                           the result has 16 bits ([1024,4096] at 128 20, 17 there, [4096,4096] 21, 18)
//   blocks of 64   above 32 tokens.  The other kernel that goes on with them there, tcgen05, has tiles of 64 tokens and splits K over a cluster
//                  where they are few: ahead above 64 tokens while its tiles fit on the SMs, the fewer they are the longer K may be, and twice
//                  as long where the tiles here are wider than 128 tokens (int8 [300,8704] at 620 tokens, 30 tiles, 34.4 us here and 23.4
//                  there; [1024,4480] at 257, 40 tiles, 26 and 22, with 8704 inputs 33 and 35; [1024,1344] at 1143, 144 tiles, 18.8 and 14.6,
//                  with 4480 28.5 and 32.6; of 128 tokens [2048,8704] at 82 26 and 23.5, [5632,1344] 15.3 and 14.3, [4096,4480] 21 and 22;
//                  int4 [3584,20416] at 114 44 and 104; at 64 and below here throughout, [512,960] at 35 7.3 and 10).  Not up to eight
//                  (int8 [8192,7424] at six 19.5 us, 14.4 on the decode kernel).
//   fp32 results   per channel only where the other kernels need as many roundings: above 64 tokens, when the items fill
//                  half of the SMs (the other kernel needs a third limb per token there; int8 [28672,8192] at 512 tokens 219 us
//                  against 312, [2432,9248] at 763 tokens 49 against 74).
//   2..8 tokens    int8 on large weights: block 128 [28672,8192] at two tokens 44 us against 50, [14336,4096] at four 15 against
//                  17 (per channel 14 against 16).
//   9..32 tokens   weights of 34 million values, 2^24 in int8 blocks and from 17 tokens, 2^22 for int8 from 17: int4 block 128
//                  [14336,4096] at 16 tokens 14.3 us against 18.4, [4096,4096] at 24 11.4 against 12.2 (at 16 11.6 against 10.3); int8
//                  per channel [1024,4096] at 32 8.8 against 11.  From 2^27 values not int4 per channel, nor int8 from 2^28, where i8tc
//                  streams faster (int4 [28672,8192] 32 against 30).  Nor int4 blocks where i8tc takes them, from 2^26 values on: up to ten
//                  tokens from 80 million or with more weight tiles than SMs ([28672,8192] 40 against 31, block 128 [29741,3072] 18.6 against
//                  13.9, [11008,8192] 18.7 against 17.4; [8192,8192] 15.1 against 15.6), up to sixteen such tiles with long blocks (block 256
//                  [29741,3072] at 12 16.9 against 14.9; block 128 18.6 against 19.5).  i8tc leaves blocks of 64 and 384
//                  to the others: [39078,4288] block 64 at ten 43 against 81 on tcgen05, [57344,7680] block 384 at nine 70 against 122 on mma.
//   33..64 tokens  from 2^22 values int4, int8 blocks, and int8 per channel below 95 million: int4 block 128 [57344,8192] at 64 tokens 87 us
//                  against 104, [4096,4096] 15 against 16.5; int8 [5120,6912] 17 against 22, [28672,8192] 55 against 51.
//   above 64       int4 and int8 blocks, when the items fill half of the SMs (also with short K: [9728,1024] block 128 at 128 tokens 11 us
//                  against 15 for int8 and 17 for int4, [9728,512] 9 against 13 and 14), or 64 of them on weights of 2^25 values: fewer
//                  leave it to i8tc's narrower ones ([4096,4096] at 128 tokens 26 us against 19; [14336,4096] at 96 25
//                  against 34, [5120,6912] at 256 33 against 51, [28672,8192] at 512 230 against 337).  int4 per channel from 384
//                  tokens, where i8tc expands the weights once, on 2^25 values ([4096,4096] at 1024 50 us against 38; [5120,6912] at
//                  512 39 against 54), from 512 on fewer than 12288 outputs ([14336,4096] at 1024 117 against 94).
//   narrow int8    up to 2048 outputs and above the 1024 tokens of one launch of the other kernel, whose launches are then
//                  a round or two of items each (per channel [1536,14592] at 4178 tokens 189 us against 313, block 128 [1024,3968] at 1131 24
//                  against 46; with two limbs there, exact products here).
static bool use_tmem(int wbits, int64_t M, int64_t N, int64_t K, int64_t bs, int x_dt, int out_dt, bool has_zp, bool decode_i8) {
  if (!tmem_gemm_shape_ok(wbits, M, N, K, bs, x_dt)) return false;
  const bool blocked = bs > 0;
  const int64_t E = N * K, items = ceil_div(N, 128) * ceil_div(M, 192);
  if (has_zp) {
    if (blocked) return zp_decode_on_tc(wbits, M, N, K, bs, decode_i8);
    if (!limb_tc_shape_ok(wbits, M, N, K, bs, x_dt, true)) return zp_decode_on_tc(wbits, M, N, K, bs, decode_i8);
    if (M <= 8) return (wbits == 4 ? E < 1 << 27 : out_dt != QMM_F32) && zp_decode_on_tc(wbits, M, N, K, bs, decode_i8);
    if (M > 64 && wbits == 8) return items >= 64 && (K >= 4096 || (M > 1008 && N <= 4096));
    if (M > 64)
      return items >= 64 || out_dt == QMM_F32 || K >= 8192 || M > 1008 || (K >= 2048 && ceil_div(N, 128) * ceil_div(M, 42) > sm_count());
    return wbits == 4 ? M > 42 || E < 1 << 25 : M <= 32 || N >= 12288;
  }
  if (M == 1) return false;
  if (bs == 64 && M <= 8) return false;
  if (bs == 64 && M > 32) {
    const int64_t there = ceil_div(N, 128) * ceil_div(M, 64), sms = sm_count();
    const bool wide = ceil_div(M, ceil_div(M, 192)) > 128;
    return M <= 64 || there > sms || K > (4 * there <= sms ? 10000 : 2 * there <= sms ? 4000 : 1700) * (wide ? 2 : 1);
  }
  if (M <= 64) {
    if (out_dt == QMM_F32 && !blocked) return false;
    if (M > 32) return E >= 1 << 22 && (wbits == 4 || blocked || E < 95000000);
    if (int4_blocks_on_limbs(wbits, M, N, K, bs, x_dt)) return false;
    if (E >= 1 << 27) {
      if (blocked) return wbits == 8 || M > 8;
      return wbits == 8 && E < 1 << 28;
    }
    if (M > 16) return E >= (wbits == 8 ? 1 << 22 : 1 << 24);
    if (M > 8) return E >= (wbits == 8 && blocked ? 1 << 24 : 34000000);
    return wbits == 8 && E >= 34000000 && M >= (blocked ? 3 : 4);
  }
  const bool filled = 2 * items >= sm_count();
  if (out_dt == QMM_F32 && filled && (wbits == 8 || blocked || M < 384)) return true;
  if (wbits == 8 && M > 1024 && N <= 2048) return true;
  if (wbits == 8 && !blocked) return false;
  if (!blocked && M >= 384 && (E < 1 << 25 || (M >= 512 && N >= 12288))) return false;
  return filled || (items >= 64 && E >= 1 << 25);
}

// Where AUTO takes the split-activation kernel ahead of the decode kernels: zero points per channel at two to eight tokens (see
// above; where the integer decode kernel goes, on long rows and later: int8 [21601,2208] at eight 18.0 us, 16.0 there; [7864,8352] at three
// 18.2, 16.2 there, [10000,6000] at four even, at five 17.7, 18.7), and weights of 100 MB without at two to sixteen (int4 block 128
// [57344,8192] at two tokens 46 us against 53, at five 47 against 65; int8 [28672,8192] 41 against 48; at two tokens from 115 MB: int4
// [49152,4096] 20.8 against 17.8, [28672,8192] even).
static bool use_limb_decode(int wbits, int64_t M, int64_t N, int64_t K, int64_t bs, int x_dt, bool has_zp, bool decode_i8) {
  if (M < 2 || M > 16 || x_dt == QMM_F32 || bs == 64 || !limb_tc_shape_ok(wbits, M, N, K, bs, x_dt, has_zp)) return false;
  if (has_zp && decode_i8 && (K < 3072 || M * N * K < 260000000)) return false;
  if (has_zp) return M <= 8 && bs <= 0 && zp_decode_on_tc(wbits, M, N, K, bs, decode_i8);
  return N * K * wbits / 8 >= (M == 2 ? 115000000 : 100000000);
}

int qmm_w8a16_perchannel(const void* x, int x_dtype, const int8_t* w, const float* scale,
                         const float* zp, void* out, int out_dtype, int64_t M, int64_t N,
                         int64_t K, int variant, void* stream) {
  int rc = check_common(x, x_dtype, w, scale, out, out_dtype, M, N, K);
  if (rc != QMM_OK || M * N == 0) return rc;
  cudaStream_t st = as_stream(stream);
  if (variant == QMM_VARIANT_AUTO) variant = pick_weight_only(8, M, N, K, 0, x, x_dtype, w, zp != nullptr, device_is_sm100());
  switch (variant) {
    case QMM_VARIANT_GENERIC:
      log_choice("w8a16_perchannel", "generic", M, N, K);
      return launch_generic_nk(false, x, x_dtype, w, scale, zp, out, out_dtype, M, N, K, 0, st);
    case QMM_VARIANT_GEMV:
      log_choice("w8a16_perchannel", "gemv", M, N, K);
      return launch_gemv_nk(8, x, x_dtype, w, scale, zp, out, out_dtype, M, N, K, 0, st);
    case QMM_VARIANT_MMA:
      log_choice("w8a16_perchannel", "mma", M, N, K);
      if (zp) return fail(QMM_ERR_UNSUPPORTED, "the register-dequant decode kernel does not take a zero point");
      return launch_decode_mma(8, x, x_dtype, w, scale, QMM_F32, out, out_dtype, M, N, K, 0, st);
    case QMM_VARIANT_TCGEN05:
      log_choice("w8a16_perchannel", "tcgen05", M, N, K);
      if (zp) return fail(QMM_ERR_UNSUPPORTED, "tcgen05 weight-only kernel does not take a zero point");
      return launch_mixed_tc(8, x, x_dtype, w, scale, QMM_F32, out, out_dtype, M, N, K, 0, st);
    default:
      return fail(QMM_ERR_UNSUPPORTED, "unknown variant %d", variant);
  }
}

int qmm_blockwise_sbn(const void* x, int x_dtype, const int8_t* w, const float* scale,
                      const float* zp, void* out, int out_dtype, int64_t M, int64_t N, int64_t K,
                      int64_t block_size, int variant, void* stream) {
  int rc = check_common(x, x_dtype, w, scale, out, out_dtype, M, N, K);
  if (rc != QMM_OK) return rc;
  if (block_size <= 0 || K % block_size != 0)
    return fail(QMM_ERR_BAD_SHAPE, "input_dim should be divisible by block_size, got input_dim: %lld, block_size: %lld",
                (long long)K, (long long)block_size);
  if (M * N == 0) return QMM_OK;
  cudaStream_t st = as_stream(stream);
  // This layout (N minor) is served by the any-shape kernel only: the streaming kernels want K-minor rows, and the
  // callers above this entry convert a weight once (qmm_pack_int4_sbn, or a transposed copy) and keep it.
  if (variant != QMM_VARIANT_AUTO && variant != QMM_VARIANT_GENERIC)
    return fail(QMM_ERR_UNSUPPORTED, "blockwise_sbn: variant %d is not available for this layout", variant);
  log_choice("blockwise_sbn", "generic", M, N, K);
  return launch_generic_sbn(x, x_dtype, w, scale, zp, out, out_dtype, M, N, K, block_size, st);
}

int qmm_w4a16_blockwise_packed(const void* x, int x_dtype, const uint8_t* wp, const float* scale,
                               const float* zp, void* out, int out_dtype, int64_t M, int64_t N,
                               int64_t K, int64_t block_size, int variant, void* stream) {
  int rc = check_common(x, x_dtype, wp, scale, out, out_dtype, M, N, K);
  if (rc != QMM_OK) return rc;
  if (K % 2 != 0) return fail(QMM_ERR_BAD_SHAPE, "packed int4 needs an even K, got %lld", (long long)K);
  if (block_size <= 0 || K % block_size != 0)
    return fail(QMM_ERR_BAD_SHAPE, "input_dim should be divisible by block_size, got input_dim: %lld, block_size: %lld",
                (long long)K, (long long)block_size);
  if (M * N == 0) return QMM_OK;
  cudaStream_t st = as_stream(stream);
  if (variant == QMM_VARIANT_AUTO) variant = pick_weight_only(4, M, N, K, block_size, x, x_dtype, wp, zp != nullptr, device_is_sm100());
  switch (variant) {
    case QMM_VARIANT_GENERIC:
      log_choice("w4a16_blockwise_packed", "generic", M, N, K);
      return launch_generic_nk(true, x, x_dtype, wp, scale, zp, out, out_dtype, M, N, K, block_size, st);
    case QMM_VARIANT_GEMV:
      log_choice("w4a16_blockwise_packed", "gemv", M, N, K);
      return launch_gemv_nk(4, x, x_dtype, wp, scale, zp, out, out_dtype, M, N, K, block_size, st);
    case QMM_VARIANT_MMA:
      log_choice("w4a16_blockwise_packed", "mma", M, N, K);
      if (zp) return fail(QMM_ERR_UNSUPPORTED, "the register-dequant decode kernel does not take a zero point");
      return launch_decode_mma(4, x, x_dtype, wp, scale, QMM_F32, out, out_dtype, M, N, K, block_size, st);
    case QMM_VARIANT_TCGEN05:
      log_choice("w4a16_blockwise_packed", "tcgen05", M, N, K);
      if (zp) return fail(QMM_ERR_UNSUPPORTED, "tcgen05 weight-only kernel does not take a zero point");
      return launch_mixed_tc(4, x, x_dtype, wp, scale, QMM_F32, out, out_dtype, M, N, K, block_size, st);
    default:
      return fail(QMM_ERR_UNSUPPORTED, "unknown variant %d", variant);
  }
}

int qmm_w8a16_blockwise(const void* x, int x_dtype, const int8_t* w, const float* scale, const float* zp, void* out,
                        int out_dtype, int64_t M, int64_t N, int64_t K, int64_t block_size, int variant, void* stream) {
  int rc = check_common(x, x_dtype, w, scale, out, out_dtype, M, N, K);
  if (rc != QMM_OK) return rc;
  if (block_size <= 0 || K % block_size != 0)
    return fail(QMM_ERR_BAD_SHAPE, "input_dim should be divisible by block_size, got input_dim: %lld, block_size: %lld",
                (long long)K, (long long)block_size);
  if (M * N == 0) return QMM_OK;
  cudaStream_t st = as_stream(stream);
  if (variant == QMM_VARIANT_AUTO) variant = pick_weight_only(8, M, N, K, block_size, x, x_dtype, w, zp != nullptr, device_is_sm100());
  switch (variant) {
    case QMM_VARIANT_GENERIC:
      log_choice("w8a16_blockwise", "generic", M, N, K);
      return launch_generic_nk(false, x, x_dtype, w, scale, zp, out, out_dtype, M, N, K, block_size, st);
    case QMM_VARIANT_GEMV:
      log_choice("w8a16_blockwise", "gemv", M, N, K);
      return launch_gemv_nk(8, x, x_dtype, w, scale, zp, out, out_dtype, M, N, K, block_size, st);
    case QMM_VARIANT_MMA:
      log_choice("w8a16_blockwise", "mma", M, N, K);
      if (zp) return fail(QMM_ERR_UNSUPPORTED, "the register-dequant decode kernel does not take a zero point");
      return launch_decode_mma(8, x, x_dtype, w, scale, QMM_F32, out, out_dtype, M, N, K, block_size, st);
    case QMM_VARIANT_TCGEN05:
      log_choice("w8a16_blockwise", "tcgen05", M, N, K);
      if (zp) return fail(QMM_ERR_UNSUPPORTED, "tcgen05 weight-only kernel does not take a zero point");
      return launch_mixed_tc(8, x, x_dtype, w, scale, QMM_F32, out, out_dtype, M, N, K, block_size, st);
    default:
      return fail(QMM_ERR_UNSUPPORTED, "unknown variant %d", variant);
  }
}

// ---- tuned kernel choice ------------------------------------------------------------------------------------------
// The counterpart of the reference's TUNED_BLOCK_SIZES / get_tuned_block_sizes
// (torch_xla/experimental/pallas_kernels/quantized_matmul_kernel.py:326-555): measured on a B200 by xla_b200/tune.py.
namespace {
struct TunedRow {
  int wbits, block_size;
  int64_t N, K;
  unsigned char choice[7];  // QMM_VARIANT_* for M <= 1, 2, 4, 8, 16, 32, 64; 0 = not measured
};
const TunedRow kTuned[] = {
#include "tuned_table.inc"
    {0, 0, 0, 0, {0, 0, 0, 0, 0, 0, 0}},  // end
};

int tuned_variant(int wbits, int64_t block_size, int64_t M, int64_t N, int64_t K) {
  if (M < 1 || M > 64) return 0;
  int bucket = 0;
  while ((1 << bucket) < M) ++bucket;
  for (const TunedRow* r = kTuned; r->wbits; ++r)
    if (r->wbits == wbits && r->block_size == block_size && r->N == N && r->K == K) return r->choice[bucket];
  return 0;
}
}  // namespace

int qmm_tuned_variant(int wbits, int64_t M, int64_t N, int64_t K, int64_t block_size) {
  return tuned_variant(wbits, block_size < 0 ? 0 : block_size, M, N, K);
}

int qmm_zero_point_in_kernel(int wbits, int64_t M, int64_t N, int64_t K, int64_t block_size, int x_dtype) {
  if (block_size < 0) block_size = 0;
  const void* ok = reinterpret_cast<const void*>(uintptr_t(256));
  return M <= 8 || use_tmem(wbits, M, N, K, block_size, x_dtype, QMM_F32, true, false) || limb_tc_shape_ok(wbits, M, N, K, block_size, x_dtype, true) ||
         decode_i8_supported(wbits, M, N, K, block_size, ok, x_dtype, ok, true);
}

// qmm_weight_only's AUTO.  `room`: bytes of usable scratch.
static int choose_weight_only(int wbits, int64_t M, int64_t N, int64_t K, int64_t bs, const void* x, int x_dt, int out_dt, const void* w,
                              bool has_zp, size_t room, bool sm100) {
  if (M == 1 && use_decode_i8(wbits, M, N, K, bs, x, x_dt, w, has_zp)) return QMM_VARIANT_I8MMA;
  const bool tma = sm100 && aligned(x, 16) && aligned(w, 16);
  const bool decode_i8 = decode_i8_supported(wbits, M, N, K, bs, x, x_dt, w, has_zp);
  if (tma && use_tmem(wbits, M, N, K, bs, x_dt, out_dt, has_zp, decode_i8) && room >= tmem_gemm_workspace_bytes(M, K)) return QMM_VARIANT_TMEM;
  if (tma && use_limb_decode(wbits, M, N, K, bs, x_dt, has_zp, decode_i8) && room >= limb_tc_workspace_bytes(M, K)) return QMM_VARIANT_I8TC;
  if (use_decode_i8(wbits, M, N, K, bs, x, x_dt, w, has_zp)) return QMM_VARIANT_I8MMA;
  // the measured table first, the shape rule where the table has no entry for this shape
  const int tuned = tuned_variant(wbits, bs, M, N, K);
  if (tma && limb_tc_shape_ok(wbits, M, N, K, bs, x_dt, has_zp) && room >= limb_tc_workspace_bytes(M, K)) {
    bool use = tuned ? tuned == QMM_VARIANT_I8TC : limb_tc_preferred(wbits, M, N, K, bs);
    // Zero points and fp32 activations: the other kernels for more than a few tokens take neither, and the any-shape
    // kernel is a hundred times slower (333 tokens of fp32 on [5120,6912] int8 with zero points: 12.2 ms, here 52 us).
    // Up to eight tokens the register-dequant GEMV takes both.
    if (has_zp || x_dt == QMM_F32) use = M > 8;
    if (use) return QMM_VARIANT_I8TC;
  }
  if (!has_zp && tuned == QMM_VARIANT_MMA && decode_mma_supported(wbits, M, N, K, bs, x, x_dt, w, false)) return QMM_VARIANT_MMA;
  if (!has_zp && tuned == QMM_VARIANT_TCGEN05 && tma && mixed_tc_shape_ok(wbits, M, N, K, bs, x_dt, false)) return QMM_VARIANT_TCGEN05;
  return pick_weight_only(wbits, M, N, K, bs, x, x_dt, w, has_zp, sm100);
}

static const char* variant_name(int variant) {
  switch (variant) {
    case QMM_VARIANT_GEMV: return "gemv";
    case QMM_VARIANT_TCGEN05: return "tcgen05";
    case QMM_VARIANT_MMA: return "mma";
    case QMM_VARIANT_I8TC: return "i8tc";
    case QMM_VARIANT_I8MMA: return "i8mma";
    case QMM_VARIANT_TMEM: return "tmem";
    default: return "generic";
  }
}

// a 256-byte aligned address, for questions about a shape
static const void* any_pointer() { return reinterpret_cast<const void*>(uintptr_t(256)); }

const char* qmm_weight_only_variant_for(int wbits, int64_t M, int64_t N, int64_t K, int64_t block_size, int has_zp) {
  const void* ok = any_pointer();
  return variant_name(choose_weight_only(wbits, M, N, K, std::max<int64_t>(block_size, 0), ok, QMM_BF16, QMM_BF16, ok, has_zp != 0,
                                         SIZE_MAX, true));
}

size_t qmm_weight_only_workspace_size(int64_t max_M, int64_t K) {
  return std::max(limb_tc_workspace_bytes(max_M, K), tmem_gemm_workspace_bytes(max_M, K));
}

size_t qmm_weight_only_workspace_size_for(int wbits, int64_t max_M, int64_t N, int64_t K) {
  const size_t base = qmm_weight_only_workspace_size(max_M, K);
  if (base == 0 || N < 1) return base;
  return (base + 255) / 256 * 256 + limb_tc_wide_bytes(wbits, max_M, N, K);
}

int qmm_weight_only(int wbits, const void* x, int x_dtype, const void* w, const float* scale, const float* zp, void* out,
                    int out_dtype, int64_t M, int64_t N, int64_t K, int64_t block_size, int variant, void* workspace,
                    size_t workspace_bytes, void* stream) {
  return qmm_weight_only_typed(wbits, x, x_dtype, w, scale, zp, QMM_F32, out, out_dtype, M, N, K, block_size, variant, workspace,
                               workspace_bytes, stream);
}

int qmm_weight_only_typed(int wbits, const void* x, int x_dtype, const void* w, const void* scale, const void* zp, int scale_dtype,
                          void* out, int out_dtype, int64_t M, int64_t N, int64_t K, int64_t block_size, int variant,
                          void* workspace, size_t workspace_bytes, void* stream) {
  if (wbits != 4 && wbits != 8) return fail(QMM_ERR_BAD_SHAPE, "weight_only: wbits must be 4 or 8, got %d", wbits);
  if (!valid_float_dtype(scale_dtype)) return fail(QMM_ERR_UNSUPPORTED, "weight_only: bad scale dtype %d", scale_dtype);
  const Scales sc{scale, zp, scale_dtype};
  if (block_size < 0) block_size = 0;
  if (variant == QMM_VARIANT_AUTO || variant == QMM_VARIANT_I8TC) {
    int rc = check_common(x, x_dtype, w, scale, out, out_dtype, M, N, K);
    if (rc != QMM_OK || M * N == 0) return rc;
    if (block_size > 0 && K % block_size != 0)
      return fail(QMM_ERR_BAD_SHAPE, "input_dim should be divisible by block_size, got input_dim: %lld, block_size: %lld",
                  (long long)K, (long long)block_size);
    if (variant == QMM_VARIANT_AUTO)
      variant = choose_weight_only(wbits, M, N, K, block_size, x, x_dtype, out_dtype, w, zp != nullptr,
                                   workspace && aligned(workspace, 256) ? workspace_bytes : 0, device_is_sm100());
    if (variant == QMM_VARIANT_I8TC) {
      log_choice("weight_only", "i8tc", M, N, K);
      return launch_limb_tc(wbits, x, x_dtype, w, sc, out, out_dtype, M, N, K, block_size, 0, workspace, workspace_bytes,
                            as_stream(stream));
    }
  }
  if (variant == QMM_VARIANT_I8MMA) {
    int rc = check_common(x, x_dtype, w, scale, out, out_dtype, M, N, K);
    if (rc != QMM_OK || M * N == 0) return rc;
    log_choice("weight_only", "i8mma", M, N, K);
    return launch_decode_i8(wbits, x, x_dtype, w, sc, out, out_dtype, M, N, K, block_size, 0, as_stream(stream));
  }
  if (variant == QMM_VARIANT_TMEM) {
    int rc = check_common(x, x_dtype, w, scale, out, out_dtype, M, N, K);
    if (rc != QMM_OK || M * N == 0) return rc;
    log_choice("weight_only", "tmem", M, N, K);
    return launch_tmem_gemm(wbits, x, x_dtype, w, sc, out, out_dtype, M, N, K, block_size, 0, workspace, workspace_bytes,
                            as_stream(stream));
  }
  if (scale_dtype != QMM_F32) {
    // the entry points below read fp32 scales; the two kernels behind them that also take others are called here
    int rc = check_common(x, x_dtype, w, scale, out, out_dtype, M, N, K);
    if (rc != QMM_OK || M * N == 0) return rc;
    if (block_size > 0 && K % block_size != 0) return fail(QMM_ERR_BAD_SHAPE, "weight_only: block_size must divide K");
    if ((variant != QMM_VARIANT_MMA && variant != QMM_VARIANT_TCGEN05) || zp)
      return fail(QMM_ERR_UNSUPPORTED, "weight_only: variant %d reads fp32 scales only", variant);
    if (variant == QMM_VARIANT_TCGEN05) {
      log_choice("weight_only", "tcgen05", M, N, K);
      return launch_mixed_tc(wbits, x, x_dtype, w, scale, scale_dtype, out, out_dtype, M, N, K, block_size, as_stream(stream));
    }
    log_choice("weight_only", "mma", M, N, K);
    return launch_decode_mma(wbits, x, x_dtype, w, scale, scale_dtype, out, out_dtype, M, N, K, block_size, as_stream(stream));
  }
  const float *s32 = static_cast<const float*>(scale), *z32 = static_cast<const float*>(zp);
  if (wbits == 8) {
    if (block_size > 0)
      return qmm_w8a16_blockwise(x, x_dtype, static_cast<const int8_t*>(w), s32, z32, out, out_dtype, M, N, K, block_size, variant,
                                 stream);
    return qmm_w8a16_perchannel(x, x_dtype, static_cast<const int8_t*>(w), s32, z32, out, out_dtype, M, N, K, variant, stream);
  }
  if (block_size > 0)
    return qmm_w4a16_blockwise_packed(x, x_dtype, static_cast<const uint8_t*>(w), s32, z32, out, out_dtype, M, N, K, block_size,
                                      variant, stream);
  return qmm_w4a16_perchannel_packed(x, x_dtype, static_cast<const uint8_t*>(w), s32, z32, out, out_dtype, M, N, K, variant, stream);
}

int qmm_gate_up_decode(int wbits, const void* x, int x_dtype, const void* w, const float* scale, void* out,
                       int out_dtype, int64_t M, int64_t N2, int64_t K, int64_t block_size, void* stream) {
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (wbits != 4 && wbits != 8) return fail(QMM_ERR_BAD_SHAPE, "gate_up_decode: wbits must be 4 or 8, got %d", wbits);
  if (!x || !w || !scale || !out) return fail(QMM_ERR_NULL, "gate_up_decode: null pointer");
  if (M < 0 || N2 < 0 || K < 0) return fail(QMM_ERR_BAD_SHAPE, "gate_up_decode: negative size");
  if (N2 % 16 != 0) return fail(QMM_ERR_BAD_SHAPE, "gate_up_decode: N2 must be a multiple of 16, got %lld", (long long)N2);
  if (block_size < 0 || (block_size > 0 && K % block_size != 0))
    return fail(QMM_ERR_BAD_SHAPE, "gate_up_decode: K (%lld) must be a multiple of block_size (%lld)", (long long)K,
                (long long)block_size);
  if (M == 0 || N2 == 0) return QMM_OK;
  if (!decode_mma_supported(wbits, M, N2, K, block_size, x, x_dtype, w, false))
    return fail(QMM_ERR_UNSUPPORTED, "gate_up_decode: needs 1<=M<=32, bf16/f16 activations, K a multiple of %d, 16-byte "
                "aligned x/w (M=%lld N2=%lld K=%lld bs=%lld)", 512 / wbits, (long long)M, (long long)N2, (long long)K,
                (long long)block_size);
  if (use_decode_i8(wbits, M, N2, K, block_size, x, x_dtype, w, false)) {
    log_choice("gate_up_decode", "i8mma", M, N2, K);
    return launch_decode_i8(wbits, x, x_dtype, w, Scales{scale, nullptr, QMM_F32}, out, out_dtype, M, N2, K, block_size, 1, st);
  }
  log_choice("gate_up_decode", "mma", M, N2, K);
  return launch_decode_mma(wbits, x, x_dtype, w, scale, QMM_F32, out, out_dtype, M, N2, K, block_size, st, 1);
}

int qmm_gate_up_on_tensor_cores(int wbits, int x_dtype, int out_dtype, int64_t M, int64_t N2, int64_t K, int64_t block_size) {
  if (M > 32) return 1;
  if (wbits != 4 && wbits != 8) return 0;
  block_size = std::max<int64_t>(block_size, 0);
  return use_tmem(wbits, M, N2, K, block_size, x_dtype, out_dtype, false, false) || use_limb_decode(wbits, M, N2, K, block_size, x_dtype, false, false) ||
         (x_dtype != QMM_F32 && int4_blocks_on_limbs(wbits, M, N2, K, block_size, x_dtype));
}

int qmm_gate_up(int wbits, const void* x, int x_dtype, const void* w, const float* scale, void* out, int out_dtype, int64_t M,
                int64_t N2, int64_t K, int64_t block_size, void* workspace, size_t workspace_bytes, void* stream) {
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (wbits != 4 && wbits != 8) return fail(QMM_ERR_BAD_SHAPE, "gate_up: wbits must be 4 or 8, got %d", wbits);
  if (!x || !w || !scale || !out) return fail(QMM_ERR_NULL, "gate_up: null pointer");
  if (M < 0 || N2 < 0 || K < 0) return fail(QMM_ERR_BAD_SHAPE, "gate_up: negative size");
  if (N2 % 16 != 0) return fail(QMM_ERR_BAD_SHAPE, "gate_up: N2 must be a multiple of 16, got %lld", (long long)N2);
  if (block_size < 0 || (block_size > 0 && K % block_size != 0))
    return fail(QMM_ERR_BAD_SHAPE, "gate_up: K (%lld) must be a multiple of block_size (%lld)", (long long)K, (long long)block_size);
  if (M == 0 || N2 == 0) return QMM_OK;
  const Scales sc{scale, nullptr, QMM_F32};
  if (use_tmem(wbits, M, N2, K, block_size, x_dtype, out_dtype, false, false) && aligned(x, 16) && aligned(w, 16) && workspace &&
      workspace_bytes >= tmem_gemm_workspace_bytes(M, K)) {
    log_choice("gate_up", "tmem", M, N2, K);
    return launch_tmem_gemm(wbits, x, x_dtype, w, sc, out, out_dtype, M, N2, K, block_size, 1, workspace, workspace_bytes, st);
  }
  log_choice("gate_up", "i8tc", M, N2, K);
  return launch_limb_tc(wbits, x, x_dtype, w, sc, out, out_dtype, M, N2, K, block_size, 1, workspace, workspace_bytes, st);
}

int qmm_w4a16_perchannel_packed(const void* x, int x_dtype, const uint8_t* wp, const float* scale,
                                const float* zp, void* out, int out_dtype, int64_t M, int64_t N,
                                int64_t K, int variant, void* stream) {
  int rc = check_common(x, x_dtype, wp, scale, out, out_dtype, M, N, K);
  if (rc != QMM_OK) return rc;
  if (K % 2 != 0) return fail(QMM_ERR_BAD_SHAPE, "packed int4 needs an even K, got %lld", (long long)K);
  if (M * N == 0) return QMM_OK;
  cudaStream_t st = as_stream(stream);
  if (variant == QMM_VARIANT_AUTO) variant = pick_weight_only(4, M, N, K, 0, x, x_dtype, wp, zp != nullptr, device_is_sm100());
  switch (variant) {
    case QMM_VARIANT_GENERIC:
      log_choice("w4a16_perchannel_packed", "generic", M, N, K);
      return launch_generic_nk(true, x, x_dtype, wp, scale, zp, out, out_dtype, M, N, K, 0, st);
    case QMM_VARIANT_GEMV:
      log_choice("w4a16_perchannel_packed", "gemv", M, N, K);
      return launch_gemv_nk(4, x, x_dtype, wp, scale, zp, out, out_dtype, M, N, K, 0, st);
    case QMM_VARIANT_MMA:
      log_choice("w4a16_perchannel_packed", "mma", M, N, K);
      if (zp) return fail(QMM_ERR_UNSUPPORTED, "the register-dequant decode kernel does not take a zero point");
      return launch_decode_mma(4, x, x_dtype, wp, scale, QMM_F32, out, out_dtype, M, N, K, 0, st);
    case QMM_VARIANT_TCGEN05:
      log_choice("w4a16_perchannel_packed", "tcgen05", M, N, K);
      if (zp) return fail(QMM_ERR_UNSUPPORTED, "tcgen05 weight-only kernel does not take a zero point");
      return launch_mixed_tc(4, x, x_dtype, wp, scale, QMM_F32, out, out_dtype, M, N, K, 0, st);
    default:
      return fail(QMM_ERR_UNSUPPORTED, "unknown variant %d", variant);
  }
}

int qmm_quantize_activation(const void* x, int x_dtype, int8_t* xq, float* x_scale,
                            int32_t* xq_rowsum, int64_t M, int64_t K, int saturate, void* stream) {
  if (M < 0 || K < 0) return fail(QMM_ERR_BAD_SHAPE, "negative dimension");
  if (!valid_float_dtype(x_dtype)) return fail(QMM_ERR_UNSUPPORTED, "bad x dtype %d", x_dtype);
  if (M == 0) return QMM_OK;
  if (!x_scale || (K > 0 && (!x || !xq))) return fail(QMM_ERR_NULL, "x, xq or x_scale is NULL");
  return launch_quantize_activation(x, x_dtype, xq, x_scale, xq_rowsum, M, K, saturate, as_stream(stream));
}

static int w8a8_gemm(const int8_t* xq, const int8_t* w, const Scales& sc, const float* x_scale, const int32_t* xq_rowsum,
                     int32_t* acc_out, void* out, int out_dtype, int64_t M, int64_t N, int64_t K, int variant, cudaStream_t st) {
  if (variant == QMM_VARIANT_AUTO)
    variant = w8a8_tc_supported(M, N, K, xq, w) ? QMM_VARIANT_TCGEN05 : QMM_VARIANT_GENERIC;
  switch (variant) {
    case QMM_VARIANT_GENERIC:
      log_choice("w8a8_gemm", "generic", M, N, K);
      if (sc.dt != QMM_F32) return fail(QMM_ERR_UNSUPPORTED, "w8a8_gemm: the any-shape kernel reads fp32 scales only");
      return launch_generic_w8a8(xq, w, static_cast<const float*>(sc.scale), static_cast<const float*>(sc.zp), x_scale, xq_rowsum, acc_out,
                                 out, out_dtype, M, N, K, st);
    case QMM_VARIANT_TCGEN05:
      log_choice("w8a8_gemm", "tcgen05", M, N, K);
      if (!acc_out && w8a8_tc_supported(M, N, K, xq, w) && pair_gemm_preferred_w8a8(M, N, K, out_dtype))
        return launch_pair_gemm(1, w, xq, sc, x_scale, xq_rowsum, 1.f, out, out_dtype, M, N, K, N, 0, nullptr, nullptr, st);
      return launch_w8a8_tc(xq, w, sc, x_scale, xq_rowsum, acc_out, out, out_dtype, M, N, K, st);
    default:
      return fail(QMM_ERR_UNSUPPORTED, "w8a8_gemm: variant %d is not available", variant);
  }
}

int qmm_w8a8_gemm(const int8_t* xq, const int8_t* w, const float* w_scale, const float* zp,
                  const float* x_scale, const int32_t* xq_rowsum, int32_t* acc_out, void* out,
                  int out_dtype, int64_t M, int64_t N, int64_t K, int variant, void* stream) {
  if (M < 0 || N < 0 || K < 0) return fail(QMM_ERR_BAD_SHAPE, "negative dimension");
  if (M * N == 0) return QMM_OK;
  if (!acc_out && !out) return fail(QMM_ERR_NULL, "acc_out and out are both NULL");
  if (out && !valid_float_dtype(out_dtype)) return fail(QMM_ERR_UNSUPPORTED, "bad out dtype %d", out_dtype);
  if (out && (!w_scale || !x_scale)) return fail(QMM_ERR_NULL, "w_scale or x_scale is NULL");
  if (zp && !xq_rowsum) return fail(QMM_ERR_NULL, "a zero point needs xq_rowsum");
  if (K > 0 && (!xq || !w)) return fail(QMM_ERR_NULL, "xq or w is NULL");
  return w8a8_gemm(xq, w, Scales{w_scale, zp, QMM_F32}, x_scale, xq_rowsum, acc_out, out, out_dtype, M, N, K, variant, as_stream(stream));
}

// qmm_w8a8_perchannel's AUTO: I8MMA is the decode kernel, the others stand for the quantizer and that GEMM.
static int choose_w8a8(int64_t M, int64_t N, int64_t K, const void* x, int x_dt, const void* w, bool has_zp, bool sm100) {
  const int gemm = sm100 && K >= 16 && K % 16 == 0 && aligned(w, 16) ? QMM_VARIANT_TCGEN05 : QMM_VARIANT_GENERIC;
  if (decode_w8a8_supported(M, N, K, x, x_dt, w, has_zp)) return QMM_VARIANT_I8MMA;
  // Thirteen to fifteen tokens on a small weight with short rows and a row count that rules the GEMM's TMA stores out: the
  // any-shape kernel ([300,512] at 15 tokens 12.3 us, the GEMM 16.4).  Where N is a multiple of eight the GEMM is the faster
  // one ([512,512] 10.2 against 12.3, [2048,512] 10.2 against 16.4, [4096,256] 10.2 against 18.4), and up to twelve tokens
  // the decode kernel (9 tokens on [300,512] 8.5 against 12.3, on [2048,512] 10.6 against 14.3).
  if (M > 8 && M < 16 && N % 8 != 0 && K <= 512 && N * K <= (1 << 20)) return QMM_VARIANT_GENERIC;
  return gemm;
}

static size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

size_t qmm_workspace_size(int op, int64_t M, int64_t N, int64_t K) {
  (void)N;
  if (op == QMM_OP_W8A8_PERCHANNEL) {
    if (M <= 0 || K < 0) return 0;
    // xq [M,K] int8 | x_scale [M] f32 | rowsum [M] i32, each 256-byte aligned
    return align_up((size_t)M * (size_t)K, 256) + 2 * align_up((size_t)M * 4, 256);
  }
  return 0;
}

int qmm_w8a8_perchannel(const void* x, int x_dtype, const int8_t* w, const float* w_scale,
                        const float* zp, void* out, int out_dtype, int64_t M, int64_t N,
                        int64_t K, int saturate, int variant, void* workspace,
                        size_t workspace_bytes, void* stream) {
  return qmm_w8a8_perchannel_typed(x, x_dtype, w, w_scale, zp, QMM_F32, out, out_dtype, M, N, K, saturate, variant, workspace,
                                   workspace_bytes, stream);
}

int qmm_w8a8_perchannel_typed(const void* x, int x_dtype, const int8_t* w, const void* w_scale, const void* zp, int scale_dtype,
                              void* out, int out_dtype, int64_t M, int64_t N, int64_t K, int saturate, int variant,
                              void* workspace, size_t workspace_bytes, void* stream) {
  if (!valid_float_dtype(scale_dtype)) return fail(QMM_ERR_UNSUPPORTED, "w8a8_perchannel: bad scale dtype %d", scale_dtype);
  const Scales sc{w_scale, zp, scale_dtype};
  int rc = check_common(x, x_dtype, w, w_scale, out, out_dtype, M, N, K);
  if (rc != QMM_OK || M * N == 0) return rc;
  const bool any = variant == QMM_VARIANT_AUTO;
  if (any) variant = choose_w8a8(M, N, K, x, x_dtype, w, zp != nullptr, device_is_sm100());
  if (any && variant == QMM_VARIANT_I8MMA) {
    // one kernel quantizes and multiplies, no scratch
    log_choice("w8a8_perchannel", "i8mma", M, N, K);
    return launch_decode_w8a8(x, x_dtype, w, sc, out, out_dtype, M, N, K, saturate, as_stream(stream));
  }
  const size_t need = qmm_workspace_size(QMM_OP_W8A8_PERCHANNEL, M, N, K);
  if (!workspace || workspace_bytes < need)
    return fail(QMM_ERR_WORKSPACE, "w8a8_perchannel needs %zu bytes of workspace, got %zu", need, workspace_bytes);
  if (!aligned(workspace, 256)) return fail(QMM_ERR_MISALIGNED, "workspace must be 256-byte aligned");
  uint8_t* base = reinterpret_cast<uint8_t*>(workspace);
  int8_t* xq = reinterpret_cast<int8_t*>(base);
  float* xs = reinterpret_cast<float*>(base + align_up((size_t)M * (size_t)K, 256));
  int32_t* rowsum = reinterpret_cast<int32_t*>(reinterpret_cast<uint8_t*>(xs) + align_up((size_t)M * 4, 256));
  // (refused before the quantizer is launched)
  if (scale_dtype != QMM_F32 && (variant == QMM_VARIANT_GENERIC || !w8a8_tc_supported(M, N, K, xq, w)))
    return fail(QMM_ERR_UNSUPPORTED, "w8a8_perchannel: the any-shape kernel reads fp32 scales only");
  rc = qmm_quantize_activation(x, x_dtype, xq, xs, zp ? rowsum : nullptr, M, K, saturate, stream);
  if (rc != QMM_OK) return rc;
  return w8a8_gemm(xq, w, sc, xs, zp ? rowsum : nullptr, nullptr, out, out_dtype, M, N, K, variant, as_stream(stream));
}

int qmm_pack_int4_nk(const int8_t* w, uint8_t* wp, int64_t N, int64_t K, void* stream) {
  if (N < 0 || K < 0 || K % 2 != 0) return fail(QMM_ERR_BAD_SHAPE, "pack_int4_nk: K must be even and sizes non-negative");
  if (N * K == 0) return QMM_OK;
  if (!w || !wp) return fail(QMM_ERR_NULL, "w or wp is NULL");
  return launch_pack_int4_nk(w, wp, N, K, as_stream(stream));
}

int qmm_pack_int4_sbn(const int8_t* w, uint8_t* wp, int64_t S, int64_t block_size, int64_t N,
                      void* stream) {
  if (S < 0 || block_size < 0 || N < 0 || (S * block_size) % 2 != 0)
    return fail(QMM_ERR_BAD_SHAPE, "pack_int4_sbn: K = S*block_size must be even and sizes non-negative");
  if (S * block_size * N == 0) return QMM_OK;
  if (!w || !wp) return fail(QMM_ERR_NULL, "w or wp is NULL");
  return launch_pack_int4_sbn(w, wp, S, block_size, N, as_stream(stream));
}

int qmm_unpack_int4_nk(const uint8_t* wp, int8_t* w, int64_t N, int64_t K, void* stream) {
  if (N < 0 || K < 0 || K % 2 != 0) return fail(QMM_ERR_BAD_SHAPE, "unpack_int4_nk: K must be even and sizes non-negative");
  if (N * K == 0) return QMM_OK;
  if (!w || !wp) return fail(QMM_ERR_NULL, "w or wp is NULL");
  return launch_unpack_int4_nk(wp, w, N, K, as_stream(stream));
}

int qmm_peer_buffer_create(size_t bytes, void** ptr, unsigned char handle[64]) {
  if (!ptr || !handle) return fail(QMM_ERR_NULL, "peer_buffer_create: null pointer");
  static_assert(sizeof(cudaIpcMemHandle_t) == 64, "IPC handle size");
  void* p = nullptr;
  cudaError_t e = cudaMalloc(&p, bytes ? bytes : 16);
  if (e == cudaSuccess) e = cudaMemset(p, 0, bytes ? bytes : 16);
  cudaIpcMemHandle_t h;
  if (e == cudaSuccess) e = cudaIpcGetMemHandle(&h, p);
  if (e != cudaSuccess) {
    if (p) cudaFree(p);
    cudaGetLastError();
    return fail(QMM_ERR_DEVICE, "peer_buffer_create: %s", cudaGetErrorString(e));
  }
  memcpy(handle, &h, 64);
  *ptr = p;
  return QMM_OK;
}

int qmm_peer_buffer_open(const unsigned char handle[64], void** ptr) {
  if (!ptr || !handle) return fail(QMM_ERR_NULL, "peer_buffer_open: null pointer");
  cudaIpcMemHandle_t h;
  memcpy(&h, handle, 64);
  void* p = nullptr;
  cudaError_t e = cudaIpcOpenMemHandle(&p, h, cudaIpcMemLazyEnablePeerAccess);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(QMM_ERR_DEVICE, "peer_buffer_open: %s", cudaGetErrorString(e));
  }
  *ptr = p;
  return QMM_OK;
}

int qmm_peer_buffer_close(void* ptr) {
  if (!ptr) return QMM_OK;
  cudaError_t e = cudaIpcCloseMemHandle(ptr);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(QMM_ERR_DEVICE, "peer_buffer_close: %s", cudaGetErrorString(e));
  }
  return QMM_OK;
}

int qmm_peer_buffer_destroy(void* ptr) {
  if (!ptr) return QMM_OK;
  cudaError_t e = cudaFree(ptr);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(QMM_ERR_DEVICE, "peer_buffer_destroy: %s", cudaGetErrorString(e));
  }
  return QMM_OK;
}

int qmm_allreduce_oneshot(void* const* data_ptrs, void* const* flag_ptrs, int rank, int world, uint32_t epoch, void* out,
                          int out_dtype, int64_t count, void* stream) {
  if (!data_ptrs || !flag_ptrs || !out) return fail(QMM_ERR_NULL, "allreduce_oneshot: null pointer");
  if (out_dtype != QMM_F32 && out_dtype != QMM_BF16 && out_dtype != QMM_F16)
    return fail(QMM_ERR_BAD_SHAPE, "allreduce_oneshot: bad out_dtype %d", out_dtype);
  return launch_peer_allreduce(data_ptrs, flag_ptrs, rank, world, epoch, out, out_dtype, count, as_stream(stream));
}

size_t qmm_rowparallel_buffer_bytes(int64_t max_M, int64_t N, int world) {
  if (max_M < 1 || N < 1 || world < 1) return 0;
  const size_t data = 2 * (size_t)world * (size_t)max_M * (size_t)N * sizeof(float);
  const size_t flags = ((size_t)world * (size_t)((N + 15) / 16) + 2) * sizeof(uint32_t);
  return (data + flags + 255) / 256 * 256;
}

int qmm_rowparallel_decode(int wbits, const void* x, int x_dtype, const void* w, const float* scale, void* out,
                           int out_dtype, int64_t M, int64_t N, int64_t K, int64_t block_size,
                           void* const* peer_bufs, int rank, int world, int64_t slot_floats, void* stream) {
  if (wbits != 4 && wbits != 8) return fail(QMM_ERR_BAD_SHAPE, "rowparallel_decode: wbits must be 4 or 8, got %d", wbits);
  if (!x || !w || !scale || !out || !peer_bufs) return fail(QMM_ERR_NULL, "rowparallel_decode: null pointer");
  if (M < 0 || N < 0 || K < 0) return fail(QMM_ERR_BAD_SHAPE, "rowparallel_decode: negative size");
  if (block_size < 0 || (block_size > 0 && K % block_size != 0))
    return fail(QMM_ERR_BAD_SHAPE, "rowparallel_decode: K (%lld) must be a multiple of block_size (%lld)", (long long)K,
                (long long)block_size);
  if (out_dtype != QMM_F32 && out_dtype != QMM_BF16 && out_dtype != QMM_F16)
    return fail(QMM_ERR_BAD_SHAPE, "rowparallel_decode: bad out_dtype %d", out_dtype);
  if (M == 0 || N == 0) return QMM_OK;
  log_choice("rowparallel_decode", "mma", M, N, K);
  return launch_decode_mma_allreduce(wbits, x, x_dtype, w, scale, out, out_dtype, M, N, K, block_size, peer_bufs, rank, world,
                                     slot_floats, as_stream(stream));
}

int qmm_device_error_flag(uint32_t* flag, void* stream) {
  if (!flag) return fail(QMM_ERR_NULL, "flag is NULL");
  uint32_t* word = device_error_word();
  if (!word) return fail(QMM_ERR_DEVICE, "no CUDA device or error word unavailable");
  cudaStream_t st = as_stream(stream);
  cudaError_t e = cudaMemcpyAsync(flag, word, sizeof(uint32_t), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return fail(QMM_ERR_LAUNCH, "reading the device error word: %s", cudaGetErrorString(e));
  if (*flag != 0) {
    cudaMemsetAsync(word, 0, sizeof(uint32_t), st);
    return fail(QMM_ERR_TIMEOUT, "a device-side wait gave up (code %u, CTA %u)", *flag & 0xff, *flag >> 8);
  }
  return QMM_OK;
}

int qmm_stream_read(const void* p, size_t bytes, void* sink, void* stream) {
  return launch_stream_read(p, bytes, sink, as_stream(stream));
}

int qmm_set_activation_limbs(int limbs) {
  if (limbs != 0 && limbs != 3) return fail(QMM_ERR_BAD_SHAPE, "qmm_set_activation_limbs: 0 (by output type) or 3, got %d", limbs);
  limb_tc_set_limbs(limbs);
  return QMM_OK;
}

int qmm_set_peer_wait_limit(double seconds) {
  if (!(seconds > 0.0) || seconds > 60.0) return fail(QMM_ERR_BAD_SHAPE, "peer wait limit must be in (0, 60] seconds, got %g", seconds);
  g_peer_wait_cycles.store((long long)(seconds * 2.0e9), std::memory_order_relaxed);  // ~2 GHz SM clock
  return QMM_OK;
}

const char* qmm_variant_for(int op, int64_t M, int64_t N, int64_t K, int64_t block_size, int has_zp) {
  // Shape-only view of the AUTO heuristic (pointer alignment is assumed to be fine).
  const void* ok = any_pointer();
  switch (op) {
    case QMM_OP_W8A16_PERCHANNEL:
    case QMM_OP_W4A16_BLOCKWISE_PACKED:
    case QMM_OP_W4A16_PERCHANNEL_PACKED: {
      const int wbits = op == QMM_OP_W8A16_PERCHANNEL ? 8 : 4;
      const int64_t bs = op == QMM_OP_W4A16_BLOCKWISE_PACKED ? block_size : 0;
      return variant_name(pick_weight_only(wbits, M, N, K, bs, ok, QMM_BF16, ok, has_zp != 0, true));
    }
    case QMM_OP_BLOCKWISE_SBN:
      return "generic";
    case QMM_OP_W8A8_PERCHANNEL:
      return variant_name(choose_w8a8(M, N, K, ok, QMM_BF16, ok, has_zp != 0, true));
    default:
      return "generic";
  }
}

}  // extern "C"
