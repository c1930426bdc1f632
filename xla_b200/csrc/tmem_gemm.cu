// Weight-only linear for batches on the tensor cores, with the converted weights in tensor memory:
//
//   out[m,n] = sum_b (scale[b,n] * sum_{k in b} x[m,k] w[n,k] - zp[b,n] * sum_{k in b} x[m,k])     (per channel: one block)
//
// "Swap-AB": 128 weight rows are the MMA's M side, tokens its N side.  Integers of up to eight bits are exact in bf16 and
// f16, so the products are exact and the sums are the tensor core's fp32; block sums are scaled and added in fp32
// registers.  (The integer form, limb_gemm.cu, needs two limb columns per token for 16-bit outputs: the same tensor-core
// cycles, but twice the accumulator columns to read back and convert at every scale block.)
//
// What bounds this shape of kernel is the shared-memory port, 128 bytes a cycle for everything TMA writes and the MMA
// reads (limb_gemm.cu at 512 tokens, per channel: 1035 cycles per slot of 64 KB written and 64 KB read, exactly that).
// So the weights never go back to shared memory: converting warps read the raw bytes and write the bf16/f16 operand to
// tensor memory, where the MMA takes its A side from, and token tiles are as wide as two accumulators allow (192 columns:
// 96 KB of port traffic for the activations of a K step of 128, and 16 or 32 KB for the weights, against 768 cycles of
// MMAs).
//
//   warp 0        TMA: raw weight tiles, 128 rows x 128 bytes
//   warp 1        MMA issuer: per K step 8 (KS = 64: 4) x tcgen05.mma.kind::f16 (M128 x N<=192 x K16, A in tensor memory)
//                 and ONE commit, which everybody who needs the step's completion waits for; the next step's barriers are
//                 looked at before the current step is issued
//   warp 2        TMA: activation tiles, one K step x up to 192 tokens
//   warps 4..11   converters: two groups of four warps that take alternate K steps; lane = weight row
//   warps 12..19  drain: thread = weight row, half of the tokens in fp32 registers: tcgen05.ld, scale, add; epilogue
//
// Schedule: (weight tile, token tile) items walk the CTAs whole; the items of a partly filled last round (all of them
// when there are fewer items than SMs) are split along K over several CTAs and summed, in CTA order, from fp32 partial
// tiles in global scratch by the CTA that has the item's first K range.
//
// Semantics: torch_xla/experimental/xla_quantized_matmul.py:113-124, :152-170.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "common.cuh"
#include "kernels.h"
#include "ptx_sm100.cuh"

namespace qmm {

namespace {

constexpr int BMW = 128;                  // weight rows per tile (UMMA M)
constexpr uint32_t kRawBytes = BMW * 128; // one raw tile: 128 rows x 128 bytes
constexpr int kACols = 64;                // tensor-memory columns per operand step (32 are used for steps of 64 values)
constexpr int kDone = 8;                  // step-complete barriers
constexpr int kThreads = 640;
constexpr int kDrain = 256;               // drain threads
constexpr int kScaleRing = 8;             // folds whose scales (and zero points) are on their way
constexpr int kMiscRegs = 40, kConvRegs = 64, kDrainRegs = 152;  // x 128, 256, 256 threads: within 640 x 96
constexpr uint32_t kErrPartial = 10;      // owner CTA never saw a partial tile arrive

struct Params {
  const void* scale;   // [N] or [S,N], of type s_dt
  const void* zp;      // like scale, or null
  int s_dt;
  int64_t sc_pitch;    // bytes from one scale block to the next
  const float* xs;     // with zp: [S][xs_pitch] sums of the activations over each scale block
  int xs_pitch;
  void* out;
  int out_dt;
  int M;
  int64_t N;
  int stages;     // K steps per tile
  int fu;         // steps per fold (accumulation in the tensor core), >= 1
  int blocked;    // scale blocks (0: per channel; folds are then plain additions)
  int S;
  int ut;         // scheduling units (folds of fu steps) per tile
  int th;         // tokens per item (a multiple of 16)
  int ytiles;
  int items1;     // items handed out whole: CTA c takes c, c + G, ...
  int units;      // units of the remaining items, dealt in equal contiguous shares to the first g2 CTAs
  int g2;
  int gate_up;
  float* partial;   // [g2][th][128]
  uint32_t* flags;  // [g2], zero between launches
  uint32_t* err_word;
  long long wait_cycles;  // for a partial tile
};

// KS: k values per step (64 for scale blocks of 64, else 128); NC: accumulator columns (tokens).
template <int WBITS, int NC, int KS>
struct Cfg {
  static constexpr int kAcc = NC <= 64 ? 4 : 2;
  static constexpr int kASlots = NC == 192 ? 2 : 4;
  static constexpr int kACol0 = 512 - kASlots * kACols;
  static constexpr uint32_t kBStage = NC * KS * 2;
  static constexpr int kB = std::min(kDone, (NC == 192 ? 3 : NC == 128 ? 4 : NC == 64 ? 6 : 8) * (128 / KS));
  static constexpr int kRaw = NC == 192 ? 4 : NC == 128 ? 5 : NC == 64 ? 6 : 8;
  static constexpr int kSPR = 1024 / (WBITS * KS);  // K steps per raw tile
  static constexpr int kDT = NC / 2;                // tokens per drain thread
  static constexpr size_t kScaleBytes = 2 * kScaleRing * kDrain * 4;
  static constexpr size_t kSmem = 1024 + (size_t)kRaw * kRawBytes + (size_t)kB * kBStage + kScaleBytes + 512;
  static_assert(kAcc * NC <= kACol0, "tensor memory");
  static_assert(kSmem <= 227 * 1024, "shared memory budget");
  // A parity wait is right only while the barrier is at most one phase away: whoever waits for step i - d does so for every
  // step in turn, and step i - d + kDone cannot complete before it has gone on.
  static_assert(kB <= kDone && kASlots <= kDone && kAcc <= kDone, "step-complete barriers");
  static_assert((2 * kRaw + kB + kASlots + 2 * kAcc + kDone) * 8 + 8 <= 512, "barrier space");
};

// The (item, unit range) fragments of this CTA, in order: whole items first, then its share of the dealt units.  These go to
// the CTAs from the last one down, so that a CTA waits only for partial tiles of CTAs with lower indices: CTAs start in the
// order of their indices, so those run already or are done, also when another launch holds a part of the SMs.
__device__ __forceinline__ int deal_place(const Params& p) { return p.g2 - 1 - (int)blockIdx.x; }

struct FragIter {
  const Params& p;
  int u, hi, nxt, item, tile, y, u0, u1;
  __device__ explicit FragIter(const Params& p) : p(p), nxt(blockIdx.x), item(0), tile(0), y(0), u0(0), u1(0) {
    const int c = deal_place(p);
    u = c >= 0 ? share(c) : 0;
    hi = c >= 0 ? share(c + 1) : 0;
  }
  __device__ int share(int c) const { return (int)((long long)c * p.units / p.g2); }
  __device__ bool next() {
    if (nxt < p.items1) {
      item = nxt;
      nxt += gridDim.x;
      u0 = 0;
      u1 = p.ut;
    } else {
      if (u >= hi) return false;
      const int rel = u / p.ut;
      item = p.items1 + rel;
      u0 = u - rel * p.ut;
      u1 = min(p.ut, u0 + (hi - u));
      u += u1 - u0;
    }
    tile = item / p.ytiles;
    y = item - tile * p.ytiles;
    return true;
  }
  __device__ int s0() const { return u0 * p.fu; }
  __device__ int s1() const { return min(p.stages, u1 * p.fu); }
};

__device__ __forceinline__ uint4 lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}

template <typename XT>
__device__ __forceinline__ uint32_t sub2(uint32_t a, uint32_t b) {
  if constexpr (std::is_same<XT, __half>::value) {
    const __half2 r = __hsub2(*reinterpret_cast<const __half2*>(&a), *reinterpret_cast<const __half2*>(&b));
    return *reinterpret_cast<const uint32_t*>(&r);
  } else {
    const __nv_bfloat162 r = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
    return *reinterpret_cast<const uint32_t*>(&r);
  }
}

// Eight nibbles -> four pairs in k order.  Offset-binary nibbles are spread to bytes, put under the exponent byte of 128
// (bf16) or 1024 (f16), and the offset is subtracted (exact).
template <typename XT>
__device__ __forceinline__ void cvt_s4x8(uint32_t w, uint32_t* p) {
  constexpr bool kHalf = std::is_same<XT, __half>::value;
  constexpr uint32_t expo = kHalf ? 0x64646464u : 0x43434343u, bias = kHalf ? 0x64086408u : 0x43084308u;
  const uint32_t lo = (w & 0x0F0F0F0Fu) ^ 0x08080808u, hi = ((w >> 4) & 0x0F0F0F0Fu) ^ 0x08080808u;
  const uint32_t q0 = __byte_perm(lo, hi, 0x5140), q1 = __byte_perm(lo, hi, 0x7362);
  p[0] = sub2<XT>(__byte_perm(q0, expo, 0x4140), bias);
  p[1] = sub2<XT>(__byte_perm(q0, expo, 0x4342), bias);
  p[2] = sub2<XT>(__byte_perm(q1, expo, 0x4140), bias);
  p[3] = sub2<XT>(__byte_perm(q1, expo, 0x4342), bias);
}

// Four bytes -> two pairs in k order.  f16: the offset-binary byte under the exponent of 1024, minus 1152.  bf16 holds
// seven bits under an exponent: the low seven go under 128, and the sign bit, which is the lowest exponent bit, makes
// the subtrahend 128 or 256.
template <typename XT>
__device__ __forceinline__ void cvt_s8x4(uint32_t w, uint32_t* p) {
  if constexpr (std::is_same<XT, __half>::value) {
    const uint32_t u = w ^ 0x80808080u;
    p[0] = sub2<XT>(__byte_perm(u, 0x64646464u, 0x4140), 0x64806480u);
    p[1] = sub2<XT>(__byte_perm(u, 0x64646464u, 0x4342), 0x64806480u);
  } else {
    const uint32_t t0 = __byte_perm(w, 0u, 0x4140), t1 = __byte_perm(w, 0u, 0x4342);
    p[0] = sub2<XT>((t0 & 0x007F007Fu) | 0x43004300u, (t0 & 0x00800080u) | 0x43004300u);
    p[1] = sub2<XT>((t1 & 0x007F007Fu) | 0x43004300u, (t1 & 0x00800080u) | 0x43004300u);
  }
}

// Sixteen tokens of one output column, `pitch` elements apart
template <typename OT>
__device__ __forceinline__ void store16_as(OT* o, int64_t pitch, const float* v, int count) {
#pragma unroll
  for (int t = 0; t < 16; ++t)
    if (t < count) o[t * pitch] = from_f32<OT>(v[t]);
}
__device__ __forceinline__ void store16(void* out, int dt, int64_t at, int64_t pitch, const float* v, int count) {
  if (dt == QMM_BF16) store16_as(reinterpret_cast<__nv_bfloat16*>(out) + at, pitch, v, count);
  else if (dt == QMM_F16) store16_as(reinterpret_cast<__half*>(out) + at, pitch, v, count);
  else store16_as(reinterpret_cast<float*>(out) + at, pitch, v, count);
}

template <int REGS>
__device__ __forceinline__ void reg_inc() {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGS));
}
template <int REGS>
__device__ __forceinline__ void reg_dec() {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS));
}

template <int WBITS, typename XT, int NC, int KS, bool W16>
__global__ void __launch_bounds__(kThreads, 1)
    tmem_gemm_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const Params p) {
  using C = Cfg<WBITS, NC, KS>;
  constexpr int kRaw = C::kRaw, kB = C::kB, kAcc = C::kAcc, DT = C::kDT, kASlots = C::kASlots, kSPR = C::kSPR;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* raw_base = smem;
  uint8_t* b_base = raw_base + (size_t)kRaw * kRawBytes;
  uint32_t* s_scale = reinterpret_cast<uint32_t*>(b_base + (size_t)kB * C::kBStage);  // [scale, zero point][kScaleRing][kDrain]
  uint64_t* bars = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(s_scale) + C::kScaleBytes);
  uint64_t* raw_full = bars;                 // [kRaw]    TMA bytes
  uint64_t* raw_empty = raw_full + kRaw;     // [kRaw]    the converting warps that share the tile
  uint64_t* b_full = raw_empty + kRaw;       // [kB]      TMA bytes
  uint64_t* a_full = b_full + kB;            // [kASlots] the four converting warps of the step's group
  uint64_t* acc_empty = a_full + kASlots;    // [kAcc]    eight drain warps
  uint64_t* acc_full = acc_empty + kAcc;     // [kAcc]    tcgen05.commit, folds of several steps only
  uint64_t* done = acc_full + kAcc;          // [kDone]   tcgen05.commit: the MMAs of step i are complete
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + kDone);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = ptx::warp_index(), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kRaw; ++s) {
      ptx::mbar_init(&raw_full[s], 1);
      ptx::mbar_init(&raw_empty[s], kSPR == 1 ? 4 : 8);
    }
    for (int s = 0; s < kB; ++s) ptx::mbar_init(&b_full[s], 1);
    for (int s = 0; s < kASlots; ++s) ptx::mbar_init(&a_full[s], 4);
    for (int s = 0; s < kAcc; ++s) {
      ptx::mbar_init(&acc_empty[s], 8);
      ptx::mbar_init(&acc_full[s], 1);
    }
    for (int s = 0; s < kDone; ++s) ptx::mbar_init(&done[s], 1);
    *abort_flag = 0;
    ptx::fence_mbar_init();
    ptx::prefetch_tensormap(&map_w);
    ptx::prefetch_tensormap(&map_x);
  }
  if (warp == 3) {
    ptx::tmem_alloc(tmem_slot, 512);
    ptx::tmem_relinquish();
  }
  ptx::tcgen05_fence_before();
  __syncthreads();
  ptx::tcgen05_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  if (warp < 4) {
    reg_dec<kMiscRegs>();
    FragIter it(p);
    if (warp == 0) {
      // ---------------- raw weight producer: static data, no wait for earlier kernels ----------------
      if (lane == 0) {
        int slot = 0;
        uint32_t ph = 0;
        while (it.next()) {
          const int s0 = it.s0(), s1 = it.s1();
          for (int s = s0; s < s1; s += kSPR) {
            ptx::mbar_wait(&raw_empty[slot], ph ^ 1, abort_flag, p.err_word, ptx::kErrWaitEmpty);
            ptx::mbar_expect_tx(&raw_full[slot], kRawBytes);
            ptx::tma_load_2d(raw_base + (size_t)slot * kRawBytes, &map_w, &raw_full[slot], s * (KS * WBITS / 8), it.tile * BMW);
            if (++slot == kRaw) { slot = 0; ph ^= 1; }
          }
        }
      }
    } else if (warp == 2) {
      // ---------------- activation producer ----------------
      if (lane == 0) {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        int slot = 0;
        uint32_t i = 0;
        while (it.next()) {
          const int s0 = it.s0(), s1 = it.s1();
          for (int s = s0; s < s1; ++s, ++i) {
            if (i >= (uint32_t)kB)
              ptx::mbar_wait(&done[(i - kB) % kDone], ((i - kB) / kDone) & 1, abort_flag, p.err_word, ptx::kErrWaitEmpty);
            ptx::mbar_expect_tx(&b_full[slot], (uint32_t)p.th * KS * 2);
            uint8_t* dst = b_base + (size_t)slot * C::kBStage;
#pragma unroll
            for (int h = 0; h < KS / 64; ++h)
              ptx::tma_load_2d(dst + h * (NC * 128), &map_x, &b_full[slot], s * KS + h * 64, it.y * p.th);
            if (++slot == kB) slot = 0;
          }
        }
      }
    } else if (warp == 1) {
      // ---------------- MMA issuer: the whole warp walks the loop, one elected thread issues ----------------
      constexpr uint32_t fmt = std::is_same<XT, __half>::value ? 0u : 1u;
      const uint32_t idesc = ptx::make_idesc(/*f32*/ 1, fmt, fmt, BMW, (uint32_t)p.th);
      // Operands of the MMA live in uniform registers.  What the compiler cannot see to be the same in all lanes (a value
      // from shared memory, a branch on a predicate computed earlier) is moved there again for every MMA: int4 block 128
      // [28672,8192] at 512 tokens 285 us moved every time, 266 so.
      const uint32_t tb = __reduce_or_sync(0xffffffffu, tmem_base);
      const uint32_t desc_hi = (uint32_t)(ptx::make_sw128_kmajor_desc(0) >> 32);
      const uint32_t b_lo0 = (uint32_t)ptx::make_sw128_kmajor_desc(ptx::smem_u32(b_base));
      int sa = 0, sb = 0, buf = 0, dn = 0;
      uint32_t pa = 0, pb = 0, pacc = 1;
      bool ready = false;  // the barriers of the coming step were seen complete
      while (it.next()) {
        const int s0 = it.s0(), s1 = it.s1();
        int in_fold = 0;
        for (int s = s0; s < s1; ++s) {
          if (!__all_sync(0xffffffffu, ready)) {
            if (in_fold == 0) ptx::mbar_wait(&acc_empty[buf], pacc, abort_flag, p.err_word, ptx::kErrWaitTmemEmpty);
            ptx::mbar_wait(&b_full[sb], pb, abort_flag, p.err_word, ptx::kErrWaitFull);
            ptx::mbar_wait(&a_full[sa], pa, abort_flag, p.err_word, ptx::kErrWaitConv);
          }
          ptx::tcgen05_fence_after();
          const uint32_t d = tb + buf * NC, a = tb + C::kACol0 + sa * kACols;
          const uint32_t lo = b_lo0 + (uint32_t)sb * (C::kBStage >> 4);
          const uint32_t acc0 = in_fold != 0 ? 1u : 0u;
          const int buf_now = buf, dn_now = dn;
          const bool last = ++in_fold == p.fu || s + 1 == s1;
          if (++sa == kASlots) { sa = 0; pa ^= 1; }
          if (++sb == kB) { sb = 0; pb ^= 1; }
          if (++dn == kDone) dn = 0;
          if (last) {
            in_fold = 0;
            if (++buf == kAcc) { buf = 0; pacc ^= 1; }
          }
          ready = ptx::mbar_test_wait(&a_full[sa], pa) & ptx::mbar_test_wait(&b_full[sb], pb) &
                  (!last | ptx::mbar_test_wait(&acc_empty[buf], pacc));
          if (ptx::elect_one()) {
#pragma unroll
            for (int k = 0; k < KS / 16; ++k)
              ptx::mma_f16_ts(d, a + k * 8, ((uint64_t)desc_hi << 32) | (uint64_t)(lo + (k >> 2) * (NC * 128 >> 4) + (k & 3) * 2), idesc,
                              acc0 | (uint32_t)k);
            ptx::mma_commit(&done[dn_now]);
            if (last && p.fu > 1) ptx::mma_commit(&acc_full[buf_now]);
          }
        }
      }
    }
    __syncwarp();
  } else if (warp < 12) {
    // ---------------- converters: lane = weight row; group g takes the steps of its parity ----------------
    reg_dec<kConvRegs>();
    const int quad = warp & 3, grp = (warp - 4) >> 2;
    const int r = quad * 32 + lane;
    const uint32_t sw = (uint32_t)(r & 7);
    const uint32_t raw_row = ptx::smem_u32(raw_base) + r * 128;
    const uint32_t t_row = tmem_base + ((uint32_t)(quad * 32) << 16) + C::kACol0;
    constexpr int kPieces = KS * WBITS / 8 / 16;  // 16-byte pieces of a row per step: 2, 4 or 8
    FragIter it(p);
    int rs = 0;
    uint32_t rph = 0, i = 0;
    while (it.next()) {
      const int s0 = it.s0(), s1 = it.s1();
      for (int s = s0; s < s1; s += kSPR) {
        if (kSPR > 1 || (int)(i & 1) == grp) {
          ptx::mbar_wait_warp(&raw_full[rs], rph, abort_flag, p.err_word, ptx::kErrWaitRaw);
          const uint32_t row = raw_row + rs * kRawBytes;
#pragma unroll 1
          for (int q = 0; q < kSPR; ++q) {
            const uint32_t j = i + q;
            if (s + q >= s1 || (int)(j & 1) != grp) continue;
            auto piece = [&](int c) { return lds128(row + (((uint32_t)(q * kPieces + c) ^ sw) << 4)); };
            uint4 v = piece(0);
            // the MMAs that read this operand slot last are complete
            if (j >= (uint32_t)kASlots)
              ptx::mbar_wait_warp(&done[(j - kASlots) % kDone], ((j - kASlots) / kDone) & 1, abort_flag, p.err_word, ptx::kErrWaitEmpty);
            ptx::tcgen05_fence_after();
            uint32_t t = t_row + (j % kASlots) * kACols;
            // Rolled: the three kinds of warps of a scheduler share its instruction cache, and this body is the longest.
#pragma unroll 1
            for (int c = 0; c < kPieces; ++c) {
              const uint4 nx = piece(min(c + 1, kPieces - 1));
              uint32_t o[16];
              if constexpr (WBITS == 4) {
                cvt_s4x8<XT>(v.x, o);
                cvt_s4x8<XT>(v.y, o + 4);
                cvt_s4x8<XT>(v.z, o + 8);
                cvt_s4x8<XT>(v.w, o + 12);
                ptx::tmem_st_32x32b_x16(t, o);
                t += 16;
              } else {
                cvt_s8x4<XT>(v.x, o);
                cvt_s8x4<XT>(v.y, o + 2);
                cvt_s8x4<XT>(v.z, o + 4);
                cvt_s8x4<XT>(v.w, o + 6);
                ptx::tmem_st_32x32b_x8(t, o);
                t += 8;
              }
              v = nx;
            }
            ptx::tmem_st_wait();
            ptx::tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(&a_full[j % kASlots]);
          }
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(&raw_empty[rs]);
        }
        i += min(kSPR, s1 - s);
        if (++rs == kRaw) { rs = 0; rph ^= 1; }
      }
    }
  } else {
    // ---------------- drain: thread = weight row (its TMEM lane), half of the item's tokens ----------------
    reg_inc<kDrainRegs>();
    const int quad = warp & 3, grp = (warp - 12) >> 2;
    const int rl = quad * 32 + lane;
    const int dt = (int)threadIdx.x - 12 * 32;  // 0..255
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quad * 32) << 16) + grp * DT;
    auto drain_bar = [&]() { asm volatile("bar.sync 1, 256;" ::: "memory"); };
    __shared__ int s_npart;
    const uint32_t* my_scale = s_scale + dt;
    const uint32_t my_scale_u32 = ptx::smem_u32(my_scale);
    // (a tile starts at an even row)
    auto value = [&](int i, int f) { return scale_in<W16, XT>(my_scale + i * kDrain, rl, f, (int)p.N, p.s_dt); };
    const int place = deal_place(p);
    bool waited = false;
    FragIter it(p);
    int buf = 0;
    uint32_t i = 0, pacc = 0;
    while (it.next()) {
      const int64_t n = (int64_t)it.tile * BMW + rl;
      const bool n_ok = n < p.N;
      const bool first = it.u0 == 0, last = it.u1 == p.ut;
      const int m0 = it.y * p.th + grp * DT;                      // first token of this thread
      const int mcount = min(p.M - m0, min(DT, p.th - grp * DT)); // its tokens
      float total[DT];
#pragma unroll
      for (int t = 0; t < DT; ++t) total[t] = 0.f;
      // Block scales and zero points are a stream of their own (a round trip to HBM each): every thread copies its own
      // row's, seven folds ahead, into a ring of its own.  (Held in registers that shift from fold to fold, the shift
      // waits for the load of the fold before, whatever the nominal distance.)
      const int64_t sc_off = min(n, p.N - 1) * (W16 ? 2 : 4);
      const uint8_t* scp = static_cast<const uint8_t*>(p.scale) + sc_off;
      const uint8_t* zpp = static_cast<const uint8_t*>(p.zp) + sc_off;
      auto fetch = [&](int f) {
        if (p.blocked && f < it.u1) {
          const uint32_t dst = my_scale_u32 + (uint32_t)(f % kScaleRing) * (kDrain * 4);
          copy_scale_word<W16>(dst, scp + f * p.sc_pitch);
          if (p.zp) copy_scale_word<W16>(dst + kScaleRing * kDrain * 4, zpp + f * p.sc_pitch);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
      };
      if (!waited) {
        // scales (a conversion may be the kernel in front), block sums, scratch and `out` belong to earlier kernels until here
        asm volatile("griddepcontrol.wait;" ::: "memory");
        waited = true;
      }
#pragma unroll 1
      for (int f = 0; f < kScaleRing - 1; ++f) fetch(it.u0 + f);
      for (int f = it.u0; f < it.u1; ++f) {
        fetch(f + kScaleRing - 1);
        if (p.fu == 1) {
          ptx::mbar_wait_warp(&done[i % kDone], (i / kDone) & 1, abort_flag, p.err_word, ptx::kErrWaitTmemFull);
          ++i;
        } else {
          ptx::mbar_wait_warp(&acc_full[buf], pacc, abort_flag, p.err_word, ptx::kErrWaitTmemFull);
        }
        ptx::tcgen05_fence_after();
        const uint32_t a = lane_addr + buf * NC;
        // the next sixteen columns are on their way while the current ones are added
        uint32_t r[2][16];
        ptx::tmem_ld_32x32b_x16(a, r[0]);
        asm volatile("cp.async.wait_group %0;" ::"n"(kScaleRing - 1) : "memory");
        const float sc = p.blocked ? value(f % kScaleRing, f) : 1.f;
#pragma unroll
        for (int c = 0; c < DT / 16; ++c) {
          uint32_t* cur = r[c & 1];
          ptx::tmem_ld_wait();
          ptx::tmem_ld_landed16(cur);
          if (c + 1 < DT / 16) {
            ptx::tmem_ld_32x32b_x16(a + 16 * (c + 1), r[(c + 1) & 1]);
          } else {
            ptx::tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(&acc_empty[buf]);
          }
#pragma unroll
          for (int t = 0; t < 16; ++t) total[16 * c + t] = fmaf(sc, __uint_as_float(cur[t]), total[16 * c + t]);
        }
        if (++buf == kAcc) {
          buf = 0;
          pacc ^= 1;
        }
        if (p.blocked && p.zp) {
          const float z = -value(kScaleRing + f % kScaleRing, f);
          const float* xs = p.xs + (int64_t)f * p.xs_pitch + m0;  // the same for all lanes; the pitch covers whole tiles
#pragma unroll
          for (int t = 0; t < DT; t += 4) {
            const float4 v = ld_ordered(reinterpret_cast<const float4*>(xs + t));
            total[t] = fmaf(z, v.x, total[t]);
            total[t + 1] = fmaf(z, v.y, total[t + 1]);
            total[t + 2] = fmaf(z, v.z, total[t + 2]);
            total[t + 3] = fmaf(z, v.w, total[t + 3]);
          }
        }
      }
      // ---- end of the fragment ----
      // Sixteen tokens at a time in a rolled loop that rotates the sums through the first sixteen registers: unrolled over
      // all tokens this part is tens of kilobytes of code that runs once per item, and fetching it took 10 to 30 us.
      int np = 0;
      if (first && !last) {
        // the sums of the CTAs that continue the item are added in CTA order, once they are all there
        if (dt == 0) {
          int cnt = 0;
          for (int c2 = place + 1; c2 < p.g2; ++c2) {
            if (it.share(c2) >= (it.item - p.items1 + 1) * p.ut) break;
            ++cnt;
          }
          s_npart = cnt;
        }
        drain_bar();
        np = s_npart;
        for (int j = dt; j < np; j += 256) {
          ptx::partial_wait(p.flags + place + 1 + j, p.wait_cycles, abort_flag, p.err_word, kErrPartial);
        }
        drain_bar();
      }
      const bool lost = *abort_flag != 0;  // a wait ran out: NaN, not what is there
      const float ps = p.blocked || !n_ok ? 1.f : scale_value(load_scale_bits(p.scale, n, p.s_dt), p.s_dt);
      const float z1 = !p.blocked && p.zp && n_ok ? -scale_value(load_scale_bits(p.zp, n, p.s_dt), p.s_dt) : 0.f;
#pragma unroll 1
      for (int c = 0; c < DT / 16; ++c) {
        const int l0 = grp * DT + 16 * c;  // token inside the item
        const int count = min(16, mcount - 16 * c);
        if (lost) {
#pragma unroll
          for (int t = 0; t < 16; ++t) total[t] = __uint_as_float(0x7fc00000u);
        }
        if (!first) {
          // a later K range of an item that another CTA started: leave the sums for that CTA
          float* dst = p.partial + ((size_t)place * p.th + l0) * BMW + rl;
#pragma unroll
          for (int t = 0; t < 16; ++t)
            if (t < count) __stcg(dst + t * BMW, total[t]);
        } else {
#pragma unroll 1
          for (int j = 0; j < np; ++j) {
            const float* src = p.partial + ((size_t)(place + 1 + j) * p.th + l0) * BMW + rl;
            float v[16];
#pragma unroll
            for (int t = 0; t < 16; ++t) v[t] = t < count ? __ldcg(src + t * BMW) : 0.f;
#pragma unroll
            for (int t = 0; t < 16; ++t) total[t] += v[t];
          }
          if (!p.blocked) {
#pragma unroll
            for (int t = 0; t < 16; ++t) {
              total[t] *= ps;
              if (p.zp && t < count) total[t] = fmaf(z1, ld_ordered(p.xs + m0 + 16 * c + t), total[t]);
            }
          }
          const int64_t row_out = m0 + 16 * c;
          if (!p.gate_up) {
            store16(p.out, p.out_dt, row_out * p.N + n, p.N, total, n_ok ? count : 0);
          } else {
            // rows come in groups of 16: eight gate rows, then the eight up rows of the same outputs
            float v[16];
#pragma unroll
            for (int t = 0; t < 16; ++t) {
              const float u = __shfl_down_sync(0xffffffffu, total[t], 8);
              v[t] = total[t] / (1.f + expf(-total[t])) * u;
            }
            store16(p.out, p.out_dt, row_out * (p.N >> 1) + ((n >> 4) << 3) + (n & 7), p.N >> 1, v, n_ok && (rl & 8) == 0 ? count : 0);
          }
        }
#pragma unroll
        for (int t = 0; t + 16 < DT; ++t) total[t] = total[t + 16];
      }
      if (!first) {
        drain_bar();  // orders every drain thread's stores before thread 0's fence, which is cumulative
        if (dt == 0) ptx::partial_publish(p.flags + place);
      }
      asm volatile("cp.async.wait_group 0;" ::: "memory");  // the ring is refilled from its start
    }
  }

  ptx::tcgen05_fence_before();
  __syncthreads();
  if (warp == 3) {
    ptx::tcgen05_fence_after();
    ptx::tmem_dealloc(tmem_base, 512);
  }
}

// Sums of the activations over each scale block, for the zero points: xs[b * pitch + m], one warp per (token, block);
// tokens from M up to the pitch get zeros.
template <typename XT>
__global__ void __launch_bounds__(256) block_sums_kernel(const XT* x, float* __restrict__ xs, int pitch, int M, int K, int S) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int lane = threadIdx.x & 31;
  const int64_t i = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (i >= (int64_t)pitch * S) return;
  const int m = (int)(i / S), b = (int)(i - (int64_t)m * S), len = K / S;
  float s = 0.f;
  if (m < M) {
    const uint4* row = reinterpret_cast<const uint4*>(x + (int64_t)m * K + (int64_t)b * len);
    for (int k = lane; k < len / 8; k += 32) {
      const uint4 v = row[k];
      const XT* e = reinterpret_cast<const XT*>(&v);
#pragma unroll
      for (int j = 0; j < 8; ++j) s += to_f32(e[j]);
    }
    s = warp_sum(s);
  }
  if (lane == 0) xs[(int64_t)b * pitch + m] = s;
}

template <typename Kernel, typename... Args>
cudaError_t launch_pdl(Kernel kern, unsigned grid, unsigned block, size_t smem, cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, args...);
}

template <int WBITS, typename XT, int NC, int KS, bool W16>
int launch_with(const CUtensorMap& map_w, const CUtensorMap& map_x, const Params& p, int grid, cudaStream_t st) {
  using C = Cfg<WBITS, NC, KS>;
  auto kern = tmem_gemm_kernel<WBITS, XT, NC, KS, W16>;
  static bool attr_set[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::kSmem);
    if (e != cudaSuccess) return fail(QMM_ERR_LAUNCH, "cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    if (dev >= 0 && dev < 64) attr_set[dev] = true;
  }
  cudaError_t e = launch_pdl(kern, (unsigned)grid, kThreads, C::kSmem, st, map_w, map_x, p);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(QMM_ERR_LAUNCH, "tmem_gemm_kernel launch: %s", cudaGetErrorString(e));
  }
  return QMM_OK;
}

template <int WBITS, typename XT, int NC, int KS>
int launch_cfg(const CUtensorMap& map_w, const CUtensorMap& map_x, const Params& p, int grid, cudaStream_t st) {
  return p.blocked && p.s_dt != QMM_F32 ? launch_with<WBITS, XT, NC, KS, true>(map_w, map_x, p, grid, st)
                                        : launch_with<WBITS, XT, NC, KS, false>(map_w, map_x, p, grid, st);
}

template <int WBITS, typename XT>
int launch_shape(int nc, int ks, const CUtensorMap& map_w, const CUtensorMap& map_x, const Params& p, int grid, cudaStream_t st) {
#define QMM_CASE(NC)                                                           \
  case NC:                                                                     \
    return ks == 64 ? launch_cfg<WBITS, XT, NC, 64>(map_w, map_x, p, grid, st) \
                    : launch_cfg<WBITS, XT, NC, 128>(map_w, map_x, p, grid, st)
  switch (nc) {
    QMM_CASE(32);
    QMM_CASE(64);
    QMM_CASE(128);
    default: QMM_CASE(192);
  }
#undef QMM_CASE
}

size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

constexpr int kMaxCtas = 256;

struct Plan {
  int nc, th, ytiles;
};

Plan plan_for(int64_t M) {
  Plan pl;
  pl.ytiles = (int)ceil_div(M, 192);
  pl.th = (int)align_up((size_t)ceil_div(M, pl.ytiles), 16);  // equal token tiles: 200 tokens are two of 112
  pl.nc = pl.th <= 32 ? 32 : pl.th <= 64 ? 64 : pl.th <= 128 ? 128 : 192;
  return pl;
}

struct Scratch {
  uint32_t* flags;
  float* xs;
  int xs_pitch;
  float* partial;
  size_t bytes;
};

// [flags: 2 KB][block sums][partial tiles]; the flag words are the same as limb_gemm.cu's and are zero between launches.
Scratch carve(void* base, int64_t M, int64_t K) {
  Scratch s;
  uint8_t* b = reinterpret_cast<uint8_t*>(base);
  size_t off = 2048;
  s.flags = reinterpret_cast<uint32_t*>(b);
  s.xs = reinterpret_cast<float*>(b + off);
  s.xs_pitch = (int)align_up((size_t)M, 4) + 192;  // a drain thread reads whole groups of columns
  off += align_up((size_t)ceil_div(K, 64) * s.xs_pitch * 4, 256);
  s.partial = reinterpret_cast<float*>(b + off);
  off += (size_t)kMaxCtas * plan_for(M).th * BMW * 4;
  s.bytes = off;
  return s;
}

}  // namespace

size_t tmem_gemm_workspace_bytes(int64_t max_M, int64_t K) {
  if (max_M < 1 || K < 1) return 0;
  // the block sums of the longest batch up to max_M, and the largest partial tiles of any
  const size_t xs = align_up((size_t)ceil_div(K, 64) * (align_up((size_t)max_M, 4) + 192) * 4, 256);
  return 2048 + xs + (size_t)kMaxCtas * std::min<int64_t>(192, align_up((size_t)max_M, 16)) * BMW * 4;
}

bool tmem_gemm_shape_ok(int wbits, int64_t M, int64_t N, int64_t K, int64_t block_size, int x_dt) {
  if (x_dt != QMM_BF16 && x_dt != QMM_F16) return false;
  if (M < 1 || N < 1 || K < 64 || M > (1 << 24)) return false;
  if (K * wbits / 8 % 16 != 0 || K % 8 != 0) return false;  // TMA row pitches
  if (block_size > 0 && (K % block_size != 0 || (block_size != 64 && block_size % 128 != 0))) return false;
  // 32-bit items and units
  return N <= (1LL << 28) && K <= (1LL << 24) && ceil_div(N, BMW) * ceil_div(M, 16) <= (1LL << 30) / std::max<int64_t>(1, K / 64);
}

bool tmem_gemm_supported(int wbits, int64_t M, int64_t N, int64_t K, int64_t block_size, const void* x, int x_dt, const void* w) {
  return tmem_gemm_shape_ok(wbits, M, N, K, block_size, x_dt) && aligned(x, 16) && aligned(w, 16) && device_is_sm100();
}

int launch_tmem_gemm(int wbits, const void* x, int x_dt, const void* w, const Scales& scales, void* out, int out_dt, int64_t M, int64_t N,
                     int64_t K, int64_t block_size, int gate_up, void* workspace, size_t workspace_bytes, cudaStream_t st) {
  const bool zp = scales.zp != nullptr;
  // (16-bit block scales: of the activations' type, and an even number of them: the branch for a last one without a partner
  // cost 5 % in every batch: asymmetric int4 block 128 [37888,3584] at 29 tokens 44.9 us, 47.2 with it)
  if (!tmem_gemm_supported(wbits, M, N, K, block_size, x, x_dt, w) || !scale_words_ok(scales, block_size) ||
      (block_size > 0 && scales.dt != QMM_F32 && (scales.dt != x_dt || scale_tail(scales, K / block_size, N))))
    return fail(QMM_ERR_UNSUPPORTED,
                "tensor-memory kernel: needs an sm_100 device, bf16/f16 activations, 16-byte row pitches, block_size 64 or a "
                "multiple of 128, 16-byte aligned x/w (M=%lld N=%lld K=%lld bs=%lld)",
                (long long)M, (long long)N, (long long)K, (long long)block_size);
  if (gate_up && (N % 16 != 0 || zp))
    return fail(QMM_ERR_BAD_SHAPE, "fused gate/up epilogue: the interleaved weight needs a multiple of 16 rows and no zero points, got %lld",
                (long long)N);
  const Plan pl = plan_for(M);
  const Scratch sc = carve(workspace, M, K);
  if (!workspace || workspace_bytes < sc.bytes)
    return fail(QMM_ERR_WORKSPACE, "tensor-memory kernel needs %zu bytes of workspace, got %zu", sc.bytes, workspace_bytes);
  if (!aligned(workspace, 256)) return fail(QMM_ERR_MISALIGNED, "workspace must be 256-byte aligned");

  Params p = {};
  p.scale = scales.scale;
  p.zp = scales.zp;
  p.s_dt = scales.dt;
  p.sc_pitch = N * (int64_t)dtype_size(scales.dt);
  p.xs = sc.xs;
  p.xs_pitch = sc.xs_pitch;
  p.out = out;
  p.out_dt = out_dt;
  p.M = (int)M;
  p.N = N;
  const int ks = block_size == 64 ? 64 : 128;
  p.stages = (int)ceil_div(K, ks);
  p.blocked = block_size > 0;
  p.S = block_size > 0 ? (int)(K / block_size) : 1;
  // Per channel the sums leave the tensor core every 512 values all the same: the additions across them are then single
  // fp32 additions in registers, and the drain stays well under the MMAs.
  p.fu = block_size > 0 ? std::max<int>(1, (int)(block_size / ks)) : 4;
  p.ut = (int)ceil_div(p.stages, p.fu);
  p.th = pl.th;
  p.ytiles = pl.ytiles;
  p.gate_up = gate_up;
  p.partial = sc.partial;
  p.flags = sc.flags;
  p.err_word = device_error_word();
  p.wait_cycles = peer_wait_cycles();

  // ---- schedule ----
  const int tiles = (int)ceil_div(N, BMW), items = tiles * pl.ytiles, ctas = std::min(sm_count(), kMaxCtas);
  const int left = items % ctas;
  p.items1 = items;
  int grid = std::min(items, ctas);
  if (left != 0) {
    // Splitting the left-over items over s CTAs each: item / s plus an exchange that grows with s (one partial tile per
    // CTA, written, and read by the item's first CTA).
    const double stage_us = std::max(wbits == 4 ? 0.2 : 0.38, 0.06 + 0.0024 * pl.th) * (ks == 64 ? 0.6 : 1.0);
    const double item_us = p.stages * stage_us, partial_us = 0.25 + 1.1 * pl.th / 256;
    double s = std::sqrt(item_us / partial_us);
    s = std::min(s, std::min((double)ctas / (double)left, (double)p.ut));
    if (s >= 1.2 && item_us / s + 2.0 + partial_us * s < 0.85 * item_us) {
      p.items1 = items - left;
      p.units = left * p.ut;
      p.g2 = std::min(ctas, std::max(left, (int)((double)left * s)));
      grid = std::max(std::min(p.items1, ctas), p.g2);
    }
  }

  if (zp) {
    const unsigned g = (unsigned)ceil_div((int64_t)sc.xs_pitch * p.S, 8);
    cudaError_t e = x_dt == QMM_BF16
                        ? launch_pdl(block_sums_kernel<__nv_bfloat16>, g, 256, 0, st, reinterpret_cast<const __nv_bfloat16*>(x), sc.xs, sc.xs_pitch, (int)M, (int)K, p.S)
                        : launch_pdl(block_sums_kernel<__half>, g, 256, 0, st, reinterpret_cast<const __half*>(x), sc.xs, sc.xs_pitch, (int)M, (int)K, p.S);
    if (e != cudaSuccess) {
      cudaGetLastError();
      return fail(QMM_ERR_LAUNCH, "block_sums_kernel launch: %s", cudaGetErrorString(e));
    }
  }
  CUtensorMap map_w, map_x;
  int rc = encode_tmap_2d(&map_w, w, 1, false, (uint64_t)N, (uint64_t)(K * wbits / 8), BMW, 128);
  if (rc != QMM_OK) return rc;
  rc = encode_tmap_2d(&map_x, x, 2, true, (uint64_t)M, (uint64_t)K, (uint32_t)pl.th, 64);
  if (rc != QMM_OK) return rc;
  if (wbits == 4)
    return x_dt == QMM_BF16 ? launch_shape<4, __nv_bfloat16>(pl.nc, ks, map_w, map_x, p, grid, st)
                            : launch_shape<4, __half>(pl.nc, ks, map_w, map_x, p, grid, st);
  return x_dt == QMM_BF16 ? launch_shape<8, __nv_bfloat16>(pl.nc, ks, map_w, map_x, p, grid, st)
                          : launch_shape<8, __half>(pl.nc, ks, map_w, map_x, p, grid, st);
}

}  // namespace qmm
