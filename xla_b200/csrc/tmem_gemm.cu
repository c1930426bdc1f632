// Weight-only linear for batches on the tensor cores, with the converted weights in tensor memory:
//
//   out[m,n] = sum_b (scale[b,n] * sum_{k in b} x[m,k] w[n,k] - zp[b,n] * sum_{k in b} x[m,k])     (per channel: one block)
//
// "Swap-AB": 128 weight rows are the MMA's M side, tokens its N side.  Integers of up to eight bits are exact in bf16 and
// f16, so the products are exact and the sums are the tensor core's fp32; block sums are scaled and added in fp32
// registers.  (The integer form, limb_gemm.cu, needs two limb columns per token for 16-bit outputs: the same tensor-core
// cycles, but twice the accumulator columns to read back and convert at every scale block.)
//
// The shared-memory port carries 128 bytes a cycle for everything TMA writes and the MMA reads, so the weights never go back to
// shared memory: converting warps read the raw bytes and write the bf16/f16 operand to tensor memory, where the MMA takes its
// A side from, and token tiles are as wide as two accumulators allow (192 columns).
//
//   warp 0        TMA: raw weight tiles, 128 rows x 128 bytes
//   warp 2        TMA: activation tiles, one K step x up to 192 tokens
//   warps 1, 3    MMA issuers, alternate folds: per K step 16, 8 or 4 x tcgen05.mma.kind::f16 (M128 x N<=192 x K16, A in
//                 tensor memory), a commit for the step's operands and one for the accumulators
//   converters    four groups of four warps (two for tiles above 128 tokens); lane = weight row.  A step of 256 values (up to
//                 64 tokens) is shared by two groups, one of 128 is a group's own; the groups take the steps in turn
//   drain         eight warps: thread = weight row, half of the tokens in fp32 registers: tcgen05.ld, scale, add; epilogue
//
// What bounds it.  Up to 64 tokens the instructions of the converters and of the hand-overs: 480 to 510 a scheduler and 128
// values all told (ten for eight int4 weights, 160 of them), issued in 61 to 65 % of the cycles, the tensor pipe busy in 14 to 26 %.
// A wait for a complete barrier costs a warp about 57 cycles and a dependent instruction 4 to 6, so a lone warp's loop of three
// waits, sixteen MMAs and a commit takes 1000 cycles: hence two issuers, steps of 256 values with two scale blocks under one
// hand-over, barriers by address, four groups of converters that wait side by side, and scales a batch at a time.  int4 block 128
// [57344,8192]: 29 tokens 121 us with one issuer and steps of 128 values, 68 now; 64 tokens 134 and 88.  Above 128 tokens a step
// of 128 values takes 1300 cycles for 704 of MMAs: instructions again (820 a scheduler: 96 sums a thread; the tensor pipe busy in
// half of the time), at 1.65 GHz under load.  512 tokens 511 us and 460.
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
#include "convert.cuh"
#include "issue_order.h"
#include "kernels.h"
#include "ptx_sm100.cuh"

namespace qmm {

namespace {

constexpr int BMW = 128;                  // weight rows per tile (UMMA M)
constexpr uint32_t kRawBytes = BMW * 128; // one raw tile: 128 rows x 128 bytes
constexpr int kDone = 8;                  // step-complete barriers
constexpr int kDrain = 256;               // drain threads
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
  int fu;         // steps per fold (accumulation in the tensor core), >= 1
  int alternate;  // the folds alternate between the two issuers (else the first one has them all)
  int blocked;    // scale blocks (0: per channel; folds are then plain additions)
  int S;
  int unit;       // steps per scheduling unit: whole folds and whole raw tiles
  int fpu;        // folds per unit
  int ut;         // units per tile (steps beyond K multiply zeros)
  int th;         // tokens per item (a multiple of 16)
  int ytiles;
  int items1;     // items handed out whole: CTA c takes c, c + G, ...
  int units;      // units of the remaining items, dealt in equal contiguous shares to the first g2 CTAs
  int g2;
  int gate_up;
  float* partial;   // [g2][th / 4][128][4]
  uint32_t* flags;  // [g2], zero between launches
  uint32_t* err_word;
  long long wait_cycles;  // for a partial tile
};

// NC: accumulator columns (tokens); KS: k values per step; SUB: scale blocks per step that have an accumulator each (a fold is
// then one step), or 1 (a fold is one or more steps).
template <int WBITS, int NC, int KS, int SUB>
struct Cfg {
  static constexpr int kAccCols = SUB * NC;
  static constexpr int kAcc = 2;
  static constexpr int kACols = KS / 2;  // tensor-memory columns per operand step
  static constexpr int kASlots = std::min(4, (512 - kAcc * kAccCols) / kACols / 2 * 2);
  static constexpr int kACol0 = 512 - kASlots * kACols;
  // Groups of four converting warps.  Teams of one group (steps of up to 128 values) or two (half of 256 each) take the steps
  // in turn.
  static constexpr int kGroups = NC == 192 ? 2 : 4, kTeamGroups = NC <= 64 ? 2 : 1, kTeams = kGroups / kTeamGroups;
  static constexpr int kThreads = 128 + 128 * kGroups + kDrain;
  // setmaxnreg: within threads x registers at launch
  static constexpr int kMiscRegs = NC == 192 ? 32 : 40;
  static constexpr int kConvRegs = 56;
  static constexpr int kDrainRegs = NC == 192 ? 168 : 120;
  static constexpr int kLaunchRegs = kThreads == 640 ? 96 : 72;
  static_assert(128 * kMiscRegs + 128 * kGroups * kConvRegs + kDrain * kDrainRegs <= kThreads * kLaunchRegs, "register split");
  static constexpr uint32_t kBStage = NC * KS * 2;
  static constexpr int kRaw = NC >= 64 ? 4 : 8;
  static constexpr int kB = std::min(kDone, (NC == 192 ? 144 : NC >= 64 ? 128 : 64) * 1024 / (int)kBStage);
  // The accumulator is what an issuer waits for longest, so its barrier comes last where the turns of the other rings are the
  // issuer's own steps, and first where they are not.
  static constexpr bool kAccLast = kB % 2 == 0 && kASlots % 2 == 0;
  static constexpr int kTV = 1024 / WBITS;          // values of a row per raw tile
  static constexpr int kVV = KS / kTeamGroups;      // values per step and converting group
  static constexpr int kDT = NC / 2;                // tokens per drain thread
  // columns per tensor-memory load of the drain, and sets of registers for them
  static constexpr int kCh = kDT == 96 || kDT == 16 ? 16 : 32, kChBufs = kDT == 96 || SUB > 1 ? 2 : 1;
  // block scales, zero points and block sums of the activations (per group of drain warps) on their way, in two batches
  static constexpr int kScaleRing = NC == 32 ? 12 : NC == 192 ? 6 : 8, kBatch = kScaleRing / 2;
  static constexpr size_t kScaleBytes = 2 * kScaleRing * kDrain * 4, kSumBytes = 2 * kScaleRing * kDT * 4;
  static constexpr size_t kSmem = 1024 + (size_t)kRaw * kRawBytes + (size_t)kB * kBStage + kScaleBytes + kSumBytes + 512;
  static_assert(kAcc * kAccCols <= kACol0 && kASlots >= 2, "tensor memory");
  static_assert(kSmem <= 227 * 1024, "shared memory budget");
  // A parity wait is right only while the barrier is at most one phase away: whoever waits for step i - d does so for every
  // step in turn (the converters: for every step of their team), and step i - d + kDone cannot complete before it has gone on.
  static_assert(kB <= kDone && kASlots <= kB && kAcc <= kDone, "turns of the rings");
  static_assert(issuers_may_alternate(1, kASlots, kB, kAccLast), "folds of one step alternate");
  static_assert(kASlots % kTeams == 0 && kDone % kTeams == 0 && kVV <= kTV, "slots of a team");
  static_assert(kRaw % std::max(1, kTeams * KS / kTV) == 0, "a group comes back to the raw slots it has waited for");
  static_assert(kBatch % SUB == 0 && kBatch * kDT / 4 <= kDrain / 2, "batches of scales and block sums");
  static_assert(SUB == 1 || (kDT <= 32 && SUB == 2), "a load per accumulator");
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
  __device__ int s0() const { return u0 * p.unit; }
  __device__ int s1() const { return u1 * p.unit; }
  // steps of all fragments, before the first next()
  __device__ int steps() const { return ((nxt < p.items1 ? (p.items1 - 1 - nxt) / (int)gridDim.x + 1 : 0) * p.ut + (hi - u)) * p.unit; }
};

__device__ __forceinline__ uint4 lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}

// C tokens of one output column, `pitch` elements apart
template <int C, typename OT>
__device__ __forceinline__ void store_tokens_as(OT* o, int64_t pitch, const float* v, int count) {
#pragma unroll
  for (int t = 0; t < C; ++t, o += pitch)
    if (t < count) *o = from_f32<OT>(v[t]);
}
template <int C>
__device__ __forceinline__ void store_tokens(void* out, int dt, int64_t at, int64_t pitch, const float* v, int count) {
  if (dt == QMM_BF16) store_tokens_as<C>(reinterpret_cast<__nv_bfloat16*>(out) + at, pitch, v, count);
  else if (dt == QMM_F16) store_tokens_as<C>(reinterpret_cast<__half*>(out) + at, pitch, v, count);
  else store_tokens_as<C>(reinterpret_cast<float*>(out) + at, pitch, v, count);
}

template <int REGS>
__device__ __forceinline__ void reg_inc() {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGS));
}
template <int REGS>
__device__ __forceinline__ void reg_dec() {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS));
}

template <int WBITS, typename XT, int NC, int KS, int SUB, bool W16>
__global__ void __launch_bounds__(Cfg<WBITS, NC, KS, SUB>::kThreads, 1)
    tmem_gemm_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const Params p) {
  using C = Cfg<WBITS, NC, KS, SUB>;
  constexpr int kRaw = C::kRaw, kB = C::kB, kAcc = C::kAcc, DT = C::kDT, kASlots = C::kASlots, kACols = C::kACols, kGroups = C::kGroups,
                kScaleRing = C::kScaleRing;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* raw_base = smem;
  uint8_t* b_base = raw_base + (size_t)kRaw * kRawBytes;
  uint32_t* s_scale = reinterpret_cast<uint32_t*>(b_base + (size_t)kB * C::kBStage);  // [scale, zero point][kScaleRing][kDrain]
  uint64_t* bars = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(s_scale) + C::kScaleBytes + C::kSumBytes);
  uint64_t* raw_full = bars;                 // [kRaw]    TMA bytes
  uint64_t* raw_empty = raw_full + kRaw;     // [kRaw]    the converting warps that read the tile
  uint64_t* b_full = raw_empty + kRaw;       // [kB]      TMA bytes
  uint64_t* a_full = b_full + kB;            // [kASlots] the converting warps of the step
  uint64_t* acc_empty = a_full + kASlots;    // [kAcc]    eight drain warps
  uint64_t* acc_full = acc_empty + kAcc;     // [kAcc]    tcgen05.commit: the fold is complete
  uint64_t* done = acc_full + kAcc;          // [kDone]   tcgen05.commit: the MMAs of step i are complete
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + kDone);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = ptx::warp_index(), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kRaw; ++s) {
      ptx::mbar_init(&raw_full[s], 1);
      ptx::mbar_init(&raw_empty[s], 4 * C::kTV / C::kVV);
    }
    for (int s = 0; s < kB; ++s) ptx::mbar_init(&b_full[s], 1);
    for (int s = 0; s < kASlots; ++s) ptx::mbar_init(&a_full[s], 4 * C::kTeamGroups);
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
    reg_dec<C::kMiscRegs>();
    FragIter it(p);
    if (warp == 0) {
      // ---------------- raw weight producer: static data, no wait for earlier kernels ----------------
      if (lane == 0) {
        int slot = 0;
        uint32_t ph = 0;
        while (it.next()) {
          const int s0 = it.s0(), s1 = it.s1();
          for (int b = s0 * (KS * WBITS / 8); b < s1 * (KS * WBITS / 8); b += 128) {
            ptx::mbar_wait(&raw_empty[slot], ph ^ 1, abort_flag, p.err_word, ptx::kErrWaitEmpty);
            ptx::mbar_expect_tx(&raw_full[slot], kRawBytes);
            ptx::tma_load_2d(raw_base + (size_t)slot * kRawBytes, &map_w, &raw_full[slot], b, it.tile * BMW);
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
    } else {
      // ---------------- MMA issuers, warps 1 and 3: the folds alternate between them ----------------
      // A whole warp walks the loop, one elected thread issues.
      constexpr uint32_t fmt = std::is_same<XT, __half>::value ? 0u : 1u;
      const uint32_t idesc = ptx::make_idesc(/*f32*/ 1, fmt, fmt, BMW, (uint32_t)p.th);
      // Operands of the MMA live in uniform registers.  What the compiler cannot see to be the same in all lanes (a value
      // from shared memory, a branch on a predicate computed earlier) is moved there again for every MMA: int4 block 128
      // [28672,8192] at 512 tokens 285 us moved every time, 266 so.
      const uint32_t tb = __reduce_or_sync(0xffffffffu, tmem_base);
      const uint32_t desc_hi = (uint32_t)(ptx::make_sw128_kmajor_desc(0) >> 32);
      const uint32_t b_lo0 = (uint32_t)ptx::make_sw128_kmajor_desc(ptx::smem_u32(b_base));
      const uint32_t b_full_a = ptx::smem_u32(b_full), a_full_a = ptx::smem_u32(a_full), acc_empty_a = ptx::smem_u32(acc_empty),
                     acc_full_a = ptx::smem_u32(acc_full), done_a = ptx::smem_u32(done);
      const bool alternate = p.alternate != 0;
      const uint32_t me = (uint32_t)warp >> 1;
      const uint32_t total = (uint32_t)it.steps(), fu = (uint32_t)p.fu;
      const uint32_t jump = alternate ? fu : 0u;  // steps of the other issuer between two folds
      uint32_t j = me * fu, buf = me, pacc = 1, sb = j % kB, pb = 0;
      const uint32_t buf_inc = alternate ? 2 : 1;
      if (!alternate && me) j = total;
      constexpr bool kAccLast = C::kAccLast;
      while (j < total) {
        if (!kAccLast) ptx::bar_wait(acc_empty_a + buf * 8, pacc, abort_flag, p.err_word, ptx::kErrWaitTmemEmpty);
        const uint32_t d = tb + buf * C::kAccCols;
        for (uint32_t q = 0; q < fu; ++q, ++j) {
          const uint32_t sa = j % kASlots;
          ptx::bar_wait(b_full_a + sb * 8, pb, abort_flag, p.err_word, ptx::kErrWaitFull);
          ptx::bar_wait(a_full_a + sa * 8, (j / kASlots) & 1, abort_flag, p.err_word, ptx::kErrWaitConv);
          if (kAccLast && q == 0) ptx::bar_wait(acc_empty_a + buf * 8, pacc, abort_flag, p.err_word, ptx::kErrWaitTmemEmpty);
          ptx::tcgen05_fence_after();
          const uint32_t a = tb + C::kACol0 + sa * kACols;
          const uint32_t lo = b_lo0 + sb * (C::kBStage >> 4);
          if (ptx::elect_one()) {
#pragma unroll
            for (int k = 0; k < KS / 16; ++k) {
              constexpr int kPerAcc = KS / 16 / SUB;
              ptx::mma_f16_ts(d + k / kPerAcc * NC, a + k * 8, ((uint64_t)desc_hi << 32) | (uint64_t)(lo + (k >> 2) * (NC * 128 >> 4) + (k & 3) * 2),
                              idesc, q | (uint32_t)(k % kPerAcc));
            }
            ptx::mma_commit_a(done_a + (j % kDone) * 8);
            if (q + 1 == fu) ptx::mma_commit_a(acc_full_a + buf * 8);
          }
          if (++sb == kB) { sb = 0; pb ^= 1; }
        }
        j += jump;
        sb += jump;
        if (sb >= kB) { sb -= kB; pb ^= 1; }
        buf += buf_inc;
        if (buf >= kAcc) { buf -= kAcc; pacc ^= 1; }
      }
    }
    __syncwarp();
  } else if (warp < 4 + 4 * kGroups) {
    // ---------------- converters: lane = weight row; two groups take half of a step's values each ----------------
    reg_dec<C::kConvRegs>();
    const int quad = warp & 3, grp = (warp - 4) >> 2;
    const uint32_t r = quad * 32 + lane;
    constexpr int kTeams = C::kTeams, kTV = C::kTV, kVV = C::kVV;
    constexpr int kWords = 32;                          // words of converted pairs per tensor-memory store
    static_assert(kVV / 2 % kWords == 0, "whole stores");
    constexpr int kPieces = kWords * 2 * WBITS / 128;   // the 16-byte pieces of a row that make them
    const uint32_t done_a = ptx::smem_u32(done), a_full_a = ptx::smem_u32(a_full);
    const int team = grp / C::kTeamGroups, part = grp % C::kTeamGroups;
    const uint32_t t_row = tmem_base + ((uint32_t)(quad * 32) << 16) + C::kACol0 + part * (kVV / 2);
    const uint32_t steps = (uint32_t)FragIter(p).steps();
    uint32_t s = team;
    uint32_t off = s * KS + part * kVV;  // of this group's values in the raw tile
    uint32_t rs = off / kTV * 8;         // eight times the raw slot
    off = off % kTV * WBITS / 8;
    uint32_t rph = 0;
    const uint32_t raw_full_a = ptx::smem_u32(raw_full), raw_empty_a = ptx::smem_u32(raw_empty);
    // the row in the first raw tile, with the swizzle: piece c is at row0 ^ (c << 4)
    const uint32_t row0 = ptx::smem_u32(raw_base) + r * 128 + ((r & 7) << 4);
    for (; s < steps; s += kTeams) {
      ptx::bar_wait(raw_full_a + rs, rph, abort_flag, p.err_word, ptx::kErrWaitRaw);
      const uint32_t row = (row0 + rs * (kRawBytes / 8)) ^ off;
      const uint32_t sa = kASlots == kTeams ? (uint32_t)team : s % kASlots, ts = t_row + sa * kACols;
#pragma unroll
      for (int h = 0; h < kVV / 2 / kWords; ++h) {
        uint32_t o[kWords];
#pragma unroll
        for (int c = 0; c < kPieces; ++c) {
          const uint4 w = lds128(row ^ ((h * kPieces + c) << 4));
          if constexpr (WBITS == 4) {
            cvt_s4x8<XT>(w.x, o + 16 * c);
            cvt_s4x8<XT>(w.y, o + 16 * c + 4);
            cvt_s4x8<XT>(w.z, o + 16 * c + 8);
            cvt_s4x8<XT>(w.w, o + 16 * c + 12);
          } else {
            cvt_s8x4<XT>(w.x, o + 8 * c);
            cvt_s8x4<XT>(w.y, o + 8 * c + 2);
            cvt_s8x4<XT>(w.z, o + 8 * c + 4);
            cvt_s8x4<XT>(w.w, o + 8 * c + 6);
          }
        }
        if (h == 0) {
          // the MMAs that read this operand slot last are complete
          if (s >= (uint32_t)kASlots)
            ptx::bar_wait(done_a + (s - kASlots) % kDone * 8, (s - kASlots) / kDone & 1, abort_flag, p.err_word, ptx::kErrWaitEmpty);
          ptx::tcgen05_fence_after();
        }
        ptx::tmem_st_32x32b_x32(ts + 32 * h, o);
      }
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive_a(raw_empty_a + rs);
      ptx::tmem_st_wait();
      ptx::tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive_a(a_full_a + sa * 8);
      if constexpr (kTeams * KS >= kTV) {
        rs += kTeams * KS / kTV * 8;
      } else {
        off += kTeams * KS * WBITS / 8;
        if (off >= 128) {
          off -= 128;
          rs += 8;
        }
      }
      if (rs >= kRaw * 8) { rs -= kRaw * 8; rph ^= 1; }
    }
  } else {
    // ---------------- drain: thread = weight row (its TMEM lane), half of the item's tokens ----------------
    reg_inc<C::kDrainRegs>();
    const int quad = warp & 3, grp = (warp - 4 - 4 * kGroups) >> 2;
    const int rl = quad * 32 + lane;
    const int dt = (int)threadIdx.x - (4 + 4 * kGroups) * 32;  // 0..255
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quad * 32) << 16) + grp * DT;
    auto drain_bar = [&]() { asm volatile("bar.sync 1, 256;" ::: "memory"); };
    __shared__ int s_npart;
    const uint32_t my_scale_a = ptx::smem_u32(s_scale + dt), acc_empty_a = ptx::smem_u32(acc_empty);
    // the scale of block f at place i of the ring
    auto value = [&](uint32_t i, int f) {
      uint32_t w;
      asm volatile("ld.shared.u32 %0, [%1];" : "=r"(w) : "r"(my_scale_a + i * (kDrain * 4)) : "memory");
      return scale_of_word<W16, XT>(w, rl, f, (int)p.N);  // (a tile starts at an even row)
    };
    const uint32_t acc_full_a = ptx::smem_u32(acc_full);
    if (!p.blocked) {
#pragma unroll 1
      for (int e = 0; e < kScaleRing; ++e) asm volatile("st.shared.f32 [%0], 0f3f800000;" ::"r"(my_scale_a + e * (kDrain * 4)) : "memory");
    }
    const bool block_zp = p.blocked && p.zp;
    const int gt = dt % (kDrain / 2);
    const uint32_t sums_a = ptx::smem_u32(reinterpret_cast<uint8_t*>(s_scale) + C::kScaleBytes) + grp * (kScaleRing * DT * 4);
    // the drain group's threads have all come here
    auto group_bar = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(2 + grp), "n"(kDrain / 2) : "memory"); };
    const int place = deal_place(p);
    FragIter it(p);
    uint32_t i = 0;  // folds of this CTA
    // Block scales and zero points are a stream of their own (a round trip to HBM each): every thread copies its own row's, one
    // to two batches of folds ahead, into a ring of its own; the first two of a fragment ahead of the epilogue of the fragment
    // before it.  (Held in registers that shift from fold to fold, the shift waits for the load of the fold before, whatever
    // the nominal distance.)
    const uint8_t *scp = nullptr, *zpp = nullptr;
    int to_fetch = 0, xs_at = 0, xs_end = 0;  // blocks of the fragment that are left; the next whose sums are fetched, and their end
    const float* xs_m = nullptr;              // block sums of the thread's piece of the group's tokens
    const int xs_e = gt / (DT / 4), xs_piece = gt % (DT / 4);
    auto fetch_batch = [&](uint32_t at) {
      const uint32_t dst = my_scale_a + at * (kDrain * 4);
      if (to_fetch >= C::kBatch) {
#pragma unroll
        for (int e = 0; e < C::kBatch; ++e) {
          copy_scale_word<W16>(dst + e * (kDrain * 4), scp);
          scp += p.sc_pitch;
        }
        if (p.zp) {
#pragma unroll
          for (int e = 0; e < C::kBatch; ++e) {
            copy_scale_word<W16>(dst + (kScaleRing + e) * (kDrain * 4), zpp);
            zpp += p.sc_pitch;
          }
        }
      } else if (p.blocked) {
        // (none past the fragment's end: with short K filling the whole ring for every item was a tenth of the time, int4 block 128
        // [28672,1024] at 60 tokens 12.0 us, 11.1 so)
        const int fill = min(C::kBatch, to_fetch + (it.u1 == p.ut ? p.ut * p.fpu * SUB - p.S : 0));
#pragma unroll 1
        for (int e = 0; e < fill; ++e) {
          const uint32_t d = dst + e * (kDrain * 4);
          if (e < to_fetch) {
            copy_scale_word<W16>(d, scp);
            scp += p.sc_pitch;
            if (p.zp) {
              copy_scale_word<W16>(d + kScaleRing * (kDrain * 4), zpp);
              zpp += p.sc_pitch;
            }
          } else {
            // beyond the last block: its sums are zero, and the factor has to be a number
            asm volatile("st.shared.u32 [%0], 0;" ::"r"(d) : "memory");
            asm volatile("st.shared.u32 [%0], 0;" ::"r"(d + kScaleRing * (kDrain * 4)) : "memory");
          }
        }
      }
      if (block_zp) {
        // the sums of the batch's blocks for the group's tokens, 16 bytes by a thread
        if (xs_e < C::kBatch && xs_at + xs_e < xs_end)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sums_a + (at + xs_e) * (DT * 4) + xs_piece * 16),
                       "l"(xs_m + (int64_t)min(xs_at + xs_e, p.S - 1) * p.xs_pitch)
                       : "memory");
        xs_at += C::kBatch;
      }
      to_fetch -= C::kBatch;
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // the scales of the fragment that `it` has come to
    auto fetch_first = [&]() {
      const int b0 = it.u0 * p.fpu * SUB, b1 = it.u1 * p.fpu * SUB;
      const int64_t off = min((int64_t)it.tile * BMW + rl, p.N - 1) * (W16 ? 2 : 4) + b0 * p.sc_pitch;
      scp = static_cast<const uint8_t*>(p.scale) + off;
      zpp = static_cast<const uint8_t*>(p.zp) + off;
      to_fetch = p.blocked ? min(b1, p.S) - b0 : 0;
      xs_at = b0;
      xs_end = b1;
      xs_m = p.xs + it.y * p.th + grp * DT + xs_piece * 4;
      fetch_batch(0);
      fetch_batch(C::kBatch);
    };
    bool more = it.next();
    if (more) {
      // scales (a conversion may be the kernel in front), block sums, scratch and `out` belong to earlier kernels until here
      asm volatile("griddepcontrol.wait;" ::: "memory");
      fetch_first();
    }
    while (more) {
      const int64_t n = (int64_t)it.tile * BMW + rl;
      const bool n_ok = n < p.N;
      const int item = it.item, f0 = it.u0 * p.fpu, f1 = it.u1 * p.fpu;  // folds
      const bool first = it.u0 == 0, last = it.u1 == p.ut;
      const int m0 = it.y * p.th + grp * DT;                      // first token of this thread
      const int mcount = min(p.M - m0, min(DT, p.th - grp * DT)); // its tokens
      float total[DT];
#pragma unroll
      for (int t = 0; t < DT; ++t) total[t] = 0.f;
      uint32_t half = 0;  // batch of the ring
#pragma unroll 1
      for (int f = f0; f < f1;) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        if (block_zp) group_bar();  // the block sums of the batch have landed
        const int fe = min(f1, f + C::kBatch / SUB);
        uint32_t at = half;
#pragma unroll 1
        for (; f < fe; ++f, ++i, at += SUB) {
          float sc[SUB];
#pragma unroll
          for (int h = 0; h < SUB; ++h) sc[h] = value(at + h, f * SUB + h);
          if (block_zp) {
            // the zero points' share first, while the fold's MMAs run: it needs the block sums only
#pragma unroll
            for (int h = 0; h < SUB; ++h) {
              const float z = value(kScaleRing + at + h, f * SUB + h) * (-1.f / Unit<XT>::kBack);  // (zero beyond the last block)
#pragma unroll
              for (int t = 0; t < DT; t += 4) {
                const uint4 v = lds128(sums_a + (at + h) * (DT * 4) + t * 4);
                total[t] = fmaf(z, __uint_as_float(v.x), total[t]);
                total[t + 1] = fmaf(z, __uint_as_float(v.y), total[t + 1]);
                total[t + 2] = fmaf(z, __uint_as_float(v.z), total[t + 2]);
                total[t + 3] = fmaf(z, __uint_as_float(v.w), total[t + 3]);
              }
            }
          }
          static_assert(kAcc == 2, "turns of the accumulators");
          const uint32_t buf = i % kAcc;
          ptx::bar_wait(acc_full_a + buf * 8, (i >> 1) & 1, abort_flag, p.err_word, ptx::kErrWaitTmemFull);
          ptx::tcgen05_fence_after();
          const uint32_t a = lane_addr + buf * C::kAccCols;
          auto release = [&]() {
            ptx::tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive_a(acc_empty_a + buf * 8);
          };
          constexpr int CH = C::kCh, NB = C::kChBufs, kChunks = DT / CH;
          uint32_t r[NB][CH];
          auto load = [&](uint32_t at, uint32_t* to) {
            static_assert(CH == 16 || CH == 32, "columns of a load");
            if constexpr (CH == 16) ptx::tmem_ld_32x32b_x16(at, to);
            else ptx::tmem_ld_32x32b_x32(at, to);
          };
          auto add = [&](const uint32_t* from, float s, float* to) {
#pragma unroll
            for (int t = 0; t < CH; ++t) to[t] = fmaf(s, __uint_as_float(from[t]), to[t]);
          };
          if constexpr (SUB > 1) {
#pragma unroll
            for (int h = 0; h < SUB; ++h) load(a + h * NC, r[h]);
            ptx::tmem_ld_wait();
#pragma unroll
            for (int h = 0; h < SUB; ++h)
#pragma unroll
              for (int t = 0; t < CH; t += 8) ptx::tmem_ld_landed8(r[h] + t);
            release();
#pragma unroll
            for (int h = 0; h < SUB; ++h) add(r[h], sc[h], total);
          } else {
            load(a, r[0]);
#pragma unroll
            for (int c = 0; c < kChunks; ++c) {
              uint32_t* cur = r[c % NB];
              ptx::tmem_ld_wait();
#pragma unroll
              for (int t = 0; t < CH; t += 8) ptx::tmem_ld_landed8(cur + t);
              if (NB > 1 && c + 1 < kChunks) load(a + (c + 1) * CH, r[(c + 1) % NB]);
              if (c + 1 == kChunks) release();
              add(cur, sc[0], total + CH * c);
              if (NB == 1 && c + 1 < kChunks) load(a + (c + 1) * CH, r[0]);
            }
          }
        }
        if (block_zp) group_bar();
        fetch_batch(half);  // the batch that was used up
        half = C::kBatch - half;
      }
      // ---- end of the fragment ----
      more = it.next();
      if (more) fetch_first();
      // Up to 32 tokens at a time in a rolled loop that rotates the sums through the first registers: unrolled over all tokens
      // this part is tens of kilobytes of code that runs once per item, and fetching it took 10 to 30 us.
      constexpr int EC = DT <= 32 ? DT : 16;
      int np = 0;
      if (first && !last) {
        // the sums of the CTAs that continue the item are added in CTA order, once they are all there
        if (dt == 0) {
          int cnt = 0;
          for (int c2 = place + 1; c2 < p.g2; ++c2) {
            if (it.share(c2) >= (item - p.items1 + 1) * p.ut) break;
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
      for (int c = 0; c < DT / EC; ++c) {
        const int l0 = grp * DT + EC * c;  // token inside the item
        const int count = min(EC, mcount - EC * c);
        if (lost) {
#pragma unroll
          for (int t = 0; t < EC; ++t) total[t] = __uint_as_float(0x7fc00000u);
        }
        if (!first) {
          // a later K range of an item that another CTA started: leave the sums for that CTA
          float4* dst = reinterpret_cast<float4*>(p.partial + ((size_t)place * p.th + l0) * BMW) + rl;
#pragma unroll
          for (int t = 0; t < EC; t += 4)
            if (t < count) __stcg(dst + t / 4 * BMW, make_float4(total[t], total[t + 1], total[t + 2], total[t + 3]));
        } else {
          // added in CTA order; two partial tiles on their way at a time where the registers allow (a round trip to L2 each)
          constexpr int kAhead = DT <= 32 ? 2 : 1;
          const float4* src = reinterpret_cast<const float4*>(p.partial + ((size_t)(place + 1) * p.th + l0) * BMW) + rl;
          const size_t pitch = (size_t)p.th * (BMW / 4);
#pragma unroll 1
          for (int j = 0; j < np; j += kAhead, src += kAhead * pitch) {
#pragma unroll
            for (int t0 = 0; t0 < EC; t0 += 16) {
              float4 v[kAhead][4];
#pragma unroll
              for (int a = 0; a < kAhead; ++a)
#pragma unroll
                for (int t = 0; t < 4; ++t)
                  v[a][t] = t0 + 4 * t < count && j + a < np ? __ldcg(src + a * pitch + (t0 / 4 + t) * BMW) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
              for (int a = 0; a < kAhead; ++a)
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                  total[t0 + 4 * t] += v[a][t].x;
                  total[t0 + 4 * t + 1] += v[a][t].y;
                  total[t0 + 4 * t + 2] += v[a][t].z;
                  total[t0 + 4 * t + 3] += v[a][t].w;
                }
            }
          }
#pragma unroll
          for (int t = 0; t < EC; ++t) total[t] *= Unit<XT>::kBack;
          if (!p.blocked) {
#pragma unroll
            for (int t = 0; t < EC; ++t) {
              total[t] *= ps;
              if (p.zp && t < count) total[t] = fmaf(z1, ld_ordered(p.xs + m0 + EC * c + t), total[t]);
            }
          }
          const int64_t row_out = m0 + EC * c;
          if (!p.gate_up) {
            store_tokens<EC>(p.out, p.out_dt, row_out * p.N + n, p.N, total, n_ok ? count : 0);
          } else {
            // Rows come in groups of 16: eight gate rows, then the eight up rows of the same outputs.  The thread of the gate
            // row does the first half of the tokens, that of the up row the second.
            const bool up_row = (rl & 8) != 0;
            float v[EC / 2];
#pragma unroll
            for (int t = 0; t < EC / 2; ++t) {
              const float got = __shfl_xor_sync(0xffffffffu, up_row ? total[t] : total[t + EC / 2], 8);
              const float g = up_row ? got : total[t], u = up_row ? total[t + EC / 2] : got;
              v[t] = g / (1.f + expf(-g)) * u;
            }
            const int t0 = up_row ? EC / 2 : 0;
            store_tokens<EC / 2>(p.out, p.out_dt, (row_out + t0) * (p.N >> 1) + ((n >> 4) << 3) + (n & 7), p.N >> 1, v, n_ok ? count - t0 : 0);
          }
        }
#pragma unroll
        for (int t = 0; t + EC < DT; ++t) total[t] = total[t + EC];
      }
      if (!first) {
        drain_bar();  // orders every drain thread's stores before thread 0's fence, which is cumulative
        if (dt == 0) ptx::partial_publish(p.flags + place);
      }
    }
  }

  ptx::tcgen05_fence_before();
  __syncthreads();
  if (warp == 3) {
    ptx::tcgen05_fence_after();
    ptx::tmem_dealloc(tmem_base, 512);
  }
}

// Sums of the activations over each scale block, for the zero points: xs[b * pitch + m]; tokens from M up to the pitch get
// zeros.  A warp takes 256 values of a row, or a whole larger block, at a time.  Several shorter blocks of a row (of 64 or 128
// values) are summed by the lanes that hold them, 8 or 16; one that is alone in its row (per channel, any multiple of eight values)
// by all lanes, of which those beyond it hold zeros.  ROW: a CTA takes a row, for long rows per channel.
// Bound by the latency of its loads, so a warp has one piece, as many loads at a time as that needs: with one CTA per SM walking the pieces,
// 2044 tokens of [735,14592] block 384 took 154 us with the GEMM, 81 so.  A long row has a CTA for the same reason ([588,27456] int4 per
// channel at 120 tokens 58 us with a warp, 41 so).
constexpr int kSumsThreads = 256;
constexpr int kLongRow = 2048;  // values
template <typename XT, bool ROW>
__global__ void __launch_bounds__(kSumsThreads) block_sums_kernel(const XT* x, float* __restrict__ xs, int pitch, int M, int K, int S) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int lane = threadIdx.x & 31;
  // 256 values by the lanes of the warp, eight each
  auto add = [](float s, const XT* at) {
    const uint4 v = *reinterpret_cast<const uint4*>(at);
    const XT* e = reinterpret_cast<const XT*>(&v);
#pragma unroll
    for (int j = 0; j < 8; ++j) s += to_f32(e[j]);
    return s;
  };
  if constexpr (ROW) {
    __shared__ float s_warp[kSumsThreads / 32];
    const int m = blockIdx.x;
    float s = 0.f;
    if (m < M) {
      const XT* row = x + (int64_t)m * K;
#pragma unroll 4
      for (int k = threadIdx.x * 8; k < K; k += kSumsThreads * 8) s = add(s, row + k);
    }
    s = warp_sum(s);
    if (lane == 0) s_warp[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
      for (int i = 1; i < kSumsThreads / 32; ++i) s += s_warp[i];
      xs[m] = s;
    }
  } else {
    const int len = K / S, per = max(len, 256), pieces = (K + per - 1) / per;
    const int group = S > 1 && len < 256 ? len / 8 : 32;  // lanes that sum a block, a power of two
    const int64_t warps = (int64_t)gridDim.x * (kSumsThreads / 32);
    for (int64_t i = (int64_t)blockIdx.x * (kSumsThreads / 32) + (threadIdx.x >> 5); i < (int64_t)pitch * pieces; i += warps) {
      const int m = (int)(i / pieces), k0 = (int)(i - (int64_t)m * pieces) * per, k1 = min(K, k0 + per);
      float s = 0.f;
      if (m < M) {
        const XT* row = x + (int64_t)m * K;
#pragma unroll 4
        for (int k = k0 + lane * 8; k < k1; k += 256) s = add(s, row + k);
        for (int o = group >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      }
      const int b = (k0 + lane * 8) / len;
      if (lane % group == 0 && b < S) xs[(int64_t)b * pitch + m] = s;
    }
  }
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

template <int WBITS, typename XT, int NC, int KS, int SUB, bool W16>
int launch_with(const CUtensorMap& map_w, const CUtensorMap& map_x, Params p, int grid, cudaStream_t st) {
  using C = Cfg<WBITS, NC, KS, SUB>;
  p.alternate = issuers_may_alternate(p.fu, C::kASlots, C::kB, C::kAccLast);
  auto kern = tmem_gemm_kernel<WBITS, XT, NC, KS, SUB, W16>;
  static bool attr_set[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::kSmem);
    if (e != cudaSuccess) return fail(QMM_ERR_LAUNCH, "cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    // the warps' shares of the registers add up to this
    cudaFuncAttributes at;
    e = cudaFuncGetAttributes(&at, kern);
    if (e != cudaSuccess || at.numRegs != C::kLaunchRegs)
      return fail(QMM_ERR_LAUNCH, "tmem_gemm_kernel: built with %d registers per thread, not %d", e == cudaSuccess ? at.numRegs : -1, C::kLaunchRegs);
    if (dev >= 0 && dev < 64) attr_set[dev] = true;
  }
  cudaError_t e = launch_pdl(kern, (unsigned)grid, C::kThreads, C::kSmem, st, map_w, map_x, p);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(QMM_ERR_LAUNCH, "tmem_gemm_kernel launch: %s", cudaGetErrorString(e));
  }
  return QMM_OK;
}

template <int WBITS, typename XT, int NC, int KS, int SUB>
int launch_cfg(const CUtensorMap& map_w, const CUtensorMap& map_x, const Params& p, int grid, cudaStream_t st) {
  return p.blocked && p.s_dt != QMM_F32 ? launch_with<WBITS, XT, NC, KS, SUB, true>(map_w, map_x, p, grid, st)
                                        : launch_with<WBITS, XT, NC, KS, SUB, false>(map_w, map_x, p, grid, st);
}

// Values per step, and scale blocks per step with an accumulator each
struct Step {
  int ks, sub;
};
Step step_for(int nc, int64_t block_size) {
  if (nc <= 64)
    return block_size == 64 ? Step{128, 2} : block_size == 128 ? Step{256, 2} : block_size > 0 && block_size % 256 != 0 ? Step{128, 1} : Step{256, 1};
  return block_size == 64 ? Step{64, 1} : Step{128, 1};
}

template <int WBITS, typename XT>
int launch_shape(int nc, const Step& sp, const CUtensorMap& map_w, const CUtensorMap& map_x, const Params& p, int grid, cudaStream_t st) {
#define QMM_CASE(NC, KS, SUB) \
  if (nc == NC && sp.ks == KS && sp.sub == SUB) return launch_cfg<WBITS, XT, NC, KS, SUB>(map_w, map_x, p, grid, st)
  QMM_CASE(32, 128, 2);
  QMM_CASE(32, 256, 2);
  QMM_CASE(32, 256, 1);
  QMM_CASE(64, 128, 2);
  QMM_CASE(64, 256, 2);
  QMM_CASE(64, 256, 1);
  QMM_CASE(32, 128, 1);
  QMM_CASE(64, 128, 1);
  QMM_CASE(128, 64, 1);
  QMM_CASE(128, 128, 1);
  QMM_CASE(192, 64, 1);
  QMM_CASE(192, 128, 1);
#undef QMM_CASE
  return fail(QMM_ERR_UNSUPPORTED, "tensor-memory kernel: no instance for %d tokens, steps of %d", nc, sp.ks);
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
  const Plan pl = plan_for(M);
  s.xs_pitch = (pl.ytiles - 1) * pl.th + pl.nc;  // a drain thread reads all of its columns
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
  const Step sp = step_for(pl.nc, block_size);
  const int ks = sp.ks;
  const int stages = (int)ceil_div(K, ks);
  p.blocked = block_size > 0;
  p.S = block_size > 0 ? (int)(K / block_size) : 1;
  // Per channel the sums leave the tensor core about every 512 values all the same: the additions across them are then single
  // fp32 additions in registers, and the drain stays well under the MMAs.
  const int spr = std::max(1, 1024 / (wbits * ks));  // steps per raw tile
  if (block_size > 0) {
    p.fu = (int)std::max<int64_t>(1, block_size / ks);
    p.unit = p.fu;
    while (p.unit % spr != 0) p.unit += p.fu;
  } else {
    const int folds = (int)ceil_div(stages, 512 / ks);
    p.fu = p.unit = (int)align_up((size_t)ceil_div(stages, folds), spr);
    // Up to 128 columns shorter folds where that means fewer steps beyond K: a fold takes a fifth of a step up to 64 tokens, near a half
    // above (int4 [674,768] at 11 tokens, three steps for four, 4.2 us -> 3.8).  int4 with 128 columns: two steps, which both issuers take
    // in turn (0.37 us for 128 values, 0.42 with four on one issuer; [6205,2304] at 92 tokens 15.8 us -> 14.4).  With 192 columns the
    // accumulators ahead are what the epilogue hides under, so folds stay long ([14336,768] at 268 tokens 22.3 us, 23.0 with two steps).
    if (pl.nc <= 128) {
      const double fold = pl.nc <= 64 ? 0.2 : 0.45;
      double best = 1e30;
      for (int fu = spr; fu <= (pl.nc == 128 && wbits == 4 ? 2 : 512 / ks); fu += spr) {
        const double t = (double)align_up((size_t)stages, (size_t)fu) * (1.0 + fold / fu);
        if (t < best) {
          best = t;
          p.fu = p.unit = fu;
        }
      }
    }
  }
  p.fpu = p.unit / p.fu;
  p.ut = (int)ceil_div(stages, p.unit);
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
    // The left-over items are split over s CTAs each where that is sooner done.  A step's time is what its 128 or 256 values take and a
    // share per fold; the exchange (one partial tile per CTA, written, and read by the item's first CTA) about 2 us and a share per
    // CTA.  Where s is not whole, CTAs have parts of two items and the exchanges come one behind the other, 1.75 times as long: int4
    // block 128 [5120,3072] at 96 tokens, 40 items, 17.7 us whole, 16.8 and 16.6 over two and three CTAs, 21.8 over 3.7 (and 33.6
    // against 29.9 whole over 1.3 with 6144 inputs).  Times read off 1036 shapes of five to 260 tiles with s forced; [5120,1536] int8
    // block 384 at 127 tokens 19.6 us by a step's time as of longer folds, 11.7 so.
    const int64_t nc = pl.nc;
    const double per_fold = nc <= 64 ? 0.12 : nc <= 128 ? 0.27 : 0.33, per_zp = !zp || !p.blocked ? 0.0 : nc <= 32 ? 0.06 : nc <= 64 ? 0.12 : 0.3;
    const double per_128 = nc <= 32 ? 0.21 : nc <= 64 ? (wbits == 4 ? 0.25 : 0.36) : nc <= 128 ? 0.3 : 0.38;
    const double step_us = (per_128 + (per_fold + per_zp) * 128.0 / (block_size > 0 ? (double)block_size : (double)(p.fu * ks))) * (ks / 128.0);
    const double share = nc <= 32 ? 0.25 : nc <= 64 ? 0.5 : 0.011 * pl.th, more_ctas = 0.011;
    const double whole_us = p.ut * p.unit * step_us, most = std::min((double)ctas / left, (double)p.ut);
    double best = 0.95 * whole_us, s = 1.0;
    for (int k = 2; k <= (int)std::min(most, 24.0); ++k) {
      const double us = (double)ceil_div(p.ut, k) * p.unit * step_us + 2.0 + share * k + more_ctas * left * (k - 1);
      if (us < best) {
        best = us;
        s = k;
      }
    }
    if (most > (int)most && whole_us / most + 1.75 * (2.0 + share * most) + more_ctas * (ctas - left) < best) s = most;
    if (s > 1.0) {
      p.items1 = items - left;
      p.units = left * p.ut;
      p.g2 = std::min(ctas, std::max(left, (int)(left * s)));
      grid = std::max(std::min(p.items1, ctas), p.g2);
    }
  }

  if (zp) {
    const bool row = p.S == 1 && K >= kLongRow;
    const int64_t pieces = ceil_div(K, std::max<int64_t>(K / p.S, 256));
    const unsigned g = row ? (unsigned)sc.xs_pitch : (unsigned)std::min<int64_t>(1 << 20, ceil_div(sc.xs_pitch * pieces, kSumsThreads / 32));
    auto sums = [&](auto kern, auto* from) { return launch_pdl(kern, g, kSumsThreads, 0, st, from, sc.xs, sc.xs_pitch, (int)M, (int)K, p.S); };
    cudaError_t e;
    if (x_dt == QMM_BF16) {
      auto* from = reinterpret_cast<const __nv_bfloat16*>(x);
      e = row ? sums(block_sums_kernel<__nv_bfloat16, true>, from) : sums(block_sums_kernel<__nv_bfloat16, false>, from);
    } else {
      auto* from = reinterpret_cast<const __half*>(x);
      e = row ? sums(block_sums_kernel<__half, true>, from) : sums(block_sums_kernel<__half, false>, from);
    }
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
    return x_dt == QMM_BF16 ? launch_shape<4, __nv_bfloat16>(pl.nc, sp, map_w, map_x, p, grid, st)
                            : launch_shape<4, __half>(pl.nc, sp, map_w, map_x, p, grid, st);
  return x_dt == QMM_BF16 ? launch_shape<8, __nv_bfloat16>(pl.nc, sp, map_w, map_x, p, grid, st)
                          : launch_shape<8, __half>(pl.nc, sp, map_w, map_x, p, grid, st);
}

}  // namespace qmm
