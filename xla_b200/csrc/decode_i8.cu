// Decode kernel on the warp-level integer tensor cores: K-minor weights (int8 [N,K] or packed int4 [N,K/2]) and up to
// 16 tokens.  The weights are never converted to floating point: int8 bytes are MMA operands as they arrive from HBM,
// int4 nibbles only move into the high half of a byte (three integer instructions per eight weights).
//
//   weight-only   out[m,n] = sum_b (scale[b,n] * sum_{k in b} x[m,k] w[n,k] - zp[b,n] * sum_{k in b} x[m,k])
//                 with every activation rewritten as three int8 limbs relative to its row's largest exponent
//                 (limbs.cuh); a limb row is a column of the MMA, the int32 sums are exact
//   W8A8          the activation row quantized to int8 in the kernel, bit for bit as act_quant.cu does it: one column
//                 per token, exact int32 accumulators, the same fp32 epilogue as the prefill kernel
//
// What bounds it: the weight stream.  At the copy-measured HBM rate an SM sub-partition receives 1 KB of weights
// (16 rows x 64 bytes, one warp step) every 176 cycles; the step costs it about 60 issue slots and, for one 8-column
// tile, 32 (int4) or 16 (int8) cycles of the tensor pipe (mma.sync.m16n8k32 measured at 8 cycles), so up to 48 limb
// columns (16 tokens) stay at or near the stream.  The bf16 form of this loop (decode_mma.cu) converts first: nine
// integer instructions per eight int4 weights at 1.5 cycles each, two per int8 weight.
//
// Work split.  A CTA of 8 or 16 warps owns a contiguous run of 16-row tiles (at most 16) and keeps the limbs of all tokens
// in shared memory.  The (tile, 64-byte step) sequence of the run is dealt to the warps in equal contiguous pieces, so
// every warp streams the same number of bytes whatever N and K, weights stay several steps ahead in a ring of cp.async
// slots private to the warp (48 KB in flight per CTA, across tile boundaries, no registers held), and the warps meet
// once, at the end, to add their pieces of each tile in warp order.  8 warps while two CTAs fit an SM (for small weights
// the second place is the next linear's, whose first weights are then in flight while this one drains), else 16.
//
// Measured (B200, launches back to back over weights larger than L2; decode_mma.cu and limb_gemm.cu in brackets):
//   int4 block 128, one token   [14336,4096] 9.5 us (13.9, 13.5)   [28672,8192] 25.1 (41.9, 28.0)   [8192,28672] 30.0 (55.5, 32.6)
//   int8 per channel, one token [14336,4096] 11.8 us = 5.0 TB/s (16.9, 13.7)   [28672,8192] 43.0 us = 5.5 TB/s (56.9, 39.6)
//   W8A8 [14336,4096]           13.1 us at 1 token, 14.4 at 4, 22 at 12 (any-shape kernel: 113; quantizer + GEMM: 23)
//
// Semantics: torch_xla/experimental/xla_quantized_matmul.py:152-170 (weight-only), :107-114, :134-135 (W8A8).
#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "kernels.h"
#include "limbs.cuh"
#include "quant.cuh"

namespace qmm {

namespace {

constexpr int kRows = 16;       // weight rows per tile = MMA rows
constexpr int kMaxTiles = 16;   // tiles per CTA
constexpr int kMaxTokens = 16;
static_assert(kW8A8DecodeTokens <= kMaxTokens, "per-token words in shared memory");
constexpr size_t kSmemMax = 227 * 1024 - 512;  // static shared memory beside it

struct Args {
  const void* x;
  const uint8_t* w;
  const void* scale;   // [N] or [S,N], of type s_dt
  const void* zp;      // like scale, or null
  void* out;
  int64_t N, K;
  int64_t sc_pitch;    // bytes from one scale block to the next
  int x_dt, out_dt, s_dt, M;
  int steps;           // 64-byte steps per weight row (the last one may be partly outside the row)
  int tiles_lo, tiles_extra;  // tiles per CTA, and how many CTAs take one more
  int fold_steps;      // steps per scale block (0: per channel)
  int fold_shift;      // log2(fold_steps), or -1
  int S;               // scale blocks (1: per channel)
  int scale_tail;      // an odd number of 16-bit block scales
  int gate_up;
  int saturate;        // W8A8: clamp (1) or wrap (0) +128
  int xpitch;          // bytes between limb rows in shared memory
  int raw_off, ring_off, part_off, xs_off;  // offsets of the raw activations, the weight ring, the partial tiles and the
                                            // block sums in shared memory
};

__device__ __forceinline__ void mma_s8(int* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t ev16(uint32_t w) { return (w << 4) & 0xF0F0F0F0u; }  // even k, value * 16
__device__ __forceinline__ uint32_t od16(uint32_t w) { return w & 0xF0F0F0F0u; }         // odd k, value * 16

// Activations -> limbs in shared memory.  Row c = NL * m + l of pitch xpitch holds limb l of token m; int4 weights take
// each group of eight k in the order 0 2 4 6 1 3 5 7, the order in which a word of nibbles expands.  Bytes from K up to
// the end of the last step are zero.  ZP: s_xs[b * NL*M + c] += sum of the limbs over scale block b (integers: exact).
//
// The raw rows come in with cp.async (one round trip to L2 for all of them), end to end behind the first limb rows, and
// are read from shared memory twice, for the row maxima and for the split.  The split goes row by row, so that limbs
// only overwrite raw rows that have been read (raw_offset places them accordingly).  The loops are rolled on purpose:
// this code runs once per CTA, and a long straight-line body costs more in instruction fetches than it saves (unrolled
// 16-fold the whole kernel took twice as long at 4096 x 4096).
template <int WBITS, int NL, bool ZP, int THREADS, typename XT>
__device__ void stage_activations(const Args& p, uint8_t* xs, const XT* raw, float* s_pw, int* s_xs, uint32_t* s_max) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int W = THREADS / 32;
  const int groups = (int)(p.K >> 3), groups_pad = p.steps * (512 / WBITS) / 8;
  const int wpr = p.M > W / 2 ? 1 : p.M > W / 4 ? 2 : p.M > W / 8 ? 4 : 8;  // warps that share a row
  const int cols = NL * p.M;
  const int block_groups = p.fold_steps > 0 ? (int)(p.K / p.S) >> 3 : groups_pad;
  for (int m = warp / wpr; m < p.M; m += W / wpr) {
    uint32_t mx = 0;
#pragma unroll 2
    for (int gi = (warp % wpr) * 32 + lane; gi < groups; gi += 32 * wpr) {
      float v[8];
      load8<XT>(raw + m * (int)p.K + gi * 8, v);
#pragma unroll
      for (int j = 0; j < 8; ++j) mx = max(mx, __float_as_uint(v[j]) & 0x7fffffffu);
    }
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (lane == 0) atomicMax(s_max + m, mx);
  }
  __syncthreads();
#pragma unroll 1
  for (int m = 0; m < p.M; ++m) {
    float mult = 0.f, pw = 0.f, qscale = 0.f, rcp = 0.f;
    if (NL == 3) row_factors<3>(s_max[m], WBITS == 4 ? 0.0625f : 1.f, mult, pw);
    else pw = qscale = quant_scale<XT>(__uint_as_float(s_max[m]));
    const bool fast = NL == 1 && std::is_same<XT, __nv_bfloat16>::value && quant_regular(qscale);
    if (fast) rcp = __frcp_rn(qscale);
    if (tid == 0) s_pw[m] = pw;
    uint8_t* r0 = xs + NL * m * p.xpitch;
#pragma unroll 1
    for (int g0 = warp * 32; g0 < groups_pad; g0 += THREADS) {
      const int gi = g0 + lane;
      uint32_t l0[2] = {0, 0}, l1[2] = {0, 0}, l2[2] = {0, 0};
      if (gi < groups) {
        float v[8];
        load8<XT>(raw + m * (int)p.K + gi * 8, v);
        if (NL == 3) {
          split8<3>(v, mult, l0, l1, l2);
        } else if (fast) {
          int q[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) q[j] = quantize_bf16_regular(v[j], qscale, rcp, p.saturate != 0);
          l0[0] = pack_bytes(q);
          l0[1] = pack_bytes(q + 4);
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j)
            l0[j >> 2] |= (uint32_t)(uint8_t)quantize_value<XT>(v[j], qscale, p.saturate != 0) << (8 * (j & 3));
        }
      }
      if (gi < groups_pad) {
        auto put = [&](uint8_t* r, const uint32_t* l) {
          if (WBITS == 4)
            *reinterpret_cast<uint2*>(r + gi * 8) = make_uint2(__byte_perm(l[0], l[1], 0x6420), __byte_perm(l[0], l[1], 0x7531));
          else
            *reinterpret_cast<uint2*>(r + gi * 8) = make_uint2(l[0], l[1]);
        };
        put(r0, l0);
        if (NL == 3) {
          put(r0 + p.xpitch, l1);
          put(r0 + 2 * p.xpitch, l2);
        }
      }
      if (ZP) {
        // eight neighbouring lanes hold 64 values: always inside one scale block
        auto sum = [&](const uint32_t* l) {
          int s = __dp4a((int)l[1], 0x01010101, __dp4a((int)l[0], 0x01010101, 0));
#pragma unroll
          for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
          return s;
        };
        const int s0 = sum(l0), s1 = NL == 3 ? sum(l1) : 0, s2 = NL == 3 ? sum(l2) : 0;
        if ((lane & 7) == 0 && gi < groups) {
          int* d = s_xs + (gi / block_groups) * cols + NL * m;
          atomicAdd(d, s0);
          if (NL == 3) {
            atomicAdd(d + 1, s1);
            atomicAdd(d + 2, s2);
          }
        }
      }
    }
    __syncthreads();
  }
}

// Where the raw rows start: row m's limbs must end before raw row m does begin, for every m.
__host__ inline int64_t raw_offset(int64_t limb_bytes, int64_t raw_bytes, int64_t M) {
  return limb_bytes >= raw_bytes ? limb_bytes * M - raw_bytes * (M - 1) : limb_bytes;
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
template <int BYTES>
__device__ __forceinline__ void cp_async_small(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst), "l"(src), "n"(BYTES) : "memory");
}

// A ring slot holds one 64-byte step of a tile: 16 bytes of weight rows g and g + 8 for each lane, and the step's block
// scales and zero points for the 16 rows (NB sets: a step of int4 weights holds two scale blocks of 64).
__host__ __device__ constexpr int slot_bytes(bool blocked, int nb) { return 1024 + (blocked ? nb * 128 : 0); }

// W warps: 8 where two CTAs fit an SM's shared memory, 16 where only one does.
template <int W>
constexpr int kDepth = W == 8 ? 7 : 4;  // ring slots per warp

template <int WBITS, int NL, int NT, bool BLOCKED, bool ZP, bool HALF, int W, bool W16>
__global__ void __launch_bounds__(W * 32, W == 8 ? 2 : 1) decode_i8_kernel(const Args p) {
  constexpr int kWarps = W, kThreads = W * 32, D = kDepth<W>;
  constexpr int VPS = 512 / WBITS;
  constexpr int NB = HALF ? 2 : 1;
  constexpr int NC = NT * 8;
  constexpr int NA = NT <= 2 ? 2 : 1;  // accumulator sets: shorter MMA chains where a step has few of them
  constexpr int kSlot = slot_bytes(BLOCKED, NB);
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ uint32_t s_max[kMaxTokens];
  __shared__ float s_pw[kMaxTokens];
  __shared__ uint8_t s_first[kMaxTiles];  // first warp whose piece reaches into a tile
  uint8_t* xs = smem;
  int* s_xs = reinterpret_cast<int*>(smem + p.xs_off);

  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  // tiles are dealt to the CTAs in contiguous runs that differ by at most one
  const int t0 = blockIdx.x * p.tiles_lo + min((int)blockIdx.x, p.tiles_extra);
  const int nt_cta = p.tiles_lo + ((int)blockIdx.x < p.tiles_extra ? 1 : 0);
  const int SP = p.steps, total_steps = nt_cta * SP;
  const int lo = warp * total_steps / kWarps, hi = (warp + 1) * total_steps / kWarps;
  const int64_t pitch = p.K * WBITS / 8;
  const int cols = NL * p.M;
  const int n_last = (int)p.N - 1;

  if ((int)threadIdx.x < nt_cta) {
    int wv = 0;
    while ((wv + 1) * total_steps / kWarps <= (int)threadIdx.x * SP) ++wv;
    s_first[threadIdx.x] = (uint8_t)wv;
  }

  // ---- load position (runs up to D - 1 steps ahead of the compute position) ----
  const uint32_t ring = (uint32_t)__cvta_generic_to_shared(smem + p.ring_off) + warp * (D * kSlot);
  int left = hi - lo, ltile = t0 + lo / SP, ls = lo - lo / SP * SP;
  const int piece_first = ls;
  uint32_t ldst = ring;
  const uint8_t *lp0, *lp1;
  const uint8_t* lsc = nullptr;  // this lane's row of the scales (lanes 0..15) or zero points (lanes 16..31)
  auto scale_row = [&](int tile) {
    return static_cast<const uint8_t*>(ZP && lane >= 16 ? p.zp : p.scale) + min(tile * kRows + (lane & 15), n_last) * (int64_t)(W16 ? 2 : 4);
  };
  // the block scales and zero points of a step, into its ring slot
  auto copy_scales = [&](uint32_t slot, const uint8_t* row, int step) {
    if (!ZP && lane >= 16) return;
    auto copy = [&](uint32_t dst, int b) {
      const uint8_t* src = row + b * p.sc_pitch;
      if (W16 && p.scale_tail && b + 1 == p.S && row == scale_row(n_last / kRows + 1)) copy_last_scale(dst, src);
      else copy_scale_word<W16>(dst, src);
    };
    if constexpr (HALF) {
      copy(slot + 1024 + lane * 4, 2 * step);
      if (2 * step + 1 < p.S) copy(slot + 1152 + lane * 4, 2 * step + 1);
    } else {
      copy(slot + 1024 + lane * 4, p.fold_shift >= 0 ? step >> p.fold_shift : step / p.fold_steps);
    }
  };
  auto set_tile = [&]() {
    // rows beyond N repeat the last one; they are not stored
    const int n0 = min(ltile * kRows + g, n_last), n1 = min(ltile * kRows + g + 8, n_last);
    lp0 = p.w + n0 * pitch + (HALF ? 8 : 16) * t;
    lp1 = p.w + n1 * pitch + (HALF ? 8 : 16) * t;
    if (BLOCKED) lsc = scale_row(ltile);
  };
  set_tile();
  lp0 += (int64_t)ls * 64;
  lp1 += (int64_t)ls * 64;
  auto issue = [&](bool with_scales) {
    if (left > 0) {
      --left;
      const uint32_t d = ldst + lane * 16;
      const int room = (int)pitch - ls * 64;  // bytes of the row from this step on: a ragged row ends inside its last step
      if constexpr (HALF) {
        cp_async_small<8>(d, lp0);
        cp_async_small<8>(d + 512, lp1);
        if (room > 32) {
          cp_async_small<8>(d + 8, lp0 + 32);
          cp_async_small<8>(d + 520, lp1 + 32);
        }
      } else if (16 * t < room) {
        cp_async16(d, lp0);
        cp_async16(d + 512, lp1);
      }
      if (BLOCKED && with_scales) copy_scales(ldst, lsc, ls);
      ldst = ldst + kSlot == ring + D * kSlot ? ring : ldst + kSlot;
      lp0 += 64;
      lp1 += 64;
      if (++ls == SP) {
        ls = 0;
        ++ltile;
        set_tile();
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int d = 0; d < D - 1; ++d) issue(false);
  // The weights are static: their first loads run under the kernel before this one.  Scales, activations, and every store
  // of this kernel, come after the wait.
  auto first_scales = [&](auto take) {
    int step = piece_first, scale_tile = t0 + lo / SP;
#pragma unroll 1
    for (int d = 0; d < min(D - 1, hi - lo); ++d) {
      take(ring + d * kSlot, scale_row(scale_tile), step);
      if (++step == SP) {
        step = 0;
        ++scale_tile;
      }
    }
  };
  if constexpr (BLOCKED) first_scales([&](uint32_t, const uint8_t* row, int step) {
    prefetch_l2(row + (HALF ? 2 * step : p.fold_shift >= 0 ? step >> p.fold_shift : step / p.fold_steps) * p.sc_pitch);
  });
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  {
    const uint8_t* raw = smem + p.raw_off;
    const int bytes = p.M * (int)p.K * (p.x_dt == QMM_F32 ? 4 : 2);  // a multiple of 16: K is one of 16
    for (int o = threadIdx.x * 16; o < bytes; o += kThreads * 16)
      cp_async16((uint32_t)__cvta_generic_to_shared(raw + o), reinterpret_cast<const uint8_t*>(p.x) + o);
    asm volatile("cp.async.commit_group;" ::: "memory");
    // the first steps' scales, behind the weights under way, are waited for when the activations have been split
    if constexpr (BLOCKED) first_scales(copy_scales);
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (threadIdx.x < kMaxTokens) s_max[threadIdx.x] = 0;
    if (ZP)
      for (int i = threadIdx.x; i < p.S * cols; i += kThreads) s_xs[i] = 0;
    // groups complete in order: the activations' with the weights' first steps
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    if (p.x_dt == QMM_BF16)
      stage_activations<WBITS, NL, ZP, kThreads>(p, xs, reinterpret_cast<const __nv_bfloat16*>(raw), s_pw, s_xs, s_max);
    else if (p.x_dt == QMM_F16)
      stage_activations<WBITS, NL, ZP, kThreads>(p, xs, reinterpret_cast<const __half*>(raw), s_pw, s_xs, s_max);
    else if constexpr (NL == 1)
      stage_activations<WBITS, NL, ZP, kThreads>(p, xs, reinterpret_cast<const float*>(raw), s_pw, s_xs, s_max);
  }

  // B operand rows of this lane: limb row 8*i + g (rows beyond the last one read row 0; their columns are not used)
  const uint8_t* xrow[NT];
#pragma unroll
  for (int i = 0; i < NT; ++i) xrow[i] = xs + (size_t)(8 * i + g < cols ? 8 * i + g : 0) * p.xpitch + (WBITS == 4 && !HALF ? 32 : 16) * t;

  int acc[NA][NT][4];
  float total[BLOCKED ? NT : 1][4];
  auto clear = [&](bool totals) {
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        acc[0][i][j] = acc[NA - 1][i][j] = 0;
        if (BLOCKED && totals) total[i][j] = 0.f;
      }
  };
  clear(true);
  auto sum_of = [&](int i, int j) { return NA == 2 ? acc[0][i][j] + acc[1][i][j] : acc[0][i][j]; };

  // partial tiles [slot][row][NC]: a piece that crosses from tile i into the next leaves its part of tile i in slot i
  // of the region behind the limbs (one warp per tile does); every warp leaves its last tile in slot `warp` of a
  // region over the limbs, once those have been read
  auto put_partial = [&](void* base, int slot) {
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      const int o = (slot * kRows + g) * NC + 8 * i + 2 * t;
      if constexpr (NL == 1) {
        int* d = reinterpret_cast<int*>(base) + o;
        *reinterpret_cast<int2*>(d) = make_int2(sum_of(i, 0), sum_of(i, 1));
        *reinterpret_cast<int2*>(d + 8 * NC) = make_int2(sum_of(i, 2), sum_of(i, 3));
      } else {
        float* d = reinterpret_cast<float*>(base) + o;
        float v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = BLOCKED ? total[i][j] : __int2float_rn(sum_of(i, j));
        *reinterpret_cast<float2*>(d) = make_float2(v[0], v[1]);
        *reinterpret_cast<float2*>(d + 8 * NC) = make_float2(v[2], v[3]);
      }
    }
  };

  // scale block b ends here: total += scale * sums, and (once per block: by the warp that runs its last step) the
  // zero-point term
  auto fold = [&](const uint32_t* sc, int b, bool zp_too) {
    if constexpr (BLOCKED) {
      // (rows g and g + 8 of a tile, which starts at an even row)
      auto value = [&](int i) { return scale_in<W16>(sc + i, g, b, (int)p.N, p.s_dt); };
      const float s0 = value(g), s1 = value(g + 8);
#pragma unroll
      for (int i = 0; i < NT; ++i) {
        total[i][0] = fmaf(s0, __int2float_rn(sum_of(i, 0)), total[i][0]);
        total[i][1] = fmaf(s0, __int2float_rn(sum_of(i, 1)), total[i][1]);
        total[i][2] = fmaf(s1, __int2float_rn(sum_of(i, 2)), total[i][2]);
        total[i][3] = fmaf(s1, __int2float_rn(sum_of(i, 3)), total[i][3]);
      }
      clear(false);
      if constexpr (ZP) {
        if (zp_too) {
          constexpr float kW = WBITS == 4 ? 16.f : 1.f;  // the weight sums carry this factor
          const float z0 = -kW * value(16 + g), z1 = -kW * value(24 + g);
#pragma unroll
          for (int i = 0; i < NT; ++i) {
            const int c = 8 * i + 2 * t;
            const float x0 = c < cols ? (float)s_xs[b * cols + c] : 0.f, x1 = c + 1 < cols ? (float)s_xs[b * cols + c + 1] : 0.f;
            total[i][0] = fmaf(z0, x0, total[i][0]);
            total[i][1] = fmaf(z0, x1, total[i][1]);
            total[i][2] = fmaf(z1, x0, total[i][2]);
            total[i][3] = fmaf(z1, x1, total[i][3]);
          }
        }
      }
    }
  };

  asm volatile("cp.async.wait_group 0;" ::: "memory");  // the first scales
  int cs = piece_first, tile = lo / SP;  // compute position
  const uint8_t* cring = smem + p.ring_off + warp * (D * kSlot);
  int cslot = 0;
  for (int j = lo; j < hi; ++j) {
    asm volatile("cp.async.wait_group %0;" ::"n"(D - 2) : "memory");
    __syncwarp();
    issue(true);  // into the slot of the step before this one, which every lane has read
    const uint8_t* slot = cring + cslot;
    cslot = cslot + kSlot == D * kSlot ? 0 : cslot + kSlot;
    const uint32_t* sc = reinterpret_cast<const uint32_t*>(slot + 1024);
    const uint4 a = *reinterpret_cast<const uint4*>(slot + lane * 16), b = *reinterpret_cast<const uint4*>(slot + 512 + lane * 16);
    if constexpr (WBITS == 8) {
#pragma unroll
      for (int i = 0; i < NT; ++i) {
        const uint4 xv = *reinterpret_cast<const uint4*>(xrow[i] + cs * 64);
        mma_s8(acc[0][i], a.x, b.x, a.y, b.y, xv.x, xv.y);
        mma_s8(acc[NA - 1][i], a.z, b.z, a.w, b.w, xv.z, xv.w);
      }
    } else {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint32_t wa0 = h ? a.z : a.x, wa1 = h ? a.w : a.y, wb0 = h ? b.z : b.x, wb1 = h ? b.w : b.y;
#pragma unroll
        for (int i = 0; i < NT; ++i) {
          const uint4 xv = *reinterpret_cast<const uint4*>(xrow[i] + cs * VPS + (HALF ? 64 * h : 16 * h));
          mma_s8(acc[0][i], ev16(wa0), ev16(wb0), od16(wa0), od16(wb0), xv.x, xv.y);
          mma_s8(acc[NA - 1][i], ev16(wa1), ev16(wb1), od16(wa1), od16(wb1), xv.z, xv.w);
        }
        if constexpr (HALF)
          if (2 * cs + h < p.S) fold(sc + 32 * h, 2 * cs + h, true);
      }
    }
    const bool tile_end = cs + 1 == SP;
    if constexpr (BLOCKED && !HALF) {
      const bool block_end = p.fold_shift >= 0 ? ((cs + 1) & (p.fold_steps - 1)) == 0 : (cs + 1) % p.fold_steps == 0;
      if (block_end || j + 1 == hi) fold(sc, p.fold_shift >= 0 ? cs >> p.fold_shift : cs / p.fold_steps, block_end);
    }
    ++cs;
    if (tile_end) {
      cs = 0;
      if (j + 1 < hi) {
        put_partial(smem + p.part_off, tile);
        clear(true);
      }
      ++tile;
    }
  }
  __syncthreads();  // the limbs have been read
  if (lo < hi) put_partial(smem, warp);
  __syncthreads();

  // ---- add the warps' pieces of each tile, in warp order, and store ----
  const int rows = nt_cta * kRows;
  auto value = [&](int row, int m) -> float {
    const int n = t0 * kRows + row;
    const int lt = row >> 4, last = (lt + 1) * SP, r = row & 15;
    int ai = 0;
    float a[3] = {0.f, 0.f, 0.f};
    for (int wv = s_first[lt]; wv < kWarps && wv * total_steps / kWarps < last; ++wv) {
      const int phi = (wv + 1) * total_steps / kWarps;
      if (phi == wv * total_steps / kWarps) continue;  // fewer steps than warps: an empty piece
      const bool in_last = phi <= last;  // this tile is the piece's last one
      const uint8_t* base = in_last ? smem : smem + p.part_off;
      const int o = ((in_last ? wv : lt) * kRows + r) * NC + NL * m;
      if constexpr (NL == 1) {
        ai += reinterpret_cast<const int*>(base)[o];
      } else {
#pragma unroll
        for (int l = 0; l < 3; ++l) a[l] += reinterpret_cast<const float*>(base)[o + l];
      }
    }
    if constexpr (NL == 1) {
      const float z = ZP ? load_as_f32(p.zp, n, p.s_dt) : 0.f;
      return w8a8_dequant(ai, load_as_f32(p.scale, n, p.s_dt), ZP ? &z : nullptr, ZP ? s_xs[m] : 0, s_pw[m]);
    } else {
      float v = fmaf(65536.f, a[2], fmaf(256.f, a[1], a[0]));
      if constexpr (!BLOCKED) {
        v *= load_as_f32(p.scale, n, p.s_dt);
        if constexpr (ZP) {
          constexpr float kW = WBITS == 4 ? 16.f : 1.f;
          const float xsum = fmaf(65536.f, (float)s_xs[3 * m + 2], fmaf(256.f, (float)s_xs[3 * m + 1], (float)s_xs[3 * m]));
          v = fmaf(-kW * load_as_f32(p.zp, n, p.s_dt), xsum, v);
        }
      }
      return v * s_pw[m];
    }
  };
  // consecutive threads -> consecutive n of one token
  for (int row = threadIdx.x % 64, m = threadIdx.x / 64; m < p.M;) {
    const int n = t0 * kRows + row;
    if (row < rows && n <= n_last) {
      if (!p.gate_up) {
        store_from_f32(p.out, (int64_t)m * p.N + n, p.out_dt, value(row, m));
      } else if ((row & 8) == 0) {
        // rows come in groups of 16: eight gate rows, then the eight up rows of the same outputs
        const float v = value(row, m), u = value(row + 8, m);
        store_from_f32(p.out, (int64_t)m * (p.N >> 1) + ((n >> 4) << 3) + (n & 7), p.out_dt, v / (1.f + expf(-v)) * u);
      }
    }
    row += 64;
    if (row >= rows) {
      row = threadIdx.x % 64;
      m += kThreads / 64;
    }
  }
}

// W = 8: up to two CTAs per SM, W = 16: one.  Weights of few tiles per SM get one CTA per SM either way: the second
// place is then the next kernel's (4096 x 4096 int8: 5.5 us with 148 CTAs of one or two tiles).  More CTAs than places
// only when a CTA would get more than kMaxTiles tiles, and then whole rounds.
int grid_for(int64_t N, int warps) {
  const int64_t tiles = ceil_div(N, kRows), sms = sm_count();
  const int64_t places = warps == 8 && tiles >= 4 * sms ? 2 * sms : sms;
  return (int)std::min<int64_t>(tiles, places * ceil_div(tiles, places * kMaxTiles));
}

struct Layout {
  int warps, grid, xpitch, raw_off, ring_off, part_off, xs_off;
  size_t bytes;
};

int tiles_n(int cols) { return cols <= 8 ? 1 : cols <= 16 ? 2 : cols <= 24 ? 3 : cols <= 32 ? 4 : 6; }

Layout layout_with(int warps, int wbits, int nl, int xbytes, int64_t M, int64_t N, int64_t K, int64_t S, bool blocked, bool half,
                   bool zp) {
  Layout l;
  l.warps = warps;
  l.grid = grid_for(N, warps);
  // Limb rows end on a multiple of a step and are pitched so that the 16-byte fragment reads of a quarter warp (two rows
  // x four k spans) fall on distinct banks: 64 bytes off for int8 and for blocks of 64 (spans of 16 bytes), 16 for int4
  // (spans of 32).
  const int64_t vps = 512 / wbits, kpad = ceil_div(ceil_div(K, vps) * vps, 128) * 128;
  l.xpitch = (int)(kpad + ((wbits == 8 || half) ? 64 : 16));
  const int64_t limbs = (int64_t)nl * l.xpitch, raw = K * xbytes, part = (int64_t)kRows * tiles_n((int)(nl * M)) * 8 * 4;
  l.raw_off = (int)raw_offset(limbs, raw, M);
  const int64_t x = std::max(std::max(limbs * M, l.raw_off + raw * M), warps * part);
  l.ring_off = (int)(ceil_div(x, 128) * 128);
  l.part_off = l.ring_off + warps * (warps == 8 ? kDepth<8> : kDepth<16>) * slot_bytes(blocked, half ? 2 : 1);
  l.xs_off = l.part_off + (int)((ceil_div(ceil_div(N, kRows), l.grid) - 1) * part);
  l.bytes = l.xs_off + (zp ? (size_t)S * nl * M * 4 : 0);
  return l;
}

Layout layout_for(int wbits, int nl, int xbytes, int64_t M, int64_t N, int64_t K, int64_t S, bool blocked, bool half, bool zp) {
  const Layout l = layout_with(8, wbits, nl, xbytes, M, N, K, S, blocked, half, zp);
  if (2 * (l.bytes + 1024 + 512) <= 228 * 1024) return l;
  return layout_with(16, wbits, nl, xbytes, M, N, K, S, blocked, half, zp);
}

template <int WBITS, int NL, int NT, bool BLOCKED, bool ZP, bool HALF, int W, bool W16>
int launch_with(const Args& a, const Layout& l, cudaStream_t st) {
  auto kern = decode_i8_kernel<WBITS, NL, NT, BLOCKED, ZP, HALF, W, W16>;
  static bool configured[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax);
    if (e != cudaSuccess) return fail(QMM_ERR_LAUNCH, "cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    if (dev >= 0 && dev < 64) configured[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)l.grid);
  cfg.blockDim = dim3(W * 32);
  cfg.dynamicSmemBytes = l.bytes;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, a);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(QMM_ERR_LAUNCH, "decode_i8_kernel launch: %s", cudaGetErrorString(e));
  }
  return QMM_OK;
}

template <int WBITS, int NL, int NT, bool BLOCKED, bool ZP, bool HALF, int W>
int launch_one(const Args& a, const Layout& l, cudaStream_t st) {
  if constexpr (BLOCKED)
    if (a.s_dt != QMM_F32) return launch_with<WBITS, NL, NT, BLOCKED, ZP, HALF, W, true>(a, l, st);
  return launch_with<WBITS, NL, NT, BLOCKED, ZP, HALF, W, false>(a, l, st);
}

template <int WBITS, int NL, bool BLOCKED, bool ZP, bool HALF>
int launch_nt(int nt, const Args& a, const Layout& l, cudaStream_t st) {
#define QMM_CASE(NT)                                                               \
  return l.warps == 8 ? launch_one<WBITS, NL, NT, BLOCKED, ZP, HALF, 8>(a, l, st) \
                      : launch_one<WBITS, NL, NT, BLOCKED, ZP, HALF, 16>(a, l, st)
  switch (nt) {
    case 1: QMM_CASE(1);
    case 2: QMM_CASE(2);
  }
  if constexpr (NL == 3) {
    switch (nt) {
      case 3: QMM_CASE(3);
      case 4: QMM_CASE(4);
      default: QMM_CASE(6);
    }
  }
  return fail(QMM_ERR_UNSUPPORTED, "decode kernel: too many tokens");
#undef QMM_CASE
}

template <int WBITS, bool ZP>
int launch_blocks(int nt, bool blocked, bool half, const Args& a, const Layout& l, cudaStream_t st) {
  if (!blocked) return launch_nt<WBITS, 3, false, ZP, false>(nt, a, l, st);
  if constexpr (WBITS == 4)
    if (half) return launch_nt<WBITS, 3, true, ZP, true>(nt, a, l, st);
  return launch_nt<WBITS, 3, true, ZP, false>(nt, a, l, st);
}

bool half_blocks(int wbits, int64_t block_size) { return wbits == 4 && block_size == 64; }

// Shapes both forms share.  K in whole 16-byte pieces of a weight row; the limbs of all tokens in shared memory.
bool shape_ok(int wbits, int nl, int xbytes, int64_t M, int64_t N, int64_t K, int64_t block_size, bool zp) {
  if (M < 1 || N < 1 || K < 64) return false;
  if (K * wbits / 8 % 16 != 0 || K > (1 << 16) || N > (1LL << 24)) return false;
  if (block_size > 0 && (K % block_size != 0 || (block_size % (512 / wbits) != 0 && !half_blocks(wbits, block_size)))) return false;
  return layout_for(wbits, nl, xbytes, M, N, K, block_size > 0 ? K / block_size : 1, block_size > 0, half_blocks(wbits, block_size), zp).bytes <= kSmemMax;
}

Args make_args(int wbits, const void* x, int x_dt, const void* w, const Scales& sc, void* out, int out_dt, int64_t M,
               int64_t N, int64_t K, int64_t block_size, const Layout& l) {
  Args a = {};
  a.x = x;
  a.w = reinterpret_cast<const uint8_t*>(w);
  a.scale = sc.scale;
  a.zp = sc.zp;
  a.s_dt = sc.dt;
  a.sc_pitch = N * (int64_t)dtype_size(sc.dt);
  a.out = out;
  a.N = N;
  a.K = K;
  a.x_dt = x_dt;
  a.out_dt = out_dt;
  a.M = (int)M;
  const int64_t vps = 512 / wbits;
  a.steps = (int)ceil_div(K, vps);
  const int tiles = (int)ceil_div(N, kRows);
  a.tiles_lo = tiles / l.grid;
  a.tiles_extra = tiles % l.grid;
  a.S = block_size > 0 ? (int)(K / block_size) : 1;
  a.scale_tail = scale_tail(sc, a.S, N);
  a.fold_steps = block_size > 0 ? std::max(1, (int)(block_size / vps)) : 0;
  a.fold_shift = -1;
  for (int s = 0; s < 16; ++s)
    if (a.fold_steps == 1 << s) a.fold_shift = s;
  a.xpitch = l.xpitch;
  a.raw_off = l.raw_off;
  a.ring_off = l.ring_off;
  a.part_off = l.part_off;
  a.xs_off = l.xs_off;
  return a;
}

}  // namespace

bool decode_i8_supported(int wbits, int64_t M, int64_t N, int64_t K, int64_t block_size, const void* x, int x_dt, const void* w,
                         bool has_zp) {
  if (x_dt != QMM_BF16 && x_dt != QMM_F16) return false;
  if (M > kMaxTokens || !shape_ok(wbits, 3, 2, M, N, K, block_size, has_zp)) return false;
  return aligned(x, 16) && aligned(w, 16);
}

int launch_decode_i8(int wbits, const void* x, int x_dt, const void* w, const Scales& sc, void* out, int out_dt, int64_t M, int64_t N,
                     int64_t K, int64_t block_size, int gate_up, cudaStream_t st) {
  const bool zp = sc.zp != nullptr;
  if (gate_up && N % 16 != 0)
    return fail(QMM_ERR_BAD_SHAPE, "fused gate/up epilogue: the interleaved weight needs a multiple of 16 rows, got %lld", (long long)N);
  if (!decode_i8_supported(wbits, M, N, K, block_size, x, x_dt, w, zp) || !scale_words_ok(sc, block_size))
    return fail(QMM_ERR_UNSUPPORTED, "integer decode kernel: M=%lld N=%lld K=%lld bs=%lld not supported", (long long)M, (long long)N,
                (long long)K, (long long)block_size);
  const bool half = half_blocks(wbits, block_size);
  const Layout l = layout_for(wbits, 3, 2, M, N, K, block_size > 0 ? K / block_size : 1, block_size > 0, half, zp);
  Args a = make_args(wbits, x, x_dt, w, sc, out, out_dt, M, N, K, block_size, l);
  a.gate_up = gate_up;
  const int nt = tiles_n((int)(3 * M));
  const bool blocked = block_size > 0;
  if (wbits == 4)
    return zp ? launch_blocks<4, true>(nt, blocked, half, a, l, st) : launch_blocks<4, false>(nt, blocked, half, a, l, st);
  return zp ? launch_blocks<8, true>(nt, blocked, half, a, l, st) : launch_blocks<8, false>(nt, blocked, half, a, l, st);
}

bool decode_w8a8_supported(int64_t M, int64_t N, int64_t K, const void* x, int x_dt, const void* w, bool has_zp) {
  if (M > kW8A8DecodeTokens || !shape_ok(8, 1, (int)dtype_size(x_dt), M, N, K, 0, has_zp)) return false;
  return aligned(x, 16) && aligned(w, 16);
}

int launch_decode_w8a8(const void* x, int x_dt, const int8_t* w, const Scales& sc, void* out, int out_dt, int64_t M, int64_t N,
                       int64_t K, int saturate, cudaStream_t st) {
  const bool zp = sc.zp != nullptr;
  if (!decode_w8a8_supported(M, N, K, x, x_dt, w, zp))
    return fail(QMM_ERR_UNSUPPORTED, "W8A8 decode kernel: M=%lld N=%lld K=%lld not supported", (long long)M, (long long)N, (long long)K);
  const Layout l = layout_for(8, 1, (int)dtype_size(x_dt), M, N, K, 1, false, false, zp);
  Args a = make_args(8, x, x_dt, w, sc, out, out_dt, M, N, K, 0, l);
  a.saturate = saturate;
  const int nt = tiles_n((int)M);
  return zp ? launch_nt<8, 1, false, true, false>(nt, a, l, st) : launch_nt<8, 1, false, false, false>(nt, a, l, st);
}

}  // namespace qmm
