// int8 x int8 -> int32 products of long batches on pairs of CTAs, for weights with a scale per output:
//
//   acc[n,c] = sum_k w[n,k] * b[c,k]          w: int8 weights [N,K]; b: int8 rows [NL * M, K], NL of them per token
//
//   NL = 1   W8A8: b is the quantized batch;       out[m,n] = ((float)acc * scale[n] - (float)rowsum[m] * zp[n]) * x_scale[m]
//   NL > 1   weight-only: b are the activations' limbs (limb_gemm.cu);
//                                                  out[m,n] = (sum_i 256^i acc_i * scale[n] - zp[n] * xsum[m]) * 2^(e_m - q)
//
// What bounds the single-CTA kernels for these shapes is the shared-memory port, 128 bytes a cycle for what TMA writes and the
// MMA reads: a 128 x 128 tile moves 32 KB in and 32 KB out for 256 cycles of MMAs (limb_gemm.cu; measured 1035 cycles where
// the port needs 1024), the 128 x 256 tile of w8a8_gemm.cu 48 KB each way for 512.  Here the two CTAs of a cluster, on the two
// SMs of a TPC, issue one MMA of 256 weight rows x 256 columns (tcgen05 cta_group::2): each holds its 128 rows of weights and
// half of the columns, and the hardware gives each tensor core the other half: 32 KB each way for 512 cycles.
//
//   warp 0        TMA: this CTA's weight rows and columns, 128 rows x 128 bytes of each per stage
//   warp 1        of the leader: MMA issuer, four tcgen05.mma.kind::i8 (M256 N256 K32) per stage for both CTAs; its commits free
//                 the stage and hand the accumulators over in both
//   warp 2        tensor memory
//   warps 4..11   epilogue: thread = weight row (its TMEM lane), half of the tile's tokens, sixteen at a time
//
// Two accumulators of 256 columns: the epilogue of one tile runs under the main loop of the next.
//
// Semantics: torch_xla/experimental/xla_quantized_matmul.py:107-118, :134-135; pallas_kernels/quantized_matmul_kernel.py:101-121.
#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "kernels.h"
#include "ptx_sm100.cuh"

namespace qmm {

namespace {

constexpr int kRows = 128;                        // weight rows per CTA; a pair has 256 (UMMA M)
constexpr int kCols = 256;                        // columns per tile (UMMA N); a CTA holds half of them
constexpr int kBK = 128;                          // int8 values per stage = one 128-byte swizzle row
constexpr int kStages = 6;
constexpr uint32_t kHalf = kRows * kBK;           // 16 KB: the weights of a stage, and its columns
constexpr uint32_t kStageBytes = 2 * kHalf;
constexpr int kThreads = 384;
constexpr int kDrain = 256;
constexpr size_t kSmem = 1024 + (size_t)kStages * kStageBytes + 2 * 2 * kCols * 4 + 256;

// Tokens per tile, and of a drain group (whole chunks of 16; the last chunk of a tile is moved back to end with it)
template <int NL>
struct Tile {
  static constexpr int kTokens = NL == 3 ? 84 : kCols / NL;
  static constexpr int kGroup = NL == 3 ? 48 : kTokens / 2;
  static_assert(kTokens * NL <= kCols && kTokens >= 16 && kGroup % 16 == 0 && 2 * kGroup >= kTokens, "tokens of a tile");
};

struct Params {
  const void* scale;  // [N], of type s_dt
  const void* zp;     // like scale, or null
  int s_dt;
  const float* tok;   // [M]: a factor per token
  const void* sums;   // with zp: [M] sums of the activations, fp32 (weight-only) or int32 (W8A8)
  float zp_mul;
  void* out;
  int out_dt;
  int out_pairs;      // a row's outputs 2i and 2i + 1 may be written with one 4-byte store
  int M;
  int64_t N;
  int64_t ld;
  int k_blocks;
  int ytiles;
  // (row tile, column tile) items, column tiles first: items1 of them whole, pair c takes c, c + pairs, ...; the rest (of a partly
  // filled last round, or all of few) in `units` of kUnit stages, dealt in equal contiguous shares to the first g2 pairs
  int items1;
  int units;
  int ut;             // units per item
  int g2;
  float* partial;     // [place of the deal][CTA][tokens / 4][128][4]
  uint32_t* flags;    // [place of the deal][CTA], zero between launches
  long long wait_cycles;
  int w_dep;          // the weights are written by the kernel before this one
  uint32_t* err_word;
};

constexpr int kUnit = 4;          // stages
constexpr int kPairMostPairs = 80;
enum PairErr : uint32_t { kErrPartialPair = 11 };  // an item's first pair never saw the sums of the pairs that continue it

// The fragments of this pair, in order: whole items, then its share of the dealt units.  The units go to the pairs from the last
// one down, so that a pair waits only for sums of pairs with lower indices, which have started already.
struct FragIter {
  const Params& p;
  int u, hi, nxt, pairs, item, u0, u1;
  __device__ explicit FragIter(const Params& p) : p(p), nxt(blockIdx.x >> 1), pairs(gridDim.x >> 1), item(0), u0(0), u1(0) {
    const int c = place();
    u = c >= 0 ? share(c) : 0;
    hi = c >= 0 ? share(c + 1) : 0;
  }
  __device__ int place() const { return p.g2 - 1 - (int)(blockIdx.x >> 1); }
  __device__ int share(int c) const { return (int)((long long)c * p.units / p.g2); }
  __device__ bool next() {
    if (nxt < p.items1) {
      item = nxt;
      nxt += pairs;
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
    return true;
  }
  __device__ int k0() const { return u0 * kUnit; }
  __device__ int k1() const { return min(p.k_blocks, u1 * kUnit); }
};

// ---- pairs: PTX of this kernel ----
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Arrives on the leader's barrier at the same place
__device__ __forceinline__ void arrive_leader(uint64_t* bar) {
  asm volatile(
      "{\n\t"
      ".reg .b32 a;\n\t"
      "mapa.shared::cluster.u32 a, %0, 0;\n\t"
      "mbarrier.arrive.release.cluster.shared::cluster.b64 _, [a];\n\t"
      "}" ::"r"(ptx::smem_u32(bar))
      : "memory");
}
// As ptx::mbar_wait by a whole warp, for arrivals from the other CTA
__device__ __forceinline__ bool try_wait_cluster(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t"
      "}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return __all_sync(0xffffffffu, ok != 0);
}
__device__ __forceinline__ void wait_cluster(uint32_t bar, uint32_t parity, volatile uint32_t* abort_flag, uint32_t* err_word, uint32_t code) {
  if (try_wait_cluster(bar, parity)) return;
  uint32_t spins = 0;
  long long t0 = 0;
  while (!try_wait_cluster(bar, parity)) {
    if ((++spins & 0xfff) == 0) {
      if (__any_sync(0xffffffffu, *abort_flag != 0)) return;
      const long long now = clock64();
      if (t0 == 0) t0 = now;
      if (__any_sync(0xffffffffu, now - t0 > ptx::kWaitLimitCycles)) {
        *abort_flag = code;
        if (err_word) atomicCAS(err_word, 0u, code | (blockIdx.x << 8));
        return;
      }
    }
  }
}
// TMA load into this CTA's shared memory whose bytes count on the leader's barrier at the same place.  (They may come before the
// leader announces them: the count of a phase goes through negative values, and its one arrival is the announcement.)
__device__ __forceinline__ uint32_t leader_address(const void* p) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(a) : "r"(ptx::smem_u32(p)));
  return a;
}
__device__ __forceinline__ void load_for_leader(uint32_t dst, const CUtensorMap* map, uint32_t leader_bar, int32_t c0, int32_t c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
      "l"(map), "r"(leader_bar), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void mma_i8_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t"
      "}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrives on the barrier at this place in both CTAs once the MMAs issued so far are complete
__device__ __forceinline__ void commit_pair(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
               "h"((uint16_t)3)
               : "memory");
}

// Sixteen tokens of one output column; PAIRS: with the neighbouring lane, which has the neighbouring column
template <typename OT>
__device__ __forceinline__ void store_tokens(OT* o, int64_t ld, const float* v, int count, bool ok, bool pairs) {
  if constexpr (sizeof(OT) == 2) {
    if (pairs) {
      const bool odd = threadIdx.x & 1;
      OT* p = o - (odd ? 1 : 0) + (odd ? ld : 0);
#pragma unroll
      for (int t = 0; t < 16; t += 2, p += 2 * ld) {
        const float got = __shfl_xor_sync(0xffffffffu, odd ? v[t] : v[t + 1], 1);
        OT two[2] = {from_f32<OT>(odd ? got : v[t]), from_f32<OT>(odd ? v[t + 1] : got)};
        if (ok && t + (odd ? 1 : 0) < count) *reinterpret_cast<uint32_t*>(p) = *reinterpret_cast<const uint32_t*>(two);
      }
      return;
    }
  }
#pragma unroll
  for (int t = 0; t < 16; ++t, o += ld)
    if (ok && t < count) *o = from_f32<OT>(v[t]);
}

template <int NL>
__global__ void __launch_bounds__(kThreads, 1)
    pair_gemm_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_b, const Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* stage_base = smem;
  float* s_tok = reinterpret_cast<float*>(smem + (size_t)kStages * kStageBytes);  // [2][kCols] factors of a tile's tokens
  uint32_t* s_sum = reinterpret_cast<uint32_t*>(s_tok + 2 * kCols);               // [2][kCols] their sums
  uint64_t* bars = reinterpret_cast<uint64_t*>(s_sum + 2 * kCols);
  uint64_t* full = bars;                          // [kStages] leader: TMA bytes of both CTAs
  uint64_t* empty = full + kStages;               // [kStages] the leader's commit
  uint64_t* acc_full = empty + kStages;           // [2]       the leader's commit
  uint64_t* acc_empty = acc_full + 2;             // [2]       leader: sixteen drain warps
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = ptx::warp_index(), lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      ptx::mbar_init(&full[s], 1);
      ptx::mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      ptx::mbar_init(&acc_full[a], 1);
      ptx::mbar_init(&acc_empty[a], 2 * kDrain / 32);
    }
    *abort_flag = 0;
    ptx::fence_mbar_init();
    ptx::prefetch_tensormap(&map_w);
    ptx::prefetch_tensormap(&map_b);
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(ptx::smem_u32(tmem_slot)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  ptx::tcgen05_fence_before();
  __syncthreads();
  cluster_sync();  // the barriers of both CTAs are there
  ptx::tcgen05_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  FragIter it(p);

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      const uint32_t stage_a = ptx::smem_u32(stage_base), leader_full = leader_address(full);
      auto row_of = [&](int item) { return (item / p.ytiles * 2 + (int)rank) * kRows; };
      auto col_of = [&](int item) { return item % p.ytiles * (Tile<NL>::kTokens * NL) + (int)rank * (kCols / 2); };
      // the weights of the first stages come under the kernel that makes the other operand
      uint32_t ahead = 0;
      if (p.w_dep) asm volatile("griddepcontrol.wait;" ::: "memory");
#pragma unroll 1
      for (int half = 0; half < 2; ++half) {
        if (half) asm volatile("griddepcontrol.wait;" ::: "memory");
        FragIter f(p);
        ahead = 0;
        while (ahead < (uint32_t)kStages && f.next()) {
#pragma unroll 1
          for (int kb = f.k0(); kb < f.k1() && ahead < (uint32_t)kStages; ++kb, ++ahead) {
            const uint32_t dst = stage_a + ahead * kStageBytes;
            if (half) {
              load_for_leader(dst + kHalf, &map_b, leader_full + ahead * 8, kb * kBK, col_of(f.item));
            } else {
              if (rank == 0) ptx::mbar_expect_tx(&full[ahead], 2 * kStageBytes);
              load_for_leader(dst, &map_w, leader_full + ahead * 8, kb * kBK, row_of(f.item));
            }
          }
        }
      }
      uint32_t s = 0, ph = 0, total = ahead;
      int skip = (int)ahead;  // stages that are on their way
      while (it.next()) {
        const int row = row_of(it.item), col = col_of(it.item), k1 = it.k1();
        int kb = it.k0();
        const int jump = min(skip, k1 - kb);
        skip -= jump;
        for (kb += jump; kb < k1; ++kb, ++total) {
          ptx::mbar_wait(&empty[s], ph, abort_flag, p.err_word, ptx::kErrWaitEmpty);
          const uint32_t dst = stage_a + s * kStageBytes, bar = leader_full + s * 8;
          if (rank == 0) ptx::mbar_expect_tx(&full[s], 2 * kStageBytes);
          load_for_leader(dst, &map_w, bar, kb * kBK, row);
          load_for_leader(dst + kHalf, &map_b, bar, kb * kBK, col);
          if (++s == kStages) { s = 0; ph ^= 1; }
        }
      }
      // the last commits arrive before this CTA may end
      for (uint32_t i = total - ahead; i < total; ++i)
        ptx::mbar_wait(&empty[i % kStages], (i / kStages) & 1, abort_flag, p.err_word, ptx::kErrWaitEmpty);
    }
    __syncwarp();
  } else if (warp == 1 && rank == 0) {
    // ---------------- MMA issuer: the whole warp walks the loop, one elected thread issues ----------------
    constexpr uint32_t idesc = ptx::make_idesc(/*s32*/ 2, /*s8*/ 1, /*s8*/ 1, 2 * kRows, kCols);
    const uint32_t tb = __reduce_or_sync(0xffffffffu, tmem_base);
    const uint32_t desc_hi = (uint32_t)(ptx::make_sw128_kmajor_desc(0) >> 32);
    const uint32_t lo0 = (uint32_t)ptx::make_sw128_kmajor_desc(ptx::smem_u32(stage_base));
    const uint32_t full_a = ptx::smem_u32(full), empty_a = ptx::smem_u32(empty), acc_full_a = ptx::smem_u32(acc_full),
                   acc_empty_a = ptx::smem_u32(acc_empty);
    uint32_t s = 0, ph = 0;
    for (int t = 0; it.next(); ++t) {
      const uint32_t ab = t & 1;
      wait_cluster(acc_empty_a + ab * 8, ((t >> 1) & 1) ^ 1, abort_flag, p.err_word, ptx::kErrWaitTmemEmpty);
      const uint32_t d = tb + ab * kCols;
      const int k0 = it.k0(), k1 = it.k1();
      for (int kb = k0; kb < k1; ++kb) {
        wait_cluster(full_a + s * 8, ph, abort_flag, p.err_word, ptx::kErrWaitFull);
        ptx::tcgen05_fence_after();
        const uint32_t a_lo = lo0 + s * (kStageBytes >> 4), b_lo = a_lo + (kHalf >> 4);
        if (ptx::elect_one()) {
#pragma unroll
          for (int k = 0; k < kBK / 32; ++k)
            mma_i8_pair(d, ((uint64_t)desc_hi << 32) | (uint64_t)(a_lo + k * 2), ((uint64_t)desc_hi << 32) | (uint64_t)(b_lo + k * 2), idesc,
                        (uint32_t)((kb - k0) | k));
          commit_pair(empty_a + s * 8);
          if (kb + 1 == k1) commit_pair(acc_full_a + ab * 8);
        }
        __syncwarp();
        if (++s == kStages) { s = 0; ph ^= 1; }
      }
    }
  } else if (warp >= 4) {
    // ---------------- epilogue ----------------
    constexpr int T = Tile<NL>::kTokens, G = Tile<NL>::kGroup;
    const int quad = warp & 3, grp = (warp - 4) >> 2;
    const int dt = (int)threadIdx.x - 128;
    asm volatile("griddepcontrol.wait;" ::: "memory");  // factors, sums, scales and `out` belong to earlier kernels until here
    __shared__ int s_npart;
    const int place = it.place();
    for (int t = 0; it.next(); ++t) {
      const int item = it.item;
      const bool first = it.u0 == 0, last = it.u1 == p.ut;
      const uint32_t ab = t & 1;
      const int64_t n = (int64_t)(item / p.ytiles * 2 + (int)rank) * kRows + quad * 32 + lane;
      const bool n_ok = n < p.N;
      const int m0 = item % p.ytiles * T;
      float* tok = s_tok + ab * kCols;
      uint32_t* sum = s_sum + ab * kCols;
      if (dt < T) {
        const bool ok = m0 + dt < p.M;
        tok[dt] = ok ? ld_ordered(p.tok + m0 + dt) : 0.f;
        if (p.zp) sum[dt] = ok ? ld_ordered(static_cast<const uint32_t*>(p.sums) + m0 + dt) : 0u;
      }
      const float sc = n_ok ? scale_value(load_scale_bits(p.scale, n, p.s_dt), p.s_dt) : 0.f;
      const float z = n_ok && p.zp ? scale_value(load_scale_bits(p.zp, n, p.s_dt), p.s_dt) : 0.f;
      auto drain_bar = [&]() { asm volatile("bar.sync 1, %0;" ::"n"(kDrain) : "memory"); };
      int np = 0;
      if (NL > 1 && first && !last) {
        if (dt == 0) {
          int cnt = 0;
          for (int c = place + 1; c < p.g2; ++c) {
            if (it.share(c) >= (item - p.items1 + 1) * p.ut) break;
            ++cnt;
          }
          s_npart = cnt;
        }
        drain_bar();
        np = s_npart;
        // the sums of the pairs that continue the item, for this CTA's rows
        for (int j = dt; j < np; j += kDrain)
          ptx::partial_wait(p.flags + 2 * (place + 1 + j) + rank, p.wait_cycles, abort_flag, p.err_word, kErrPartialPair);
      }
      drain_bar();  // (and the tile before the last is through)
      ptx::mbar_wait_warp(&acc_full[ab], (t >> 1) & 1, abort_flag, p.err_word, ptx::kErrWaitTmemFull);
      ptx::tcgen05_fence_after();
      const bool lost = *abort_flag != 0;  // a wait ran out: NaN, not what is there
      const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + ab * kCols;
#pragma unroll 1
      for (int c = grp * G; c < min((grp + 1) * G, T); c += 16) {
        const int t0 = min(c, T - 16);
        uint32_t r[16 * NL];
#pragma unroll
        for (int j = 0; j < NL; ++j) ptx::tmem_ld_32x32b_x16(taddr + t0 * NL + 16 * j, r + 16 * j);
        ptx::tmem_ld_wait();
        float v[16];
        // the row's share of partial tile q, four tokens side by side
        auto part = [&](int q) {
          return reinterpret_cast<float4*>(p.partial) + ((size_t)(2 * q + rank) * (T / 4) + t0 / 4) * kRows + quad * 32 + lane;
        };
        if constexpr (NL > 1) {
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            v[i] = fmaf(__int2float_rn((int)r[NL * i + 1]), 256.f, __int2float_rn((int)r[NL * i]));
            if constexpr (NL == 3) v[i] = fmaf(__int2float_rn((int)r[NL * i + 2]), 65536.f, v[i]);
          }
          if (!first) {
#pragma unroll
            for (int i = 0; i < 16; i += 4) {
              const float nan = __uint_as_float(0x7fc00000u);
              __stcg(part(place) + i / 4 * kRows, lost ? make_float4(nan, nan, nan, nan) : make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]));
            }
            continue;
          }
          for (int j = 0; j < np; ++j) {
            float4 w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) w[i] = __ldcg(part(place + 1 + j) + i * kRows);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              v[4 * i] += w[i].x;
              v[4 * i + 1] += w[i].y;
              v[4 * i + 2] += w[i].z;
              v[4 * i + 3] += w[i].w;
            }
          }
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          if constexpr (NL == 1) {
            v[i] = w8a8_dequant((int32_t)r[i], sc, p.zp ? &z : nullptr, (int32_t)sum[t0 + i], tok[t0 + i]);
          } else {
            float f = v[i] * sc;
            if (p.zp) f = fmaf(-p.zp_mul * z, __uint_as_float(sum[t0 + i]), f);
            v[i] = f * tok[t0 + i];
          }
          if (lost) v[i] = __uint_as_float(0x7fc00000u);
        }
        const int count = p.M - m0 - t0;
        const int64_t at = (int64_t)(m0 + t0) * p.ld + n;
        if (p.out_dt == QMM_F32) store_tokens(static_cast<float*>(p.out) + at, p.ld, v, count, n_ok, false);
        else if (p.out_dt == QMM_BF16) store_tokens(static_cast<__nv_bfloat16*>(p.out) + at, p.ld, v, count, n_ok, p.out_pairs != 0);
        else store_tokens(static_cast<__half*>(p.out) + at, p.ld, v, count, n_ok, p.out_pairs != 0);
      }
      ptx::tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) arrive_leader(&acc_empty[ab]);
      if (NL > 1 && !first) {
        drain_bar();  // orders every drain thread's stores before thread 0's fence, which is cumulative
        if (dt == 0) ptx::partial_publish(p.flags + 2 * place + rank);
      }
    }
  }

  ptx::tcgen05_fence_before();
  __syncthreads();
  cluster_sync();  // nothing of the pair is under way any more
  if (warp == 2) {
    ptx::tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem_base) : "memory");
  }
  cluster_sync();
}

template <int NL>
int launch_with(const CUtensorMap& map_w, const CUtensorMap& map_b, const Params& p, int pairs, cudaStream_t st) {
  auto kern = pair_gemm_kernel<NL>;
  static bool attr_set[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
    if (e != cudaSuccess) return fail(QMM_ERR_LAUNCH, "cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    if (dev >= 0 && dev < 64) attr_set[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(2 * pairs));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = 2;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, map_w, map_b, p);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(QMM_ERR_LAUNCH, "pair_gemm_kernel launch: %s", cudaGetErrorString(e));
  }
  return check_launch("pair_gemm_kernel");
}

}  // namespace

int pair_gemm_tokens(int nl) { return nl == 3 ? Tile<3>::kTokens : kCols / nl; }

// Weight-only, against limb_gemm.cu's 128 x 64 (42 with three limbs) tiles on single CTAs.  A round of tiles takes about as long there as
// here, a little less, with half of the work in it.  So here where that saves a round: int8 [11008,5120] at 256 tokens, 86 items in two
// rounds against 344 in three, 32 us, 36 there; at 129, 258 in two there as well, 31 and 27; [5120,5120] at 256 (40 items, 160)
// 21 and 26, at 129 (40, 120) 19.5 and 17.7.  At equal rounds from 12288 inputs on, which are split over K here ([2560,28672] at 256 tokens
// 46 and 65), and few items from 8192 ([2560,9472] at 128 22.6 and 25.2); not between 28 items and a round, which split badly ([5839,12288]
// at 129, 46 items, 37 and 32, with three limbs at 93 40 and 34; [4096,14336] at 150, 32 items, 33.5 and 30.6).
bool pair_gemm_preferred(int nl, int64_t M, int64_t N, int64_t K) {
  const int64_t items = ceil_div(N, 2 * kRows) * ceil_div(M, pair_gemm_tokens(nl));
  const int64_t there = ceil_div(N, kRows) * ceil_div(M, nl == 3 ? 42 : 64);  // limb_gemm.cu's items
  const int sms = sm_count();
  if (M <= (nl == 3 ? 42 : 64) || items < 16) return false;
  return ceil_div(items, sms / 2) < ceil_div(there, sms) || (K >= 12288 && (items <= 28 || items > sms / 2)) || (K >= 8192 && items < 24);
}

// W8A8, against w8a8_gemm.cu's 128 x 256 tiles on single CTAs: by rounds of tiles, at 0.31 us a stage here and 0.5 there, and a
// launch that takes 6 us longer ([4096,4096] at 64 tokens 18.3 us against 21.5, at 2048 34.1 and 40.6, at 4096 59 and 73;
// [28672,8192] at 64 tokens, two rounds for one, 53 against 49).  Outputs whose rows TMA cannot store (an odd number of them, or
// fp32) are written by threads there: always here ([300,512] at 128 tokens 9.8 us against 45).
bool pair_gemm_preferred_w8a8(int64_t M, int64_t N, int64_t K, int out_dt) {
  if (out_dt != QMM_F32 && N % 8 != 0) return true;
  const int64_t items = ceil_div(N, 2 * kRows) * ceil_div(M, kCols), other = ceil_div(M, 128) * ceil_div(N, 256);
  const double kb = (double)ceil_div(K, kBK);
  const int sms = sm_count();
  return items >= 8 && ceil_div(items, sms / 2) * kb * 0.31 + 6.0 < ceil_div(other, sms) * kb * 0.5;
}

int launch_pair_gemm(int nl, const int8_t* w, const int8_t* b, const Scales& scales, const float* tok, const void* sums, float zp_mul,
                     void* out, int out_dt, int64_t M, int64_t N, int64_t K, int64_t ld, int w_dep, float* partial, uint32_t* flags, cudaStream_t st) {
  CUtensorMap map_w, map_b;
  int rc = encode_tmap_2d(&map_w, w, 1, false, (uint64_t)N, (uint64_t)K, kRows, kBK);
  if (rc != QMM_OK) return rc;
  rc = encode_tmap_2d(&map_b, b, 1, false, (uint64_t)(nl * M), (uint64_t)K, kCols / 2, kBK);
  if (rc != QMM_OK) return rc;
  Params p = {};
  p.scale = scales.scale;
  p.zp = scales.zp;
  p.s_dt = scales.dt;
  p.tok = tok;
  p.sums = sums;
  p.zp_mul = zp_mul;
  p.out = out;
  p.out_dt = out_dt;
  p.out_pairs = out_dt != QMM_F32 && ld % 2 == 0 && N % 2 == 0 && aligned(out, 4);
  p.M = (int)M;
  p.N = N;
  p.ld = ld;
  p.k_blocks = (int)ceil_div(K, kBK);
  p.ytiles = (int)ceil_div(M, pair_gemm_tokens(nl));
  p.w_dep = w_dep;
  p.err_word = device_error_word();
  p.wait_cycles = peer_wait_cycles();
  p.partial = partial;
  p.flags = flags;
  const int items = (int)ceil_div(N, 2 * kRows) * p.ytiles, most = std::min(sm_count() / 2, kPairMostPairs);
  int pairs = std::min(items, most);
  p.items1 = items;
  p.ut = (int)ceil_div(p.k_blocks, kUnit);
  p.g2 = 1;
  const int left = items % most;
  if (partial && left != 0) {
    // Splitting the left-over items over s pairs each: item / s plus an exchange that grows with s (one partial tile per pair,
    // written, and read by the item's first pair).  A stage takes about 0.3 us, the exchange 8 ([4096,14336] at 128 tokens 41 us
    // in whole items, 31 over 2.3 pairs each; [28672,8192] at 200, two items left over, 88 and 83; [14336,4096] at 333 39 and 43).
    const double item_us = p.k_blocks * 0.3, partial_us = (double)pair_gemm_tokens(nl) / 128.0;
    double s = std::sqrt(item_us / partial_us);
    s = std::min(s, std::min((double)most / left, (double)p.ut));
    if (s >= 1.2 && item_us / s + 6.0 + partial_us * s < 0.85 * item_us) {
      p.items1 = items - left;
      p.units = left * p.ut;
      p.g2 = std::min(most, std::max(left, (int)(left * s)));
      pairs = std::max(std::min(p.items1, most), p.g2);
    }
  }
  return nl == 1 ? launch_with<1>(map_w, map_b, p, pairs, st) : nl == 2 ? launch_with<2>(map_w, map_b, p, pairs, st)
                                                                         : launch_with<3>(map_w, map_b, p, pairs, st);
}

}  // namespace qmm
