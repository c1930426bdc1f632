// Thin inline-PTX wrappers for the sm_100a features the tensor-core kernels use:
// mbarrier, TMA (cp.async.bulk.tensor), tcgen05.mma / TMEM, plus the shared-memory and
// instruction descriptors tcgen05.mma consumes.
//
// Every wait is bounded: a wait that does not complete within kWaitLimitCycles records a code in the
// library's device error word and in a CTA-local abort flag; once that flag is set all later
// waits return at once, so a kernel with a broken pipeline drains and exits instead of hanging.  Whoever stores results
// looks at the flag first and stores NaN when it is set.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace qmm {
namespace ptx {

constexpr long long kWaitLimitCycles = 4000000000ll;  // about 2 s of SM clock per wait

enum ErrCode : uint32_t {
  kErrNone = 0,
  kErrWaitFull = 1,       // consumer never saw a TMA stage land
  kErrWaitEmpty = 2,      // producer never got a stage back
  kErrWaitTmemFull = 3,   // epilogue never saw the accumulator committed
  kErrWaitTmemEmpty = 4,  // MMA issuer never got the accumulator back
  kErrWaitConv = 5,       // MMA issuer never saw a dequantised stage
  kErrWaitRaw = 6,        // dequant warps never saw the raw stage
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t"
      "}"
      : "=r"(pred));
  return pred != 0;
}

// ---- mbarrier -----------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t"
      "}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Non-blocking look at a phase: for a barrier that is needed a little later, so that the result's latency (about 45 cycles
// until a branch on it resolves, 85 behind issued MMAs) passes under other work.
__device__ __forceinline__ bool mbar_test_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t"
      "}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait.  `abort_flag` is a CTA-shared word; `err_word` the library's global error word.
// The first try stands alone: a phase that is complete costs 43 cycles this way, 65 to 170 when the loop below is entered
// for it.  The SM cycle counter is looked at only once every 4096 polls (a %globaltimer read per wait costs about a
// microsecond and would dominate short waits).
template <int SLEEP_NS = 0>
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity,
                                          volatile uint32_t* abort_flag, uint32_t* err_word,
                                          uint32_t code) {
  if (mbar_try_wait(bar, parity)) return true;
  uint32_t spins = 0;
  long long t0 = 0;
  while (!mbar_try_wait(bar, parity)) {
    if (SLEEP_NS > 0) __nanosleep(SLEEP_NS);  // back off: pollers share the barrier unit with the MMA issuer
    if ((++spins & 0xfff) == 0) {
      if (*abort_flag) return false;
      const long long now = clock64();
      if (t0 == 0) {
        t0 = now;
      } else if (now - t0 > kWaitLimitCycles) {
        *abort_flag = code;
        if (err_word) atomicCAS(err_word, 0u, code | (blockIdx.x << 8));
        return false;
      }
    }
  }
  return true;
}

// Whole-warp wait: after one look by all lanes, lane 0 polls and the rest of the warp parks at the warp barrier.  Keeps 31
// of 32 lanes from hammering the same mbarrier word while the MMA issuer needs that unit.
template <int SLEEP_NS = 0>
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity,
                                               volatile uint32_t* abort_flag, uint32_t* err_word,
                                               uint32_t code) {
  if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
  bool ok = true;
  if ((threadIdx.x & 31) == 0) ok = mbar_wait<SLEEP_NS>(bar, parity, abort_flag, err_word, code);
  __syncwarp();
  return ok;
}

// The same by address, for loops in which every instruction counts (a lone warp issues a dependent one every 4 to 6 cycles,
// and a generic pointer costs several to turn into an address).  All lanes look; a wait costs about 57 cycles when the phase
// is complete.
__device__ __forceinline__ bool bar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t"
      "}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return __all_sync(0xffffffffu, ok != 0);
}
__device__ __forceinline__ void bar_wait(uint32_t bar, uint32_t parity, volatile uint32_t* abort_flag, uint32_t* err_word, uint32_t code) {
  if (__builtin_expect(bar_try_wait(bar, parity), 1)) return;
  uint32_t spins = 0;
  long long t0 = 0;
  while (!bar_try_wait(bar, parity)) {
    if ((++spins & 0xfff) == 0) {
      if (__any_sync(0xffffffffu, *abort_flag != 0)) return;
      const long long now = clock64();
      if (t0 == 0) t0 = now;
      if (__any_sync(0xffffffffu, now - t0 > kWaitLimitCycles)) {
        *abort_flag = code;
        if (err_word) atomicCAS(err_word, 0u, code | (blockIdx.x << 8));
        return;
      }
    }
  }
}
__device__ __forceinline__ void mbar_arrive_a(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// ---- partial tiles between the CTAs of a launch ------------------------------------------------
// A CTA that works on a later K range of a tile leaves its sums in global scratch for the tile's first CTA.  The flag word
// beside them: 0 idle, 1 written, 2 given up by the reader; 0 again after every launch, also after one that gave up.
// Both are called by one thread, the writer's behind a barrier that its CTA's stores precede.
__device__ __forceinline__ void partial_publish(uint32_t* flag) {
  __threadfence();
  if (atomicCAS(flag, 0u, 1u) == 2u) atomicExch(flag, 0u);  // nobody waits for it any more
}
__device__ __forceinline__ bool partial_wait(uint32_t* flag, long long limit_cycles, volatile uint32_t* abort_flag, uint32_t* err_word,
                                             uint32_t code) {
  const long long t0 = clock64();
  uint32_t spins = 0, v;
  while (true) {
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
    if (v == 1u) break;
    if ((++spins & 0xff) == 0 && (*abort_flag || clock64() - t0 > limit_cycles)) {
      if (atomicCAS(flag, 0u, 2u) == 1u) {  // there after all
        __threadfence();
        break;
      }
      *abort_flag = code;
      if (err_word) atomicCAS(err_word, 0u, code | (blockIdx.x << 8));
      return false;
    }
  }
  atomicExch(flag, 0u);
  return true;
}

// ---- proxies / fences ---------------------------------------------------------------------
// Makes generic-proxy writes to shared memory visible to the async proxy (TMA, tcgen05.mma).
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void tcgen05_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}

__device__ __forceinline__ void tcgen05_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// ---- TMA ----------------------------------------------------------------------------------
__device__ __forceinline__ void prefetch_tensormap(const CUtensorMap* m) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(m) : "memory");
}

// 2-D tile load, global -> this CTA's shared memory, completion counted on `bar`.
// c0 is the innermost (contiguous) coordinate and must keep c0 * elem_size 16-byte aligned.
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const CUtensorMap* map, uint64_t* bar,
                                            int32_t c0, int32_t c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, "
      "%4}], [%2];" ::"r"(smem_u32(smem_dst)),
      "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1)
      : "memory");
}

// ---- TMEM ---------------------------------------------------------------------------------
// Whole-warp, .sync.aligned: call from one full warp.  ncols: power of two, 32..512.
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_result, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_u32(smem_result)),
               "r"(ncols)
               : "memory");
}

__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}

// ---- descriptors --------------------------------------------------------------------------
// Shared-memory matrix descriptor for a K-major operand tile stored with the 128-byte swizzle:
// rows are 128 bytes apart, 8 rows form one 1024-byte swizzle atom (stride-byte-offset 1024).
// Field layout (bits): [0,14) start address >> 4, [16,30) leading byte offset >> 4,
// [32,46) stride byte offset >> 4, [46,48) version = 1, [61,64) layout = 2 (128B swizzle).
__device__ __forceinline__ uint64_t make_sw128_kmajor_desc(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);
  d |= (uint64_t)1 << 16;              // leading byte offset: unused for swizzled K-major
  d |= (uint64_t)(1024 >> 4) << 32;    // stride byte offset: next group of 8 rows
  d |= (uint64_t)1 << 46;              // descriptor version for sm_100
  d |= (uint64_t)2 << 61;              // SWIZZLE_128B
  return d;
}

// Instruction descriptor (32 bits): [4,6) accumulator format (0 f16, 1 f32, 2 s32),
// [7,10) A format, [10,13) B format (kind::f16: 0 f16, 1 bf16; kind::i8: 0 u8, 1 s8),
// bit 15 / 16: A / B major (0 = K-major), [17,23) N >> 3, [24,29) M >> 4.
__host__ __device__ constexpr uint32_t make_idesc(uint32_t c_fmt, uint32_t a_fmt, uint32_t b_fmt,
                                                  uint32_t M, uint32_t N) {
  return (c_fmt << 4) | (a_fmt << 7) | (b_fmt << 10) | ((N >> 3) << 17) | ((M >> 4) << 24);
}

// ---- MMA ----------------------------------------------------------------------------------
// D[tmem] (+)= A[smem] * B[smem]; issue from ONE thread.
__device__ __forceinline__ void mma_i8_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc,
                                          uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t"
      "}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ void mma_f16_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc,
                                           uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t"
      "}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// How to issue: the warp index that selects the issuing warp must come from warp_index() and ONE elected thread must issue
// from inside a branch, so that the compiler keeps descriptors in uniform registers.  Predicating the instruction on a
// lane instead costs 62 to 77 cycles of instructions per MMA whatever its size; this form issues one in 11 and leaves the
// tensor pipe as the limit (measured, kind::f16 with A in tensor memory: 11 / 32 / 64 / 96 cycles for N = 16 / 64 / 128 /
// 192; kind::i8 with A in shared memory: 40 / 48 / 64 / 128 for N = 16 / 64 / 128 / 256).
__device__ __forceinline__ int warp_index() { return __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0); }

// Arrives on `bar` once every tcgen05.mma issued so far by this thread has completed.
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   smem_u32(bar))
               : "memory");
}

__device__ __forceinline__ void mma_commit_a(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// ---- TMEM -> registers --------------------------------------------------------------------
// Each thread of the warp reads 32 consecutive 32-bit columns of its own TMEM lane
// (lane = 32 * (warp_id % 4) + lane_id; the lane quadrant goes into bits [16,32) of taddr).
__device__ __forceinline__ void tmem_ld_32x32b_x32(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
        "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}

__device__ __forceinline__ void tmem_ld_32x32b_x16(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}

__device__ __forceinline__ void tmem_ld_wait() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// After a tmem_ld_wait that follows OTHER instructions issued since the load: tells the compiler that the 16
// registers of that load change here, so that it neither reads nor moves them between the load and the wait.
__device__ __forceinline__ void tmem_ld_landed16(uint32_t* r) {
  asm volatile(""
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]),
                 "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
               :
               : "memory");
}

__device__ __forceinline__ void tmem_ld_landed8(uint32_t* r) {
  asm volatile("" : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]) : : "memory");
}

// ---- registers -> TMEM --------------------------------------------------------------------
// Each thread of the warp writes 32 consecutive 32-bit columns of its own TMEM lane.
__device__ __forceinline__ void tmem_st_32x32b_x32(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}

// Each thread of the warp writes 8 consecutive 32-bit columns of its own TMEM lane.
__device__ __forceinline__ void tmem_st_32x32b_x8(uint32_t taddr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]),
               "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}

__device__ __forceinline__ void tmem_st_wait() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// D[tmem] (+)= A[tmem] * B[smem]: the A operand is read from tensor memory (row m = lane m, two 16-bit
// k values per 32-bit column, 8 columns per K=16 step).  Call from ONE thread.
__device__ __forceinline__ void mma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                           uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
      "}" ::"r"(d_tmem),
      "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// The same with int8 operands: four k values per 32-bit column, 8 columns per K=32 step.
__device__ __forceinline__ void mma_i8_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                           uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t"
      "}" ::"r"(d_tmem),
      "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

}  // namespace ptx

// ---- host: tensor maps --------------------------------------------------------------------
// cuTensorMapEncodeTiled is fetched through the runtime so the library does not link libcuda.
// Encodes a 2-D row-major tensor [rows][cols] of `elem_bytes` elements with a box of
// [box_rows][box_cols] and the 128-byte swizzle; out-of-range reads return zero.
int encode_tmap_2d(CUtensorMap* map, const void* base, int elem_bytes, bool is_bf16or_f16,
                   uint64_t rows, uint64_t cols, uint32_t box_rows, uint32_t box_cols);

}  // namespace qmm
