// Thin inline-PTX layer for sm_100a: mbarrier, TMA (no cluster broadcast forms), tcgen05
// (TMEM allocation, UMMA issue/commit, TMEM loads, smem->TMEM copies) and descriptor builders.
// Every wait in this file is bounded: a wait that runs out records a code and returns false so
// the kernel can unwind (await what it has in flight, free TMEM) instead of spinning forever.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>
#include <cuda_bf16.h>

namespace dq {

// ---- error codes written to the status word (first error wins) -------------------------------
enum : int {
  ERR_NONE = 0,
  ERR_WAIT_FULL = 1,      // consumer waited for a filled smem stage
  ERR_WAIT_EMPTY = 2,     // producer waited for a free smem stage
  ERR_WAIT_ACC_FULL = 3,  // epilogue waited for an accumulator
  ERR_WAIT_ACC_EMPTY = 4, // MMA issuer waited for a drained accumulator
  ERR_WAIT_DRAIN = 5,     // teardown waited for copies in flight
  ERR_WAIT_SF = 6,        // scale factors: mover waited for the tiles, or the issuer for the movers
};

// ~1.5 s at the boost clock; clock64() ticks at the SM clock.
constexpr long long kWaitLimitCycles = 3000000000LL;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// ---- mbarrier ----------------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// One poll.  `suspend_ns` is the hardware suspend-time hint: the thread sleeps inside the instruction
// (no issue slots used) until the phase completes or roughly that long has passed.
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity, uint32_t suspend_ns = 0) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity), "r"(suspend_ns)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// A poll of a sleeping wait: suspended in hardware, or, under a short limit (see AB_POLL), a plain test, since a suspended
// poll may outlast its hint by many microseconds.
__device__ __forceinline__ bool mbar_poll(uint32_t bar, uint32_t parity, int suspend_ns) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p, l;\n\t"
      "setp.ge.s32 l, %3, 20000;\n\t"
      "@l mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "@!l mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity), "r"(suspend_ns)
      : "memory");
  return ok != 0;
}
// Two phase tests issued back to back, so that their latencies overlap (a test costs about a hundred cycles even when the
// phase has long completed).  Bit i of the result: barrier i's phase is complete.
__device__ __forceinline__ uint32_t mbar_test2(uint32_t b0, uint32_t p0, uint32_t b1, uint32_t p1) {
  uint32_t m;
  asm volatile(
      "{\n\t.reg .pred q0, q1;\n\t.reg .u32 t0, t1;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 q0, [%1], %2;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 q1, [%3], %4;\n\t"
      "selp.u32 t0, 1, 0, q0;\n\t"
      "selp.u32 t1, 2, 0, q1;\n\t"
      "or.b32 %0, t0, t1;\n\t}"
      : "=r"(m)
      : "r"(b0), "r"(p0), "r"(b1), "r"(p1)
      : "memory");
  return m;
}
// Shared words of a CTA's failure handling, behind its barriers.  Once any role gave up, all later waits of the CTA -- of
// both CTAs of a pair, whose flags are raised together -- return at once; every role stops, and the CTA tears down what the
// roles left in flight (see drain_ring).
enum : int {
  AB_FLAG = 0,      // a role gave up
  AB_LIMIT = 1,     // the launch's wait limit in units of 1024 cycles
  AB_POLL = 2,      // how long one poll may sleep (ns): 20 us, less under a short limit
  AB_PEER = 3,      // shared::cluster address of the peer's AB_FLAG (0 = no peer)
  AB_ISSUED = 4,    // stages the producer has issued copies for, written when it stops
  AB_ISSUED2 = 5,   // the same of a second producer
  AB_UMMA = 6,      // stages and accumulators the issuer has committed UMMAs for
  AB_ACC = 7,
  AB_MAX = 8,       // pairs: stages any role of the CTA has got to
  AB_WARP = 9,      // per warp of a role that arrives on a pair's barriers: stages it has arrived for
  AB_WORDS = 17,
};
__device__ __forceinline__ void abort_init(volatile int* w, int limit_k, uint32_t peer_flag = 0) {
  w[AB_FLAG] = 0;
  w[AB_LIMIT] = limit_k > 0 ? limit_k : (int)(kWaitLimitCycles >> 10);
  w[AB_POLL] = limit_k > 0 && limit_k < 80 ? 250 * limit_k : 20000;
  w[AB_PEER] = (int)peer_flag;
  w[AB_ISSUED] = w[AB_ISSUED2] = w[AB_UMMA] = w[AB_ACC] = w[AB_MAX] = 0;
}
// System scope: the word may be host memory, which the host clears while kernels of other streams still run.
__device__ __forceinline__ void report_status(int* status, int code) {
  if (status) atomicCAS_system(status, 0, code);
}
__device__ __forceinline__ void abort_raise(volatile int* abort_flag, int* status, int code) {
  abort_flag[AB_FLAG] = 1;
  if (const uint32_t peer = (uint32_t)abort_flag[AB_PEER])
    asm volatile("st.relaxed.cluster.shared::cluster.u32 [%0], %1;" ::"r"(peer), "r"(1u) : "memory");
  report_status(status, code);
}
__device__ __forceinline__ bool abort_late(volatile int* abort_flag, long long t0) {
  return clock64() - t0 > (long long)abort_flag[AB_LIMIT] << 10;
}
// The code after the roles starts from scratch: values it shared with what comes before would have to be kept through the
// roles (in the epilogue of a 256-wide tile, as spills).
template <typename T> __device__ __forceinline__ T anew(T v) {
  if constexpr (sizeof(T) == 8) asm volatile("" : "+l"(v));
  else asm volatile("" : "+r"(v));
  return v;
}
__device__ __forceinline__ uint32_t tid_anew() {
  uint32_t t;
  asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
  return t;
}

// Bounded wait.  Waiters sleep in hardware (up to 20 us per poll) instead of spinning, so they do not
// compete with the working warps for issue slots; between polls the shared abort flag and the clock
// are checked.  For one thread of a warp; a warp whose lanes all wait uses the forms below.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag,
                                          int* status, int code) {
  if (mbar_test(bar, parity)) return true;
  const long long t0 = clock64();
  while (true) {
    if (mbar_poll(bar, parity, abort_flag[AB_POLL])) return true;
    __nanosleep(128);            // keep pollers off the issue ports of the working warps
    if (abort_flag[AB_FLAG]) return false;
    if (abort_late(abort_flag, t0)) {
      abort_raise(abort_flag, status, code);
      return false;
    }
  }
}

// A short limit leaves no room for polls that do not look at the clock
__device__ __forceinline__ bool hot_polls(volatile int* abort_flag) { return abort_flag[AB_POLL] >= 20000; }
// Bounded wait for roles on the critical path (a stage hand-off every few hundred cycles): polls
// back to back for a while -- a suspended waiter wakes up too late for such short intervals -- and
// only then falls into the sleeping loop of mbar_wait.
__device__ __forceinline__ bool mbar_wait_hot(uint32_t bar, uint32_t parity, volatile int* abort_flag,
                                              int* status, int code) {
  if (mbar_test(bar, parity)) return true;
  if (hot_polls(abort_flag)) {
#pragma unroll 1
    for (int i = 0; i < 4096; ++i)
      if (mbar_try(bar, parity)) return true;
  }
  return mbar_wait(bar, parity, abort_flag, status, code);
}

// The same for whole warps: one verdict for all lanes, by vote.  Lanes that poll for themselves could see a phase complete
// and the flag raised, part each, and the warp would come apart in front of its next aligned instruction.
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* status, int code) {
  if (__all_sync(0xffffffffu, mbar_test(bar, parity))) return true;
  const long long t0 = clock64();
  while (true) {
    if (__all_sync(0xffffffffu, mbar_poll(bar, parity, abort_flag[AB_POLL]))) return true;
    __nanosleep(128);
    const bool raised = abort_flag[AB_FLAG] != 0, late = abort_late(abort_flag, t0);
    if (__any_sync(0xffffffffu, raised || late)) {
      if (late && !raised) abort_raise(abort_flag, status, code);
      return false;
    }
  }
}
// Hot waits of whole warps: polls back to back, every eighth with a look at the abort flag and the clock, all in one short loop.
// They stand in the middle of loops that use every register they have: with mbar_wait_warp's sleeping loop behind a first,
// shorter one of their own they cost spills and instruction fetches.  Linears of a 2240-wide block (batch 1) 124.5 -> 121.2 us, of
// a 1152-wide one 208.5 -> 205.6; in the rotation, which slept before, 4608 x 3072 56.5 -> 55.7.  (Looking at a short limit as
// closely as mbar_wait_warp does, by a load or another branch, loses most of that; the epilogues, which wait longest, do.)
__device__ __forceinline__ bool wait_ends(volatile int* abort_flag, int* status, int code, long long t0) {
  const bool raised = abort_flag[AB_FLAG] != 0, late = abort_late(abort_flag, t0);
  if (!__any_sync(0xffffffffu, raised || late)) return false;
  if (late && !raised) abort_raise(abort_flag, status, code);
  return true;
}
__device__ __forceinline__ bool mbar_wait_hot_warp(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* status, int code) {
  if (__all_sync(0xffffffffu, mbar_test(bar, parity))) return true;
  const long long t0 = clock64();
#pragma unroll 1
  for (uint32_t i = 1;; ++i) {
    if (__all_sync(0xffffffffu, mbar_try(bar, parity))) return true;
    if (i % 8 == 0 && wait_ends(abort_flag, status, code, t0)) return false;
  }
}

// Two phases, tested back to back (the latencies of the tests overlap)
__device__ __forceinline__ bool mbar_wait2_hot_warp(uint32_t b0, uint32_t p0, uint32_t b1, uint32_t p1, volatile int* abort_flag, int* status,
                                                    int code) {
  if (__all_sync(0xffffffffu, mbar_test2(b0, p0, b1, p1) == 3u)) return true;
  const long long t0 = clock64();
#pragma unroll 1
  for (uint32_t i = 1;; ++i) {
    if (__all_sync(0xffffffffu, mbar_test2(b0, p0, b1, p1) == 3u)) return true;
    if (i % 8 == 0 && wait_ends(abort_flag, status, code, t0)) return false;
  }
}

// One lane of a warp whose lanes are all here, the same one every time.  Issuer warps, and the producers of the rotation and the
// FP4 GEMMs, run their loops with all lanes (waits by vote) and let the elected lane issue (in one lane remain the exact-integer
// GEMM's issuer and producers, the activation producer of the other integer GEMM and the FP4 pair GEMM's scale-factor waits): under elect.sync the compiler knows that one thread is active and keeps
// descriptors and addresses in uniform registers.  The same loop run by `lane == 0` alone took 395 cycles per stage of four
// UMMAs of 128 columns (nominal 256), this one 278 on CTA pairs and 304 on single CTAs; with 256 columns both are hidden behind
// the UMMAs.  Rotation of 4096 x 1152 14.1 -> 11.9 us, of 1024 x 2240 14.1 -> 11.6; INT GEMM 4096 x 1152 x 1152 20.7 -> 19.4;
// launches of many 256-wide tiles 0-3 %.
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p) :: "memory");
  return p != 0;
}

// Teardown after a wait ran out, once every role has stopped: wait (bounded) for one phase, and for those of the last `issued`
// uses of a ring -- the copies a producer issued, the UMMAs an issuer committed.  `bar_of` gives a slot's barrier.  A commit
// that arrives in both CTAs of a pair is awaited in both: nothing else holds a CTA until the arrival, which is on its way
// asynchronously, has reached it.
__device__ __forceinline__ void drain_wait(uint32_t bar, uint32_t parity, int* status) {
  const long long t0 = clock64();
  while (!mbar_try(bar, parity, 20000u))
    if (clock64() - t0 > kWaitLimitCycles / 8) {
      report_status(status, ERR_WAIT_DRAIN);
      return;
    }
}
template <typename F>
__device__ __forceinline__ void drain_ring(F bar_of, int slots, int issued, int* status) {
  for (int q = max(0, issued - slots); q < issued; ++q) drain_wait(bar_of(q % slots), (uint32_t)((q / slots) & 1), status);
}

// GELU, tanh form (torch.nn.functional.gelu(approximate="tanh")), applied to a value that was first rounded
// to bf16 -- the tensor the reference's activation module sees -- with the hardware tanh (relative error about
// 2^-11, below the bf16 rounding of the result).
__device__ __forceinline__ float gelu_tanh_bf16(float x) {
  x = __bfloat162float(__float2bfloat16_rn(x));
  const float u = 0.7978845608028654f * __fmaf_rn(0.044715f * x * x, x, x);
  float t;
  asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(u));
  return 0.5f * x * (1.f + t);
}

// Programmatic dependent launch: a kernel launched with the programmatic-serialization attribute may start
// (and run its prologue: barrier init, TMEM allocation, descriptor prefetch) while the previous kernel of the
// stream is still finishing.  pdl_wait() returns once that kernel has completed and its writes are visible;
// nothing may touch global memory before it.  pdl_launch_dependents() lets the NEXT kernel start early.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// generic-proxy writes to smem -> visible to the async proxy (UMMA / TMA reads)
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// ---- TMA ---------------------------------------------------------------------------------------
__device__ __forceinline__ void prefetch_tmap(const void* tmap) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(tmap) : "memory");
}
// 2-D tiled load, completion on an mbarrier of this CTA.  x = innermost coordinate (elements).
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const void* tmap, uint32_t bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(tmap), "r"(bar), "r"(x), "r"(y)
      : "memory");
}
// 32 bytes (a whole sector) in one store; p 32-byte aligned
__device__ __forceinline__ void st_global_32(void* p, uint4 a, uint4 b) {
  asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b.x), "r"(b.y),
               "r"(b.z), "r"(b.w)
               : "memory");
}
// TMA store smem -> global (box clipped at the tensor's edges); completion is tracked per thread in bulk groups
__device__ __forceinline__ void tma_store_2d(const void* tmap, uint32_t src, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
               ::"l"(tmap), "r"(src), "r"(x), "r"(y)
               : "memory");
}
__device__ __forceinline__ void bulk_commit_group() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// all of this thread's groups have finished READING their shared-memory source (it may be overwritten)
__device__ __forceinline__ void bulk_wait_read0() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
// all but the most recent of this thread's groups have finished reading their shared-memory source
__device__ __forceinline__ void bulk_wait_read1() { asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory"); }
// all of this thread's groups are complete (the global writes are done)
__device__ __forceinline__ void bulk_wait_all0() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
// untiled bulk copy global -> smem (16-byte aligned addresses, size multiple of 16)
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
      ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
      : "memory");
}

// ---- TMEM --------------------------------------------------------------------------------------
// One full warp calls these.  ncols: power of two in [32, 512].
__device__ __forceinline__ void tmem_alloc(uint32_t dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem), "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// completion of all UMMAs issued so far by this thread -> one arrival on `bar`
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// ---- descriptors -------------------------------------------------------------------------------
// Shared-memory matrix descriptor, K-major operand stored as rows of 128 bytes with the 128-byte
// swizzle (what a TMA box of 128 bytes x rows with SWIZZLE_128B writes): 8-row groups are 1024
// bytes apart.  The tile base must be 1024-byte aligned; advancing along K inside the 128-byte
// row is done by adding the byte offset (>>4) to the start-address field.
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr & 0x3FFFF) >> 4);   // start address, bits [0,14)
  d |= (uint64_t)1 << 16;                   // leading byte offset (ignored for swizzled K-major)
  d |= (uint64_t)(1024 >> 4) << 32;         // stride byte offset: 8 rows * 128 B
  d |= (uint64_t)1 << 46;                   // descriptor version (sm_100)
  d |= (uint64_t)2 << 61;                   // SWIZZLE_128B
  return d;
}
// Unswizzled K-major, rows of 16 bytes, 8-row groups 128 bytes apart (scale-factor tiles).
__device__ __forceinline__ uint64_t smem_desc_rows16(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr & 0x3FFFF) >> 4);
  d |= (uint64_t)(128 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  return d;
}

enum : uint32_t { FMT_F16 = 0, FMT_BF16 = 1, FMT_U8 = 0, FMT_S8 = 1, FMT_E2M1_MX = 1 };
enum : uint32_t { ACC_F16 = 0, ACC_F32 = 1, ACC_S32 = 2 };

// Instruction descriptor for kind::f16 / kind::i8 (dense, both operands K-major).
__host__ __device__ constexpr uint32_t idesc_dense(uint32_t acc, uint32_t afmt, uint32_t bfmt, uint32_t M, uint32_t N) {
  return (acc << 4) | (afmt << 7) | (bfmt << 10) | ((N >> 3) << 17) | ((M >> 4) << 24);
}
// Instruction descriptor for kind::mxf4nvf4 with UE4M3 scale factors (scale_format bit 23 = 0),
// scale-factor ids 0 (a whole 32-bit TMEM column holds the four factors of one row).
__host__ __device__ constexpr uint32_t idesc_nvf4(uint32_t M, uint32_t N) {
  return (FMT_E2M1_MX << 7) | (FMT_E2M1_MX << 10) | ((N >> 3) << 17) | ((M >> 4) << 24);
}

// ---- UMMA issue (one thread) -------------------------------------------------------------------
__device__ __forceinline__ void umma_f16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accum) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accum)
      : "memory");
}
// The four K = 16 UMMAs of one 64-wide operand stage in one block: A from tensor memory (8 columns per step), B through a
// shared-memory descriptor whose low word advances by 2 (32 bytes) per step; `accum0` = 0 clears the accumulator first.
__device__ __forceinline__ void umma_f16_ts_x4(uint32_t d_tmem, uint32_t a_tmem, uint32_t bdesc_lo, uint32_t bdesc_hi,
                                               uint32_t idesc, uint32_t accum0) {
  asm volatile(
      "{\n\t.reg .pred p, t;\n\t.reg .b64 d0, d1, d2, d3;\n\t.reg .b32 l1, l2, l3, a1, a2, a3;\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "setp.eq.b32 t, 0, 0;\n\t"
      "add.u32 l1, %2, 2;\n\tadd.u32 l2, %2, 4;\n\tadd.u32 l3, %2, 6;\n\t"
      "add.u32 a1, %1, 8;\n\tadd.u32 a2, %1, 16;\n\tadd.u32 a3, %1, 24;\n\t"
      "mov.b64 d0, {%2, %3};\n\tmov.b64 d1, {l1, %3};\n\tmov.b64 d2, {l2, %3};\n\tmov.b64 d3, {l3, %3};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], d0, %4, p;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [a1], d1, %4, t;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [a2], d2, %4, t;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [a3], d3, %4, t;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "r"(bdesc_lo), "r"(bdesc_hi), "r"(idesc), "r"(accum0)
      : "memory");
}
// the same as a stage's last one
__device__ __forceinline__ uint32_t umma_f16_ts_stage(uint32_t d_tmem, uint32_t a_tmem, uint32_t bdesc_lo, uint32_t bdesc_hi, uint32_t idesc,
                                                      uint32_t accum0, uint32_t done, uint32_t next, uint32_t nph, uint32_t next2) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, t, q, q2;\n\t.reg .b64 d0, d1, d2, d3;\n\t.reg .b32 l1, l2, l3, a1, a2, a3;\n\t"
      "setp.ne.b32 p, %6, 0;\n\t"
      "setp.eq.b32 t, 0, 0;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 q, [%8], %9;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 q2, [%10], %9;\n\t"
      "add.u32 l1, %3, 2;\n\tadd.u32 l2, %3, 4;\n\tadd.u32 l3, %3, 6;\n\t"
      "add.u32 a1, %2, 8;\n\tadd.u32 a2, %2, 16;\n\tadd.u32 a3, %2, 24;\n\t"
      "mov.b64 d0, {%3, %4};\n\tmov.b64 d1, {l1, %4};\n\tmov.b64 d2, {l2, %4};\n\tmov.b64 d3, {l3, %4};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%1], [%2], d0, %5, p;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%1], [a1], d1, %5, t;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%1], [a2], d2, %5, t;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%1], [a3], d3, %5, t;\n\t"
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%7];\n\t"
      "and.pred q, q, q2;\n\tselp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"(d_tmem), "r"(a_tmem), "r"(bdesc_lo), "r"(bdesc_hi), "r"(idesc), "r"(accum0), "r"(done), "r"(next), "r"(nph), "r"(next2)
      : "memory");
  return r;
}
__device__ __forceinline__ void umma_i8(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accum) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accum)
      : "memory");
}
// E2M1 x E2M1, one UE4M3 scale factor per 16 elements along K, K = 64 per instruction.
__device__ __forceinline__ void umma_nvf4(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accum,
                                          uint32_t sfa_tmem, uint32_t sfb_tmem) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.block16 [%0], %1, %2, %3, [%5], [%6], p;\n\t}"
      ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accum), "r"(sfa_tmem), "r"(sfb_tmem)
      : "memory");
}
// The four K = 16 UMMAs of one 64-wide unit, both operands through shared-memory descriptors (see below)
__device__ __forceinline__ void umma_f16_ss_x4(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t hi, uint32_t idesc,
                                               uint32_t accum0) {
  asm volatile(
      "{\n\t.reg .pred p, t;\n\t.reg .b64 da, db;\n\t.reg .b32 x, y;\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "setp.eq.b32 t, 0, 0;\n\t"
      "mov.b64 da, {%1, %3};\n\tmov.b64 db, {%2, %3};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, p;\n\t"
      "add.u32 x, %1, 2;\n\tadd.u32 y, %2, 2;\n\tmov.b64 da, {x, %3};\n\tmov.b64 db, {y, %3};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, t;\n\t"
      "add.u32 x, %1, 4;\n\tadd.u32 y, %2, 4;\n\tmov.b64 da, {x, %3};\n\tmov.b64 db, {y, %3};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, t;\n\t"
      "add.u32 x, %1, 6;\n\tadd.u32 y, %2, 6;\n\tmov.b64 da, {x, %3};\n\tmov.b64 db, {y, %3};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, t;\n\t}"
      ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(hi), "r"(idesc), "r"(accum0)
      : "memory");
}
// One 64-wide operand stage in one block: the four K = 16 UMMAs, the commit that frees the stage (on `done`), and a test of the
// NEXT stage's barrier (`next`, parity `nph`), whose latency the UMMAs' issue hides; returns whether that phase is complete.
// Both operands through shared-memory descriptors given as low words (address >> 4, advancing by 2 = 32 bytes per step) and one
// common high word; `accum0` = 0 clears the accumulator first.
__device__ __forceinline__ uint32_t umma_f16_ss_stage(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t hi, uint32_t idesc,
                                                      uint32_t accum0, uint32_t done, uint32_t next, uint32_t nph) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, t, q;\n\t.reg .b64 da, db;\n\t.reg .b32 x, y;\n\t"
      "setp.ne.b32 p, %6, 0;\n\t"
      "setp.eq.b32 t, 0, 0;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 q, [%8], %9;\n\t"
      "mov.b64 da, {%2, %4};\n\tmov.b64 db, {%3, %4};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%1], da, db, %5, p;\n\t"
      "add.u32 x, %2, 2;\n\tadd.u32 y, %3, 2;\n\tmov.b64 da, {x, %4};\n\tmov.b64 db, {y, %4};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%1], da, db, %5, t;\n\t"
      "add.u32 x, %2, 4;\n\tadd.u32 y, %3, 4;\n\tmov.b64 da, {x, %4};\n\tmov.b64 db, {y, %4};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%1], da, db, %5, t;\n\t"
      "add.u32 x, %2, 6;\n\tadd.u32 y, %3, 6;\n\tmov.b64 da, {x, %4};\n\tmov.b64 db, {y, %4};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%1], da, db, %5, t;\n\t"
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%7];\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(hi), "r"(idesc), "r"(accum0), "r"(done), "r"(next), "r"(nph)
      : "memory");
  return r;
}
// One whole NVFP4 operand stage (four 64-element k-blocks) in one block: eight scale-factor copies shared memory ->
// tensor memory (4 columns per k-block and operand), then four block-scaled UMMAs.  Descriptors are given as low
// words (address >> 4, advancing by 2 per k-block for the operands and by 32 for the 512-byte scale tiles) with the
// two constant high words; `accum0` = 0 clears the accumulator first.
__device__ __forceinline__ void umma_nvf4_stage4(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t hi_op, uint32_t idesc,
                                                 uint32_t accum0, uint32_t sfa_tmem, uint32_t sfb_tmem, uint32_t sfa_lo,
                                                 uint32_t sfb_lo, uint32_t hi_sf) {
  asm volatile(
      "{\n\t.reg .pred p, t;\n\t.reg .b64 da, db;\n\t.reg .b32 x, y, u, v;\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "setp.eq.b32 t, 0, 0;\n\t"
      // scale factors of the four k-blocks
      "mov.b64 da, {%8, %10};\n\tmov.b64 db, {%9, %10};\n\t"
      "tcgen05.cp.cta_group::1.32x128b.warpx4 [%6], da;\n\ttcgen05.cp.cta_group::1.32x128b.warpx4 [%7], db;\n\t"
      "add.u32 x, %8, 32;\n\tadd.u32 y, %9, 32;\n\tadd.u32 u, %6, 4;\n\tadd.u32 v, %7, 4;\n\t"
      "mov.b64 da, {x, %10};\n\tmov.b64 db, {y, %10};\n\t"
      "tcgen05.cp.cta_group::1.32x128b.warpx4 [u], da;\n\ttcgen05.cp.cta_group::1.32x128b.warpx4 [v], db;\n\t"
      "add.u32 x, %8, 64;\n\tadd.u32 y, %9, 64;\n\tadd.u32 u, %6, 8;\n\tadd.u32 v, %7, 8;\n\t"
      "mov.b64 da, {x, %10};\n\tmov.b64 db, {y, %10};\n\t"
      "tcgen05.cp.cta_group::1.32x128b.warpx4 [u], da;\n\ttcgen05.cp.cta_group::1.32x128b.warpx4 [v], db;\n\t"
      "add.u32 x, %8, 96;\n\tadd.u32 y, %9, 96;\n\tadd.u32 u, %6, 12;\n\tadd.u32 v, %7, 12;\n\t"
      "mov.b64 da, {x, %10};\n\tmov.b64 db, {y, %10};\n\t"
      "tcgen05.cp.cta_group::1.32x128b.warpx4 [u], da;\n\ttcgen05.cp.cta_group::1.32x128b.warpx4 [v], db;\n\t"
      // the four UMMAs
      "mov.b64 da, {%1, %3};\n\tmov.b64 db, {%2, %3};\n\t"
      "tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.block16 [%0], da, db, %4, [%6], [%7], p;\n\t"
      "add.u32 x, %1, 2;\n\tadd.u32 y, %2, 2;\n\tadd.u32 u, %6, 4;\n\tadd.u32 v, %7, 4;\n\t"
      "mov.b64 da, {x, %3};\n\tmov.b64 db, {y, %3};\n\t"
      "tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.block16 [%0], da, db, %4, [u], [v], t;\n\t"
      "add.u32 x, %1, 4;\n\tadd.u32 y, %2, 4;\n\tadd.u32 u, %6, 8;\n\tadd.u32 v, %7, 8;\n\t"
      "mov.b64 da, {x, %3};\n\tmov.b64 db, {y, %3};\n\t"
      "tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.block16 [%0], da, db, %4, [u], [v], t;\n\t"
      "add.u32 x, %1, 6;\n\tadd.u32 y, %2, 6;\n\tadd.u32 u, %6, 12;\n\tadd.u32 v, %7, 12;\n\t"
      "mov.b64 da, {x, %3};\n\tmov.b64 db, {y, %3};\n\t"
      "tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.block16 [%0], da, db, %4, [u], [v], t;\n\t}"
      ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(hi_op), "r"(idesc), "r"(accum0), "r"(sfa_tmem), "r"(sfb_tmem), "r"(sfa_lo),
        "r"(sfb_lo), "r"(hi_sf)
      : "memory");
}
// 32 rows x 16 bytes of smem -> TMEM lanes 0..31 (4 columns), replicated to all four lane quarters.
__device__ __forceinline__ void tmem_cp_32x128b_x4(uint32_t taddr, uint64_t sdesc) {
  asm volatile("tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], %1;" ::"r"(taddr), "l"(sdesc) : "memory");
}

// ---- TMEM -> registers: warp w of a warpgroup reads lanes 32*(w%4).. ; thread i gets lane i ----
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
// waits for this thread's TMEM loads and names the registers they fill, so that no use of these moves before the wait
__device__ __forceinline__ void tmem_wait_ld16(uint32_t* r) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]),
                 "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
               :: "memory");
}
// Register split between the warpgroups of a block (all four warps of a group execute the same one).  The sum over the
// groups must not exceed what the block was launched with.  regs_even gives every group the launch's share back, for code that
// all run; only behind a barrier that all have passed: a group that took registers back while another still waited for its own
// would leave both waiting for good.
template <int N> __device__ __forceinline__ void reg_alloc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N> __device__ __forceinline__ void reg_dealloc() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }
template <int LAUNCH> __device__ __forceinline__ void regs_even(bool grew) {
  if (grew) reg_dealloc<LAUNCH>();
  else reg_alloc<LAUNCH>();
}
// registers -> TMEM: 32 consecutive 32-bit columns of this thread's lane
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
      "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
        "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
        "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
// registers -> TMEM: 16 consecutive 32-bit columns of this thread's lane
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}


}  // namespace dq
