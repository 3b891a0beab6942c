// Inline PTX for CTA pairs (clusters of two CTAs on neighbouring SMs driving ONE tcgen05.mma with cta_group::2):
// cluster rank and barrier, addresses in the peer's shared memory, TMA loads whose completion is counted on the
// leader's mbarrier, pair-wide TMEM allocation, pair UMMAs / scale-factor copies / commits.  Every load here brings
// its bytes into the issuing CTA's own shared memory only; the two CTAs of a pair each fetch their own halves.
#pragma once
#include <cstdint>
#include "ptx.cuh"

namespace dq {

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_id_x() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%clusterid.x;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_count_x() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%nclusterid.x;" : "=r"(r));
  return r;
}
// shared::cluster address of the same shared-memory offset in CTA `rank` of this cluster
__device__ __forceinline__ uint32_t map_to_rank(uint32_t smem_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
  return r;
}
// all threads of both CTAs; orders the shared-memory writes before it (barrier initialisation) cluster-wide
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// One arrival on an mbarrier that may live in the peer CTA (shared::cluster address), without memory ordering: for hand-offs
// whose payload is TENSOR memory, not shared or global memory.  Tensor-memory accesses of two threads are ordered by the
// tcgen05 fences around the barrier, which itself has to order execution only; this is the pattern that the PTX ISA gives for
// it (tcgen05, memory consistency model, synchronization between different threads): tcgen05.wait::ld or ::st,
// tcgen05.fence::before_thread_sync and a relaxed cluster-scope arrival on this side, the barrier's wait and
// tcgen05.fence::after_thread_sync on the other.  A cluster-scope release has to drain the thread's
// earlier stores first and costs on the order of a microsecond per arrival on this kernel's critical path.
__device__ __forceinline__ void mbar_arrive_cluster_relaxed(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}

// A word of either CTA's shared memory (shared::cluster address)
__device__ __forceinline__ int ld_cluster_s32(uint32_t cluster_addr) {
  int v;
  asm volatile("ld.relaxed.cluster.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(cluster_addr) : "memory");
  return v;
}
// Takes `bytes` off a barrier's pending count, as a copy of that size would when it lands
__device__ __forceinline__ void mbar_complete_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.complete_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// Teardown of a pair's ring after a wait ran out, by the leader's producer thread once both CTAs have stopped.  A stage's
// barrier (in the leader) expects one arrival with the bytes of both halves, `half_of(stage)` from each CTA; of the stages below
// `upto` -- as far as any role of either CTA got -- the leader has armed `own` and the peer issued copies for `peer`.
// What one CTA did and the other did not is made up for, so that every such phase completes exactly when the copies that
// were issued have landed (the warps that also arrive on these barriers make up for theirs); then the last ring of them
// is awaited.  No role is more than a ring behind another: a slot is reused only after all arrived for its last stage.
// (`upto` must not count a stage that a role merely walked past: two stages on one barrier would arrive more often than the
// phase at hand expects while bytes are missing, which is a fault.)
template <typename F, typename H>
__device__ __forceinline__ void drain_pair_ring(F bar_of, int slots, int own, int peer, int upto, H half_of, int* status) {
  for (int q = own; q < upto; ++q) mbar_expect_tx(bar_of(q % slots), q < peer ? half_of(q) : 0u);
  for (int q = peer; q < own; ++q) mbar_complete_tx(bar_of(q % slots), half_of(q));
  drain_ring(bar_of, slots, upto, status);
}

// 2-D tiled load into THIS CTA's shared memory; the bytes are counted on `bar`, a shared::cluster address that may
// name the leader CTA's mbarrier (the cta_group::2 form is what allows the barrier to sit in the peer).
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const void* tmap, uint32_t bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(tmap), "r"(bar), "r"(x), "r"(y)
      : "memory");
}

// ---- TMEM for a pair: one full warp of EACH CTA calls these with the same arguments ----------------------------------
__device__ __forceinline__ void tmem_alloc_pair(uint32_t dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem), "r"(ncols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// Completion of all pair UMMAs issued so far by this thread -> one arrival on the barrier at this shared-memory offset in
// BOTH CTAs of the pair.  One commit of this form instead of two (the second to an address mapped from the peer), with a
// stage's FP4 UMMAs in one block, took the NVFP4 GEMM on 128-wide tiles from 150 to 130 us for 1152 -> 3456 at 32768 rows (which
// now takes 256-wide ones): what the issuing thread does is time the pipe idles.
__device__ __forceinline__ void umma_commit_pair_both(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(bar), "h"((uint16_t)3) : "memory");
}
// E2M1 x E2M1 with UE4M3 scale factors, 256 x N x 64 over the pair: each CTA contributes its 128 rows of A, its
// N/2 rows of B and holds its 128 x N half of the accumulator
__device__ __forceinline__ void umma_nvf4_pair(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accum,
                                               uint32_t sfa_tmem, uint32_t sfb_tmem) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::mxf4nvf4.block_scale.block16 [%0], %1, %2, %3, [%5], [%6], p;\n\t}"
      ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accum), "r"(sfa_tmem), "r"(sfb_tmem)
      : "memory");
}
// A whole operand stage in one block: the four UMMAs, the commit that frees the stage in both CTAs (on `done`), and a test of the
// NEXT stage's barrier (`next`, parity `nph`), whose latency the UMMAs' issue hides; returns whether that phase is complete.
// Descriptors as low words (address >> 4, advancing by 2 = 32 bytes per step) with one high word; `accum0` = 0 clears the
// accumulator first.  FP4: the scale factors 4 (activations) and SFB (weights) columns apart.
template <int SFB>
__device__ __forceinline__ uint32_t umma_nvf4_stage_pair(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t hi, uint32_t idesc,
                                                         uint32_t accum0, uint32_t sfa, uint32_t sfb, uint32_t done, uint32_t next,
                                                         uint32_t nph) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, t, q;\n\t.reg .b64 da, db;\n\t.reg .b32 x, y, u, v;\n\t"
      "setp.ne.b32 p, %6, 0;\n\t"
      "setp.eq.b32 t, 0, 0;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 q, [%8], %9;\n\t"
      "mov.b64 da, {%2, %4};\n\tmov.b64 db, {%3, %4};\n\t"
      "tcgen05.mma.cta_group::2.kind::mxf4nvf4.block_scale.block16 [%1], da, db, %5, [%11], [%12], p;\n\t"
      "add.u32 x, %2, 2;\n\tadd.u32 y, %3, 2;\n\tmov.b64 da, {x, %4};\n\tmov.b64 db, {y, %4};\n\t"
      "add.u32 u, %11, 4;\n\tadd.u32 v, %12, %13;\n\t"
      "tcgen05.mma.cta_group::2.kind::mxf4nvf4.block_scale.block16 [%1], da, db, %5, [u], [v], t;\n\t"
      "add.u32 x, %2, 4;\n\tadd.u32 y, %3, 4;\n\tmov.b64 da, {x, %4};\n\tmov.b64 db, {y, %4};\n\t"
      "add.u32 u, %11, 8;\n\tadd.u32 v, %12, %14;\n\t"
      "tcgen05.mma.cta_group::2.kind::mxf4nvf4.block_scale.block16 [%1], da, db, %5, [u], [v], t;\n\t"
      "add.u32 x, %2, 6;\n\tadd.u32 y, %3, 6;\n\tmov.b64 da, {x, %4};\n\tmov.b64 db, {y, %4};\n\t"
      "add.u32 u, %11, 12;\n\tadd.u32 v, %12, %15;\n\t"
      "tcgen05.mma.cta_group::2.kind::mxf4nvf4.block_scale.block16 [%1], da, db, %5, [u], [v], t;\n\t"
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%7], %10;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(hi), "r"(idesc), "r"(accum0), "r"(done), "r"(next), "r"(nph), "h"((uint16_t)3), "r"(sfa),
        "r"(sfb), "n"(SFB), "n"(2 * SFB), "n"(3 * SFB)
      : "memory");
  return r;
}
__device__ __forceinline__ void umma_f16_ss_x4_pair(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t hi, uint32_t idesc,
                                               uint32_t accum0) {
  asm volatile(
      "{\n\t.reg .pred p, t;\n\t.reg .b64 da, db;\n\t.reg .b32 x, y;\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "setp.eq.b32 t, 0, 0;\n\t"
      "mov.b64 da, {%1, %3};\n\tmov.b64 db, {%2, %3};\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %4, p;\n\t"
      "add.u32 x, %1, 2;\n\tadd.u32 y, %2, 2;\n\tmov.b64 da, {x, %3};\n\tmov.b64 db, {y, %3};\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %4, t;\n\t"
      "add.u32 x, %1, 4;\n\tadd.u32 y, %2, 4;\n\tmov.b64 da, {x, %3};\n\tmov.b64 db, {y, %3};\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %4, t;\n\t"
      "add.u32 x, %1, 6;\n\tadd.u32 y, %2, 6;\n\tmov.b64 da, {x, %3};\n\tmov.b64 db, {y, %3};\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %4, t;\n\t}"
      ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(hi), "r"(idesc), "r"(accum0)
      : "memory");
}
__device__ __forceinline__ uint32_t umma_f16_ss_stage_pair(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t hi, uint32_t idesc,
                                                           uint32_t accum0, uint32_t done, uint32_t next, uint32_t nph) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, t, q;\n\t.reg .b64 da, db;\n\t.reg .b32 x, y;\n\t"
      "setp.ne.b32 p, %6, 0;\n\t"
      "setp.eq.b32 t, 0, 0;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 q, [%8], %9;\n\t"
      "mov.b64 da, {%2, %4};\n\tmov.b64 db, {%3, %4};\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%1], da, db, %5, p;\n\t"
      "add.u32 x, %2, 2;\n\tadd.u32 y, %3, 2;\n\tmov.b64 da, {x, %4};\n\tmov.b64 db, {y, %4};\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%1], da, db, %5, t;\n\t"
      "add.u32 x, %2, 4;\n\tadd.u32 y, %3, 4;\n\tmov.b64 da, {x, %4};\n\tmov.b64 db, {y, %4};\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%1], da, db, %5, t;\n\t"
      "add.u32 x, %2, 6;\n\tadd.u32 y, %3, 6;\n\tmov.b64 da, {x, %4};\n\tmov.b64 db, {y, %4};\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%1], da, db, %5, t;\n\t"
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%7], %10;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(hi), "r"(idesc), "r"(accum0), "r"(done), "r"(next), "r"(nph), "h"((uint16_t)3)
      : "memory");
  return r;
}
// A from the tensor memory of both CTAs (each holds its own 128 rows at the same columns, 8 per step), B through a shared-memory
// descriptor (each CTA holds N/2 rows at the same offset)
__device__ __forceinline__ void umma_f16_ts_x4_pair(uint32_t d_tmem, uint32_t a_tmem, uint32_t bdesc_lo, uint32_t bdesc_hi,
                                                    uint32_t idesc, uint32_t accum0) {
  asm volatile(
      "{\n\t.reg .pred p, t;\n\t.reg .b64 d0, d1, d2, d3;\n\t.reg .b32 l1, l2, l3, a1, a2, a3;\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "setp.eq.b32 t, 0, 0;\n\t"
      "add.u32 l1, %2, 2;\n\tadd.u32 l2, %2, 4;\n\tadd.u32 l3, %2, 6;\n\t"
      "add.u32 a1, %1, 8;\n\tadd.u32 a2, %1, 16;\n\tadd.u32 a3, %1, 24;\n\t"
      "mov.b64 d0, {%2, %3};\n\tmov.b64 d1, {l1, %3};\n\tmov.b64 d2, {l2, %3};\n\tmov.b64 d3, {l3, %3};\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], d0, %4, p;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], [a1], d1, %4, t;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], [a2], d2, %4, t;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], [a3], d3, %4, t;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "r"(bdesc_lo), "r"(bdesc_hi), "r"(idesc), "r"(accum0)
      : "memory");
}
__device__ __forceinline__ uint32_t umma_f16_ts_stage_pair(uint32_t d_tmem, uint32_t a_tmem, uint32_t bdesc_lo, uint32_t bdesc_hi,
                                                           uint32_t idesc, uint32_t accum0, uint32_t done, uint32_t next, uint32_t nph) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, t, q;\n\t.reg .b64 d0, d1, d2, d3;\n\t.reg .b32 l1, l2, l3, a1, a2, a3;\n\t"
      "setp.ne.b32 p, %6, 0;\n\t"
      "setp.eq.b32 t, 0, 0;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 q, [%8], %9;\n\t"
      "add.u32 l1, %3, 2;\n\tadd.u32 l2, %3, 4;\n\tadd.u32 l3, %3, 6;\n\t"
      "add.u32 a1, %2, 8;\n\tadd.u32 a2, %2, 16;\n\tadd.u32 a3, %2, 24;\n\t"
      "mov.b64 d0, {%3, %4};\n\tmov.b64 d1, {l1, %4};\n\tmov.b64 d2, {l2, %4};\n\tmov.b64 d3, {l3, %4};\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%1], [%2], d0, %5, p;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%1], [a1], d1, %5, t;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%1], [a2], d2, %5, t;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%1], [a3], d3, %5, t;\n\t"
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%7], %10;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"(d_tmem), "r"(a_tmem), "r"(bdesc_lo), "r"(bdesc_hi), "r"(idesc), "r"(accum0), "r"(done), "r"(next), "r"(nph), "h"((uint16_t)3)
      : "memory");
  return r;
}

}  // namespace dq
