// Kernel 2 (INT4, tensor-rate variant): W4A4 GEMM whose 4-bit operands are dequantised to fp16 on their
// way to the tensor core, so that ONE fp32 accumulator runs over the whole K and the per-chunk
// CUDA-core drain of the exact-integer kernel (gemm_int.cu) disappears.
//
//   y[m,n] = rs[m] cs[n] ( sum_k a'[m,k] b'[n,k] + xt'[m,:] . wt'[n,:] ) + bias[n]
//   a'[m,k] = (qx[m,k] - zx[m,c]) * sx[m,c] / rs[m]      exact in fp16 for symmetric codes
//   b'[n,k] =  qw[n,k]            * sw[n,c] / cs[n]      rounded once to fp16 (11 bits; the reference
//                                                         keeps bf16(qw * sw), 8 bits)
//   rs[m], cs[n] = powers of two that bring a row's / a column's largest scale to [2^-10, 2^-9)
//
// This is the arithmetic of the reference's own linear on the fake-quantised tensor
// (DiRotQ dirotq_fused_unrotation_fast.py:141: a 16-bit GEMM with fp32 accumulation over
// s*(q-z) and the stored weight), with operands that stay 4-bit in HBM, L2 and the TMA ring.
//
// Nibble -> fp16 without integer-to-float conversion: a nibble m left in the low mantissa bits of an
// otherwise zero half is the subnormal m * 2^-24; one fused multiply-add with the pre-scaled group
// scale (s * 2^24) and the addend -(z * s) gives (m - z) * s with a single rounding.  Two nibbles
// of a byte are taken in place (bits 0-3 and 4-7, the latter with the multiplier s * 2^20), so a
// 32-bit word of eight codes costs one shift, four logic ops and four packed FMAs.
// The order in which a chunk's 64 values land along K is a fixed permutation, the same for both
// operands, which a dot product does not see.
//
// Conversion work (issue slots, shared-memory stores), not tensor arithmetic, bounds a kernel that expands
// operands on chip, and every CTA that expands a weight tile repeats what M / 128 other CTAs do.  So:
//   * the weight operand is expanded ONCE per call by a small pre-pass (expand_weight_panel_kernel: codes
//     + records -> an fp16 [N, K] panel in scratch, 2 bytes per weight, L2-resident for DiT layer sizes;
//     the stored weights stay 4-bit) and reaches the operand ring by TMA, already swizzled;
//   * the activation operand never touches shared memory in expanded form: its converter threads (one
//     per row = one TMEM lane) store the fp16 values straight into tensor memory, and the UMMA takes A
//     from TMEM, B from smem.
//
// Data flow per persistent CTA (128 x BN output tiles, K walked in 64-wide units, one or two to an operand stage):
//   TMA (A)        4-bit codes (four chunks = 128 B per row per stage, 128-byte swizzle) + the chunks' scales and zero
//                  points, or (REC) the records a folding kernel made of them (bulk copies) -> "raw" ring
//   TMA (B)        BN x 64 fp16 tiles of the panel (or of the bf16 tail weights), one per unit, straight into the stage's
//                  128-byte-swizzled K-major slot as soon as the UMMAs that read it retire
//   converter warps  two groups of four taking alternate stages; a warp expands 32 activation rows into TMEM
//                  (tcgen05.st); for a tail stage it copies the bf16 rows from the raw ring instead
//   UMMA issuer    tcgen05.mma kind::f16 (A from TMEM, B from smem descriptor), 4 x K=16 per chunk, fp32
//                  128 x BN accumulator in TMEM; the bf16 tail accumulates into the same tile
//   8 epilogue warps  tcgen05.ld, * rs[m] * cs[n], + bias, bf16 in registers, accumulator handed back, then 32 x 32 staging
//                  patches -> TMA stores.  128-wide tiles have two accumulators, wider ones one (the columns it leaves hold
//                  eight units of activations)
// PAIR (192- and 256-wide tiles): clusters of two CTAs drive one tcgen05.mma.cta_group::2 on a 256-row tile, which halves the
// weight traffic and issues one UMMA for two SMs.  Each CTA converts its own 128 rows into its own tensor memory, fetches half of the weight tile (the tensor core reads the other
// half from the peer's shared memory) and runs the epilogue of its 128 rows.  One barrier per stage in the leader counts the
// weight bytes of both CTAs and one arrival per converter warp of both (from the peer without memory ordering: their payload
// is tensor memory); commits arrive in both CTAs; accumulator-empty in the leader counts the epilogue warps of both.
#include <cuda.h>
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <atomic>
#include "layout.cuh"
#include "launchers.cuh"
#include "ptx.cuh"
#include "ptx_pair.cuh"
#include "tma_host.cuh"
#include "quant_math.cuh"

namespace dq {

#ifndef GF_CPS_DEF
#define GF_CPS_DEF 4
#endif
#ifndef GF_RAW_DEF
#define GF_RAW_DEF 2
#endif
#ifndef GF_EXP_MAX
#define GF_EXP_MAX 8
#endif
#ifndef GF_GROUPS
#define GF_GROUPS 2
#endif
constexpr int GF_CPS = GF_CPS_DEF;   // chunks per raw stage: 128 bytes of codes per row and stage
constexpr int GF_EPI_WARPS = 8;

// A chunk of a 128-row tile is four conversion units of 32 rows (a thread per row = TMEM lane); a group is
// the four warps that cover the four lane quarters.
template <int BN, bool A8 = false, bool PAIR = false, bool REC = false> struct GfCfg {
  // 64-wide pieces of K ("units") per operand stage.  A stage costs every role a wait (a barrier test takes 110 cycles even when the
  // phase is complete) and the issuer, all in all, 270 cycles besides its UMMAs, which narrow tiles do not hide: two units (us, one /
  // two: 512 x 12288 x 3072 on 128 columns 56.5 / 48.7, 4096 x 4608 x 1152 44 / 39.3, 4096 x 1152 x 1152 16.8 / 15.6; 8192 x 2240 x
  // 2240 on 192 67.6 / 65.5).  256-wide tiles do hide them and would rather have eight small stages in flight than four large ones (16384 x
  // 2240 x 2240 113.9 / 117.2, 32768 x 1152 x 3456 197 / 206).
  static constexpr int UNITS = BN == 256 ? 1 : 2;
  static constexpr int GROUP_WARPS = 4;
  static constexpr int GROUPS = GF_GROUPS;
  static constexpr int CONV_WARPS = GROUPS * GROUP_WARPS;
  // Warpgroups: epilogue (warps 0..7), issuer and the two producers (8..11, the last one idle), converters (12..19).  The
  // launch gives every thread 96 registers; the producers' and converters' groups hand some back to the epilogue's, which
  // holds a quarter row of the tile (64 registers of bf16 pairs) besides the piece in work and the one being fetched.
  // Epilogue / issuer and producers / converters.  On pairs 128 / 48 / 88 spills 52 bytes a thread in the issuer and 120 / 80 / 80 does
  // not (32768 x 1152 x 3456 205 -> 201 us); 8-bit converters hold twice the codes and take 88 from the producers (32768 x 1152 x 3456
  // 208.9 with 80 / 80, 210.5 with 112 / 80 / 88, 206.9 with 120 / 64 / 88).  128-wide tiles spill 24 bytes with 128 / 48 / 88 and are no
  // faster with 128 / 64 / 80 or 120 / 80 / 80 (1024 x 2240 x 2240 14.3 / 14.8).
  static constexpr int THREADS = (GF_EPI_WARPS + 4 + CONV_WARPS) * 32;
  static constexpr int REGS_LAUNCH = 96, REGS_EPI = PAIR ? 120 : 128, REGS_PROD = !PAIR ? 48 : A8 ? 64 : 80, REGS_CONV = PAIR && !A8 ? 80 : 88;
  static_assert(GF_EPI_WARPS * REGS_EPI + 4 * REGS_PROD + CONV_WARPS * REGS_CONV <= THREADS / 32 * REGS_LAUNCH,
                "setmaxnreg draws on the registers of the launch");
  static constexpr int BN_OWN = PAIR ? BN / 2 : BN;         // weight rows this CTA fetches
  static constexpr int B_EXP = BN_OWN * 128;               // BN_OWN rows x 64 halves
  static constexpr int EXP_STAGE = UNITS * B_EXP;          // only the weight operand is staged in shared memory
  static constexpr int A_COLS = UNITS * 32;                // tensor-memory columns of a stage's activations
  static constexpr int RAW_A = 128 * 32 * GF_CPS * (A8 ? 2 : 1);   // 8-bit activation codes: two 128-byte boxes per row
  static constexpr int OFF_C = RAW_A;                      // REC: [chunk][128] 8-byte records; else [chunk][128] bf16 scales
  static constexpr int OFF_Z = OFF_C + GF_CPS * 128 * 2;   // and as many zero points
  static constexpr int RAW_STAGE = OFF_C + GF_CPS * 128 * 8;
  // Accumulators: two of 128 columns (the next tile's UMMAs overlap the epilogue); a wider tile has one, and its
  // UMMAs wait until the epilogue has read the previous tile out of tensor memory.
  static constexpr int NACC = BN > 128 ? 1 : 2;
  // Operand stages in flight: every tensor-memory column the accumulators leave free holds activations
  // (32 columns per unit), as far as shared memory holds the weight tiles beside them.
  static constexpr int RAW_STAGES = GF_RAW_DEF;
  static constexpr int STG_BYTES = GF_EPI_WARPS * 2048;     // per epilogue warp: 32 rows x 32 bf16 output staging
  static constexpr int PIECES = BN / 32;                    // 16-column pieces of an epilogue warp
  static constexpr int TAB_WARP = PIECES * 8 * 8;           // per epilogue warp: {cs pair, bias pair} in bf16 per column pair
  static constexpr int TAB_BYTES = GF_EPI_WARPS * TAB_WARP;
  // 1 / rs per row, for several tiles: the epilogue warps write a tile's once the accumulator before last has come, when
  // every converter warp has at least released the raw stage RAW_STAGES before that tile's last one
  static constexpr int ROW_TILES = 4;
  static constexpr int ROW_BYTES = ROW_TILES * 128 * 4;
  static_assert(ROW_TILES >= RAW_STAGES + 2, "a slot of the row table may still be in use");
  static constexpr int EXP_TMEM = (512 - NACC * BN) / A_COLS;
  static constexpr int BAR_BYTES = 384;                     // barriers, tensor-memory address, failure words
  static constexpr int EXP_SMEM = (232448 - 1024 - BAR_BYTES - STG_BYTES - TAB_BYTES - ROW_BYTES - RAW_STAGES * RAW_STAGE) / EXP_STAGE;
  static constexpr int EXP_CAP = EXP_TMEM < GF_EXP_MAX ? EXP_TMEM : GF_EXP_MAX;
  static constexpr int EXP_STAGES = EXP_CAP < EXP_SMEM ? EXP_CAP : EXP_SMEM;
  static constexpr int SMEM_BYTES = EXP_STAGES * EXP_STAGE + RAW_STAGES * RAW_STAGE + STG_BYTES + TAB_BYTES + ROW_BYTES + 1024 + BAR_BYTES;
  static constexpr int NBARS = 2 * RAW_STAGES + 3 * EXP_STAGES + 4 + ROW_TILES;
  static_assert(NBARS * 8 + 4 + AB_WORDS * 4 <= BAR_BYTES && CONV_WARPS <= AB_WORDS - AB_WARP, "barrier area");
  static constexpr int TMEM_A0 = NACC * BN;                 // first column of the activation operand slots
  static constexpr int TMEM_COLS = 512;                     // accumulators + EXP_STAGES x A_COLS columns of A
  static_assert(NACC * BN + EXP_STAGES * A_COLS <= 512 && EXP_STAGES >= 2, "tensor memory");
  static_assert(SMEM_BYTES <= 232448, "shared memory");
  static_assert(RAW_A >= 128 * 128 && GF_CPS == 4, "a raw stage must hold one 128 x 64 bf16 tail tile of the activations");
};

struct GfMaps {
  CUtensorMap xq, xs, xz, wp, xt, wt, y;
};

template <int N> struct GfRing {
  int s = 0;
  uint32_t ph = 0;
  __device__ __forceinline__ void next() { if (++s == N) { s = 0; ph ^= 1; } }
};

__device__ __forceinline__ void gf_sts128(uint32_t addr, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
  asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
__device__ __forceinline__ void gf_sts64(uint32_t addr, uint32_t x, uint32_t y) {
  asm volatile("st.shared.v2.b32 [%0], {%1,%2};" ::"r"(addr), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ uint2 gf_lds64(uint32_t addr) {
  uint2 v;
  asm volatile("ld.shared.v2.b32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ uint4 gf_lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}
// (a & b) ^ c in one logic op
__device__ __forceinline__ uint32_t and_xor(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t r;
  asm("lop3.b32 %0, %1, %2, %3, 0x6A;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
  return r;
}
__device__ __forceinline__ uint32_t hfma2_u(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t r;
  asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
  return r;
}

// One 32-bit word of eight planar nibbles -> four fp16 pairs.
//   xr : per-nibble XOR (0x8 turns a two's-complement nibble into offset binary; 0 for unsigned codes)
//   mlo = (s * 2^24) twice, mhi = (s * 2^20) twice, add = -(z * s) twice (z = 8 for signed codes)
__device__ __forceinline__ void expand_word(uint32_t w, uint32_t xr, uint32_t mlo, uint32_t mhi, uint32_t add, uint32_t* y) {
  const uint32_t t = w >> 8;
  y[0] = hfma2_u(and_xor(w, 0x000F000Fu, xr), mlo, add);
  y[1] = hfma2_u(and_xor(w, 0x00F000F0u, xr << 4), mhi, add);
  y[2] = hfma2_u(and_xor(t, 0x000F000Fu, xr), mlo, add);
  y[3] = hfma2_u(and_xor(t, 0x00F000F0u, xr << 4), mhi, add);
}
__device__ __forceinline__ uint32_t hmul2_2m4(uint32_t m) {
  uint32_t r;
  asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(m), "r"(0x2C002C00u));     // * 2^-4
  return r;
}

// 32 codes of one row, as loaded, -> 16 fp16 pairs of (code - z) * s, by the record k of their chunk: 16 planar bytes ...
template <bool ASYM>
__device__ __forceinline__ void expand_nibbles32(uint4 p, uint2 k, uint32_t* y) {
  const uint32_t mhi = hmul2_2m4(k.x), xr = ASYM ? 0u : 0x00080008u;
  expand_word(p.x, xr, k.x, mhi, k.y, y);
  expand_word(p.y, xr, k.x, mhi, k.y, y + 4);
  expand_word(p.z, xr, k.x, mhi, k.y, y + 8);
  expand_word(p.w, xr, k.x, mhi, k.y, y + 12);
}
// ... or 32 bytes: a byte alone in a zero half is the subnormal q * 2^-24, so (q - z) * s is one packed FMA again; the values
// are emitted in the K order the 4-bit weight expansion produces (see expand_word)
__device__ __forceinline__ void expand_bytes32(const uint4* p, uint2 k, uint32_t* y) {
  const uint32_t w[8] = {p[0].x, p[0].y, p[0].z, p[0].w, p[1].x, p[1].y, p[1].z, p[1].w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    y[4 * i] = hfma2_u(__byte_perm(w[i], 0u, 0x4240), k.x, k.y);
    y[4 * i + 1] = hfma2_u(__byte_perm(w[4 + i], 0u, 0x4240), k.x, k.y);
    y[4 * i + 2] = hfma2_u(__byte_perm(w[i], 0u, 0x4341), k.x, k.y);
    y[4 * i + 3] = hfma2_u(__byte_perm(w[4 + i], 0u, 0x4341), k.x, k.y);
  }
}

__device__ __forceinline__ uint32_t hmul2_m8(uint32_t m) {
  uint32_t r;
  asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(m), "r"(0x80088008u));     // * -8 * 2^-24
  return r;
}
__device__ __forceinline__ uint32_t gf_lds16(uint32_t addr) {
  uint16_t v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ float gf_lds_f32(uint32_t addr) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void gf_sts_f32(uint32_t addr, float v) {
  asm volatile("st.shared.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ uint32_t half_twice(float v) {
  const __half2 h = __floats2half2_rn(v, v);
  return *reinterpret_cast<const uint32_t*>(&h);
}
// larger magnitudes of two bf16 pairs (a NaN gives way to the other value)
__device__ __forceinline__ uint32_t abs_max_bf16x2(uint32_t m, uint32_t v) {
  v &= 0x7FFF7FFFu;
  const __nv_bfloat162 r = __hmax2(*reinterpret_cast<const __nv_bfloat162*>(&m), *reinterpret_cast<const __nv_bfloat162*>(&v));
  return *reinterpret_cast<const uint32_t*>(&r);
}
// The power of two of a row (token or output channel) whose largest chunk scale is smax: rs = 2^(10 + E) for smax = 1.f * 2^E, so
// that smax / rs lies in [2^-10, 2^-9).  Returns 1 / rs.
__device__ __forceinline__ float row_inverse_power(float smax, float& rs) {
  int E = (int)((__float_as_uint(smax) >> 23) & 0xFF) - 127;
  E = max(-100, min(100, E));
  rs = __uint_as_float((uint32_t)(127 + 10 + E) << 23);
  return __uint_as_float((uint32_t)(127 - 10 - E) << 23);
}
// A chunk's multiplier and addend as fp16 pairs, { (s * 2^24 / rs) twice, -(z * s / rs) twice }, ready to be used as packed-FMA
// operands; inv = 1 / rs (E >= -100 keeps inv * 2^24 finite).
__device__ __forceinline__ uint2 chunk_record(float s, float z, float inv) {
  return make_uint2(half_twice(s * (inv * 16777216.f)), half_twice(-z * s * inv));
}

// bf16 pair of { v0 * rs * cs0 + b0, v1 * rs * cs1 + b1 } from bf16 pairs cs and b; rs and cs are powers of two, so only the
// sum and the conversion round
__device__ __forceinline__ uint32_t scale_pair(uint32_t v0, uint32_t v1, float rs, uint32_t cs, uint32_t b) {
  uint32_t r;
  asm("{\n\t.reg .b64 v, s, c, b;\n\t.reg .b32 lo, hi, c0, c1, b0, b1;\n\t"
      "shl.b32 c0, %4, 16;\n\tand.b32 c1, %4, 0xffff0000;\n\t"
      "shl.b32 b0, %5, 16;\n\tand.b32 b1, %5, 0xffff0000;\n\t"
      "mov.b64 v, {%1, %2};\n\tmov.b64 s, {%3, %3};\n\tmov.b64 c, {c0, c1};\n\tmov.b64 b, {b0, b1};\n\t"
      "mul.rn.f32x2 c, c, s;\n\t"
      "fma.rn.f32x2 v, v, c, b;\n\t"
      "mov.b64 {lo, hi}, v;\n\t"
      "cvt.rn.bf16x2.f32 %0, hi, lo;\n\t}"
      : "=r"(r)
      : "r"(v0), "r"(v1), "r"(__float_as_uint(rs)), "r"(cs), "r"(b));
  return r;
}

// After a wait ran out, by all threads (of both CTAs of a pair) once the roles have stopped: await what is in flight.
template <int BN, bool A8, bool PAIR, typename F>
__device__ __forceinline__ void gf_teardown(uint8_t* bars, F half_of, int* status) {
  using Cfg = GfCfg<BN, A8, PAIR>;
  constexpr int GF_EXP_STAGES = Cfg::EXP_STAGES, GF_RAW_STAGES = Cfg::RAW_STAGES;
  constexpr int W_MMA = GF_EPI_WARPS, W_TMA = GF_EPI_WARPS + 1, W_TMB = GF_EPI_WARPS + 2, W_CONV = GF_EPI_WARPS + 4;
  volatile int* const ab = reinterpret_cast<volatile int*>(bars + 8 * Cfg::NBARS) + 1;
  const int warp = threadIdx.x >> 5;
  const uint32_t b0 = smem_u32(bars);
  auto ring = [&](int first_bar) { return [=](int s) { return b0 + 8u * (first_bar + s); }; };
  const auto rawf = ring(0), expf = ring(2 * GF_RAW_STAGES), expe = ring(2 * GF_RAW_STAGES + GF_EXP_STAGES),
             expw = ring(2 * GF_RAW_STAGES + 2 * GF_EXP_STAGES), accf = ring(2 * GF_RAW_STAGES + 3 * GF_EXP_STAGES);
  const uint32_t ab0 = b0 + 8u * Cfg::NBARS + 4u;
  const bool one = (threadIdx.x & 31) == 0;                 // one lane per warp
  const int own = ab[AB_ISSUED2];
  if (warp == W_TMA && one) drain_ring(rawf, GF_RAW_STAGES, ab[AB_ISSUED], status);
  if constexpr (PAIR) {
    // see drain_pair_ring; converters run ahead of the weight tiles, so the furthest role is looked for among all
    const uint32_t cta = cluster_ctarank();
    if (threadIdx.x == 0) {
      int m = own;
      for (int i = 0; i < Cfg::CONV_WARPS; ++i) m = max(m, ab[AB_WARP + i]);
      ab[AB_MAX] = m;
    }
    __syncwarp();
    __syncthreads();
    cluster_sync_all();
    const uint32_t other = map_to_rank(ab0, cta ^ 1);
    const int peer = ld_cluster_s32(other + 4u * AB_ISSUED2);
    const int upto = max((int)ab[AB_MAX], ld_cluster_s32(other + 4u * AB_MAX));
    if (warp >= W_CONV && one) {
      const int cw = warp - W_CONV, grp = cw / Cfg::GROUP_WARPS;
      const uint32_t fb = map_to_rank(expf(0), 0);
      for (int n = ab[AB_WARP + cw]; n < upto; ++n)
        if (n % Cfg::GROUPS == grp) mbar_arrive_cluster_relaxed(fb + 8u * (n % GF_EXP_STAGES));
    }
    if (warp == W_TMB && one && cta == 0) drain_pair_ring(expf, GF_EXP_STAGES, own, peer, upto, half_of, status);
  } else if (warp == W_TMB && one) {
    drain_ring(expw, GF_EXP_STAGES, own, status);
  }
  if (warp == W_MMA && one) {                          // in both CTAs of a pair, where the leader's commits arrive
    int stages = ab[AB_UMMA], accs = ab[AB_ACC];
    if constexpr (PAIR) {
      const uint32_t lead = map_to_rank(ab0, 0);
      stages = ld_cluster_s32(lead + 4u * AB_UMMA);
      accs = ld_cluster_s32(lead + 4u * AB_ACC);
    }
    drain_ring(expe, GF_EXP_STAGES, stages, status);
    drain_ring(accf, Cfg::NACC, accs, status);
  }
  __syncwarp();
  __syncthreads();
  if constexpr (PAIR) cluster_sync_all();
}

// AMODE: 0 = signed 4-bit activation codes, 1 = unsigned 4-bit with zero points, 2 = unsigned 8-bit with zero points
// PAIR: see the head of this file
template <int BN, int AMODE, bool PAIR, bool REC>
__global__ void __launch_bounds__(GfCfg<BN, AMODE == 2, PAIR>::THREADS, 1)
gemm_int_f16_kernel(const __grid_constant__ GfMaps tm, const GemmIntF16Args a) {
  constexpr bool ASYM = AMODE != 0, A8 = AMODE == 2;
  using Cfg = GfCfg<BN, A8, PAIR>;
  constexpr int GF_EXP_STAGES = Cfg::EXP_STAGES, GF_RAW_STAGES = Cfg::RAW_STAGES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* raw_area = smem + GF_EXP_STAGES * Cfg::EXP_STAGE;
  uint8_t* stg_area = raw_area + GF_RAW_STAGES * Cfg::RAW_STAGE;       // 1024-byte aligned
  uint8_t* tab_area = stg_area + Cfg::STG_BYTES;
  uint8_t* row_area = tab_area + Cfg::TAB_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(row_area + Cfg::ROW_BYTES);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + Cfg::NBARS);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = PAIR ? cluster_ctarank() : 0u;            // 0 = leader (issues the pair's UMMAs)
  const uint32_t bar0 = smem_u32(bars);
  auto rawf_bar = [&](int s) { return bar0 + 8u * s; };
  auto rawe_bar = [&](int s) { return bar0 + 8u * (GF_RAW_STAGES + s); };
  auto expf_bar = [&](int s) { return bar0 + 8u * (2 * GF_RAW_STAGES + s); };
  auto expe_bar = [&](int s) { return bar0 + 8u * (2 * GF_RAW_STAGES + GF_EXP_STAGES + s); };
  auto expw_bar = [&](int s) { return bar0 + 8u * (2 * GF_RAW_STAGES + 2 * GF_EXP_STAGES + s); };   // weight tile landed
  auto accf_bar = [&](int b) { return bar0 + 8u * (2 * GF_RAW_STAGES + 3 * GF_EXP_STAGES + b); };
  auto acce_bar = [&](int b) { return bar0 + 8u * (2 * GF_RAW_STAGES + 3 * GF_EXP_STAGES + 2 + b); };
  auto rows_bar = [&](int b) { return bar0 + 8u * (2 * GF_RAW_STAGES + 3 * GF_EXP_STAGES + 4 + b); };   // a tile's 1 / rs

  constexpr int W_MMA = GF_EPI_WARPS, W_TMA = GF_EPI_WARPS + 1, W_TMB = GF_EPI_WARPS + 2, W_CONV = GF_EPI_WARPS + 4;
  if (threadIdx.x == 0) {
    for (int s = 0; s < GF_RAW_STAGES; ++s) { mbar_init(rawf_bar(s), 1); mbar_init(rawe_bar(s), Cfg::CONV_WARPS); }
    for (int s = 0; s < GF_EXP_STAGES; ++s) {
      // pairs: one barrier per stage, in the leader, counts the weight bytes and the converter warps of both CTAs
      mbar_init(expf_bar(s), PAIR ? 1 + 2 * Cfg::GROUP_WARPS : Cfg::GROUP_WARPS);
      mbar_init(expe_bar(s), 1);
      mbar_init(expw_bar(s), 1);
    }
    for (int b = 0; b < 2; ++b) { mbar_init(accf_bar(b), 1); mbar_init(acce_bar(b), (PAIR ? 2 : 1) * GF_EPI_WARPS); }
    for (int b = 0; b < Cfg::ROW_TILES; ++b) mbar_init(rows_bar(b), 4);
    abort_init(abort_flag, a.wait_limit_k, PAIR ? map_to_rank(bar0 + 8u * Cfg::NBARS + 4u, rank ^ 1) : 0u);
    fence_mbar_init();
    prefetch_tmap(&tm.xq);
    prefetch_tmap(&tm.wp);
  }
  if (warp == W_MMA) {
    if constexpr (PAIR) tmem_alloc_pair(smem_u32(tmem_slot), Cfg::TMEM_COLS);
    else tmem_alloc(smem_u32(tmem_slot), Cfg::TMEM_COLS);
  }
  tc_fence_before();
  __syncthreads();
  if constexpr (PAIR) cluster_sync_all();   // both CTAs' barriers exist before anything arrives on them remotely
  tc_fence_after();
  pdl_launch_dependents();
  pdl_wait();                       // the kernels that produced the codes, scales or records have completed
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t exp_base = smem_u32(smem);
  const uint32_t raw_base = smem_u32(raw_area);

  const int n_raw = a.n_chunks;                                    // chunks of codes in the raw stream
  const bool hc = a.half_chunks != 0;                              // two half-padded chunks per unit
  const int n_main = hc ? (a.n_chunks + 1) >> 1 : a.n_chunks;      // units of codes
  const int n_tail = (a.kt + 63) >> 6;
  constexpr int UNITS = Cfg::UNITS;
  const int s_main = (n_main + UNITS - 1) / UNITS, ns = s_main + (n_tail + UNITS - 1) / UNITS;    // operand stages
  auto units_of = [&](int st) { return UNITS == 1 ? 1 : min(2, st < s_main ? n_main - 2 * st : n_tail - 2 * (st - s_main)); };
  const int n_tiles_n = (int)((a.N + BN - 1) / BN);
  constexpr int TILE_M = PAIR ? 256 : 128;
  const int n_tiles_m = (int)((a.M + TILE_M - 1) / TILE_M);
  const int total_tiles = n_tiles_n * n_tiles_m;
  // Tile order: column tiles in groups of `a.raster` (n fastest inside a group, then m, then the next group), so the
  // tiles in flight at one time share a bounded set of weight columns and activation rows in L2.
  const int rast = a.raster > 0 && a.raster < n_tiles_n ? a.raster : n_tiles_n;
  auto tile_mn = [&](int t, int& tm_, int& tn_) {
    const int per_group = rast * n_tiles_m;
    const int grp = t / per_group, r = t - grp * per_group;
    const int width = min(rast, n_tiles_n - grp * rast);
    tm_ = r / width;
    tn_ = grp * rast + (r - tm_ * width);
  };
  const int first = PAIR ? (int)cluster_id_x() : (int)blockIdx.x, step = PAIR ? (int)cluster_count_x() : (int)gridDim.x;
  // Persistent CTA (pair): tiles first, first + step, ... with n fastest, so CTAs running at
  // the same time read the same activation rows through L2.  Rings and the accumulator counter run on
  // across tiles.  Operand stage q of the kernel-wide sequence (chunks and tail stages of all tiles)
  // lives in slot q % EXP_STAGES; its barrier phase is (q / EXP_STAGES) & 1.

  if (warp >= W_CONV) {
    reg_dealloc<Cfg::REGS_CONV>();
    // ------------------------------ converters ------------------------------------------------
    // Two groups take alternate operand stages (stage q goes to group q % GROUPS), so one group's barrier
    // waits, shared-memory latencies and fences overlap the other group's arithmetic.  A warp owns the 32
    // activation rows of its own TMEM lane quarter (warp index mod 4).
    const int cw = warp - W_CONV;
    constexpr int GW = Cfg::GROUP_WARPS;
    const int grp = cw / GW;
    const int quarter = warp & 3;
    const int rowA = quarter * 32 + lane;
    constexpr bool LATE = A8 && UNITS == 2;
    const uint32_t never = (uint32_t)a.half_chunks & 0x100u;      // half_chunks is 0 or 1
    GfRing<GF_RAW_STAGES> r;
    int q = 0;
    bool ok = true;
    auto exp_ready = [&](int es) {                          // this warp's rows of the stage are in tensor memory
      if (PAIR && rank != 0) mbar_arrive_cluster_relaxed(map_to_rank(expf_bar(es), 0));
      else mbar_arrive(expf_bar(es));
    };
    auto exp_slot = [](int qq) { return qq % Cfg::EXP_STAGES; };
    auto exp_phase = [](int qq) { return (uint32_t)((qq / Cfg::EXP_STAGES) & 1); };
    int tile_no = 0;
    for (int t = first; t < total_tiles && ok; t += step, ++tile_no) {
      float inv = 0.f;
      if constexpr (!REC) {
        const int rslot = tile_no % Cfg::ROW_TILES;
        if (!mbar_wait_hot_warp(rows_bar(rslot), (uint32_t)((tile_no / Cfg::ROW_TILES) & 1), abort_flag, a.status, ERR_WAIT_FULL)) { ok = false; break; }
        inv = gf_lds_f32(smem_u32(row_area) + (uint32_t)(rslot * 128 + rowA) * 4);
      }
      auto record = [&](uint32_t sraw, int j) {             // chunk j of a raw stage, this thread's row
        if constexpr (REC) return gf_lds64(sraw + Cfg::OFF_C + j * 128 * 8 + rowA * 8);
        const uint32_t at = sraw + (uint32_t)(j * 128 + rowA) * 2;
        const float s = __uint_as_float(gf_lds16(at + Cfg::OFF_C) << 16);
        if constexpr (ASYM) return chunk_record(s, __uint_as_float(gf_lds16(at + Cfg::OFF_Z) << 16), inv);
        const uint32_t m = half_twice(s * (inv * 16777216.f));       // s has 8 bits: exact, so 8 s / rs may be taken from it
        return make_uint2(m, hmul2_m8(m));
      };
      // Only once what was read has arrived in registers: an arrival overtakes shared-memory loads that still wait in their queue, behind
      // stores of the quantising epilogue for instance, and the next copy would overwrite what they read.  Either instructions
      // that use it have been issued, or the arrival's own address depends on it (`read`, a word of every load, under a mask that
      // is zero for reasons the compiler does not know).  A record made here comes of two loads where there are zero points, the
      // scale's (and 1 / rs) in its multiplier, the zero point's only in its addend.
      auto words_of = [](uint2 k) { return ASYM && !REC ? k.x ^ k.y : k.x; };
      auto release_raw = [&](uint32_t read = 0u) {
        __syncwarp();
        if (lane == 0) mbar_arrive(rawe_bar(r.s) + (read & never));
        r.next();
      };
      // A unit's values, in registers, go to tensor memory, the first of a stage as soon as the slot is free.  (The empty statement
      // keeps the expansion in front of the wait: the compiler would move it behind, onto the path between "slot free" and
      // "stage ready".)
      auto slot_free = [&](int qq, uint32_t (&y)[32]) {
#pragma unroll
        for (int i = 0; i < 32; ++i) asm volatile("" : "+r"(y[i]));
        if (!mbar_wait_hot_warp(expe_bar(exp_slot(qq)), exp_phase(qq) ^ 1, abort_flag, a.status, ERR_WAIT_EMPTY)) { q = qq; return false; }
        tc_fence_after();
        return true;
      };
      auto put = [&](int qq, int unit, uint32_t (&y)[32]) {
        tmem_st32(tmem_base + ((uint32_t)(quarter * 32) << 16) + Cfg::TMEM_A0 + exp_slot(qq) * Cfg::A_COLS + unit * 32, y);
      };
      auto stage_done = [&](int qq) {
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) exp_ready(exp_slot(qq));
      };
      for (int c = 0; c < n_raw && ok; c += GF_CPS) {
        if (!mbar_wait_hot_warp(rawf_bar(r.s), r.ph, abort_flag, a.status, ERR_WAIT_FULL)) { ok = false; break; }
        const uint32_t sraw = raw_base + r.s * Cfg::RAW_STAGE;
        const int nv = min(GF_CPS, n_raw - c);
        const int nu = hc ? (nv + 1) >> 1 : nv, nst = (nu + UNITS - 1) / UNITS;   // units and operand stages this raw stage feeds
        const int j = (grp ^ q) & 1, qq = q + j;               // this group's first stage of them, if there is one
        q += nst;
        if (j >= nst) { release_raw(); continue; }
        const int u0 = UNITS * j, u1 = UNITS == 2 ? u0 + 1 : u0 + 2;    // its units: of one stage, or of two stages
        const bool two = u1 < nu;
        uint32_t y[32];
        if (hc) {
          // half chunks: the first 32 slots of chunks 2 u and 2 u + 1, each with its own record, side by side
          constexpr int PC = A8 ? 2 : 1;
          auto fetch = [&](int ch, uint4 (&p)[PC]) {           // (slots past the last chunk: codes 0 under a record of zeros)
#pragma unroll
            for (int u = 0; u < PC; ++u)
              p[u] = ch >= nv ? make_uint4(0u, 0u, 0u, 0u)
                     : A8     ? gf_lds128(sraw + (ch >> 1) * (128 * 128) + rowA * 128 + ((((ch & 1) * 4 + u) ^ (rowA & 7)) << 4))
                              : gf_lds128(sraw + rowA * 128 + (((2 * ch) ^ (rowA & 7)) << 4));
            return ch < nv ? record(sraw, ch) : make_uint2(0u, 0u);
          };
          auto expand = [&](const uint4 (&p)[PC], uint2 k, uint32_t* d) {
            if constexpr (A8) expand_bytes32(p, k, d);
            else expand_nibbles32<ASYM>(p[0], k, d);
          };
          uint4 p0[PC], p1[PC], p2[PC], p3[PC];
          const uint2 k0 = fetch(2 * u0, p0), k1 = fetch(2 * u0 + 1, p1);
          uint2 k2, k3;
          auto fetch1 = [&]() {
            if constexpr (UNITS == 2) { k2 = fetch(2, p2), k3 = fetch(3, p3); }
          };
          if constexpr (!LATE) {
            fetch1();
            uint32_t read = words_of(k0) ^ words_of(k1);
#pragma unroll
            for (int i = 0; i < PC; ++i) read ^= p0[i].x ^ p1[i].x;
            if constexpr (UNITS == 2) {
              read ^= words_of(k2) ^ words_of(k3);
#pragma unroll
              for (int i = 0; i < PC; ++i) read ^= p2[i].x ^ p3[i].x;
            }
            release_raw(read);
          }
          expand(p0, k0, y);
          expand(p1, k1, y + 16);
          if (!slot_free(qq, y)) { ok = false; break; }
          put(qq, 0, y);
          if (UNITS == 2 && two) {
            if constexpr (LATE) fetch1();
            expand(p2, k2, y);
            expand(p3, k3, y + 16);
            put(qq, 1, y);
          }
          if constexpr (LATE) release_raw();
          stage_done(qq);
          continue;
        }
        // 4-bit codes: two 16-byte pieces of the swizzled 128-byte raw row; 8-bit codes: 64 bytes of this row = four pieces of box
        // u0 >> 1.  Both units' codes are read before the first is expanded; 8-bit codes, twice the registers, one after the
        // other in stages of two units.
        constexpr int PC = A8 ? 4 : 2;
        auto fetch = [&](int u, uint4 (&p)[PC]) {
#pragma unroll
          for (int i = 0; i < PC; ++i)
            p[i] = A8 ? gf_lds128(sraw + (u >> 1) * (128 * 128) + rowA * 128 + ((((u & 1) * 4 + i) ^ (rowA & 7)) << 4))
                      : gf_lds128(sraw + rowA * 128 + (((2 * u + i) ^ (rowA & 7)) << 4));
        };
        auto expand = [&](const uint4 (&p)[PC], uint2 k) {
          if constexpr (A8) {
            expand_bytes32(p, k, y);
            expand_bytes32(p + 2, k, y + 16);
          } else {
            expand_nibbles32<ASYM>(p[0], k, y);
            expand_nibbles32<ASYM>(p[1], k, y + 16);
          }
        };
        uint4 p0[PC], p1[PC];
        const uint2 k0 = record(sraw, u0);
        fetch(u0, p0);
        uint2 k1 = make_uint2(0u, 0u);
        auto fetch1 = [&]() {
          if (two) {
            k1 = record(sraw, u1);
            fetch(u1, p1);
          }
        };
        if constexpr (!LATE) {
          fetch1();
          uint32_t read = words_of(k0) ^ words_of(k1);
#pragma unroll
          for (int i = 0; i < PC; ++i) read ^= two ? p0[i].x ^ p1[i].x : p0[i].x;
          release_raw(read);
        }
        expand(p0, k0);
        if (!slot_free(qq, y)) { ok = false; break; }
        put(qq, 0, y);
        if constexpr (UNITS == 2) {
          if constexpr (LATE) fetch1();
          if (two) {
            expand(p1, k1);
            put(qq, 1, y);
          }
          if constexpr (LATE) release_raw();
          stage_done(qq);
        } else {
          stage_done(qq);
          if (two) {
            expand(p1, k1);
            if (!slot_free(qq + 2, y)) { ok = false; break; }
            put(qq + 2, 0, y);
            stage_done(qq + 2);
          }
        }
      }
      // tail: the activations' bf16 tiles arrive in the raw ring, a unit each; their rows, divided by rs (exact; with records the
      // folding kernel has done that), go to TMEM like expanded chunks
      for (int st = 0; st < n_tail && ok; st += UNITS) {
        const int qq = q++;
        const bool mine = ((qq ^ grp) & 1) == 0;
        for (int u = 0; u < min(UNITS, n_tail - st); ++u) {
          if (!mbar_wait_hot_warp(rawf_bar(r.s), r.ph, abort_flag, a.status, ERR_WAIT_FULL)) { q = qq; ok = false; break; }
          if (!mine) { release_raw(); continue; }
          const uint32_t rb = raw_base + r.s * Cfg::RAW_STAGE + rowA * 128;
          uint32_t y[32];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const uint4 v = gf_lds128(rb + (uint32_t)((i ^ (rowA & 7)) << 4));
            y[4 * i] = v.x; y[4 * i + 1] = v.y; y[4 * i + 2] = v.z; y[4 * i + 3] = v.w;
          }
          if constexpr (!REC) {
            const __nv_bfloat162 inv2 = __float2bfloat162_rn(inv);
#pragma unroll
            for (int i = 0; i < 32; ++i) {
              const __nv_bfloat162 h = __hmul2(*reinterpret_cast<const __nv_bfloat162*>(&y[i]), inv2);
              y[i] = *reinterpret_cast<const uint32_t*>(&h);
            }
          }
          if (u == 0 && !slot_free(qq, y)) { ok = false; break; }
          put(qq, u, y);
          release_raw();
        }
        if (!ok) break;
        if (mine) stage_done(qq);
      }
    }
    if (PAIR && lane == 0) {
      // for the teardown: one past the last stage this warp has arrived for.  Not q: a group walks past the other group's
      // stages without waiting for their slots, and a stage counted before its slot is free would share its barrier's phase
      // with the slot's last one.
      while (q > 0 && (q - 1) % Cfg::GROUPS != grp) --q;
      abort_flag[AB_WARP + cw] = q;
    }
  } else if (warp >= W_MMA) {
  reg_dealloc<Cfg::REGS_PROD>();
  if (warp == W_TMA) {
    // ------------------------------ TMA producer ---------------------------------------------
    if (lane == 0) {
      GfRing<GF_RAW_STAGES> r;
      int issued = 0;
      bool ok = true;
      for (int t = first; t < total_tiles && ok; t += step) {
        int tm_, tn_;
        tile_mn(t, tm_, tn_);
        const int m0 = tm_ * TILE_M + (int)rank * 128;
        // the second half of a pair's last tile may lie past the end: codes arrive as zero fill, and the records (bulk
        // copies know no bounds) are those of the last row block; none of its rows is ever stored
        const int64_t mrec = REC ? min((int64_t)m0, a.ld_rec - 128) : (int64_t)m0;
        for (int c = 0; c < n_raw; c += GF_CPS) {
          if (!mbar_wait_hot(rawe_bar(r.s), r.ph ^ 1, abort_flag, a.status, ERR_WAIT_EMPTY)) { ok = false; break; }
          const uint32_t sb = raw_base + r.s * Cfg::RAW_STAGE;
          const uint32_t bar = rawf_bar(r.s);
          const int nv = min(GF_CPS, n_raw - c);
          // 8-bit codes: the second 128-byte box is issued only when it holds a chunk (a box that lies
          // wholly outside the tensor is never requested; its bytes are not part of the count either)
          const bool second_box = A8 && nv > 2;
          // boxes of scales are counted whole, zero fill included
          mbar_expect_tx(bar, (uint32_t)(Cfg::RAW_A - ((A8 && !second_box) ? 128 * 128 : 0) +
                                         (REC ? nv * 128 * 8 : (ASYM ? 2 : 1) * GF_CPS * 128 * 2)));
          if constexpr (!REC) {
            tma_load_2d(sb + Cfg::OFF_C, &tm.xs, bar, m0, c);
            if constexpr (ASYM) tma_load_2d(sb + Cfg::OFF_Z, &tm.xz, bar, m0, c);
          }
          if constexpr (A8) {
            tma_load_2d(sb, &tm.xq, bar, c * 64, m0);
            if (second_box) tma_load_2d(sb + 128 * 128, &tm.xq, bar, c * 64 + 128, m0);
          } else {
            tma_load_2d(sb, &tm.xq, bar, c * 32, m0);
          }
          if constexpr (REC)
            for (int j = 0; j < nv; ++j)
              bulk_load(sb + Cfg::OFF_C + j * 128 * 8, a.a_const + ((int64_t)(c + j) * a.ld_rec + mrec), 128 * 8, bar);
          ++issued;
          r.next();
        }
        // tail: the activations' bf16 tile travels through the raw ring like a chunk (its rows go on to TMEM)
        for (int st = 0; st < n_tail && ok; ++st) {
          if (!mbar_wait_hot(rawe_bar(r.s), r.ph ^ 1, abort_flag, a.status, ERR_WAIT_EMPTY)) { ok = false; break; }
          const uint32_t bar = rawf_bar(r.s);
          mbar_expect_tx(bar, 128u * 128u);                    // one 128 x 64 bf16 tile
          tma_load_2d(raw_base + r.s * Cfg::RAW_STAGE, &tm.xt, bar, st * 64, m0);
          ++issued;
          r.next();
        }
      }
      abort_flag[AB_ISSUED] = issued;
    }
  } else if (warp == W_TMB) {
    // ------------------------------ weight-tile producer ---------------------------------------
    // Operand stage q's weight tile goes straight into slot q % EXP_STAGES as soon as the slot is free.  A whole warp waits and its
    // elected lane issues, as in the issuer: in one lane this loop took 450 cycles a stage, more than the four UMMAs of a 128-wide
    // tile, and was what such launches waited for.
    GfRing<GF_EXP_STAGES> e;
    int issued = 0;
    bool ok = true;
    const uint32_t full_lead = PAIR ? map_to_rank(expf_bar(0), 0) : 0u;   // the bytes of both halves are counted in the leader
    for (int t = first; t < total_tiles && ok; t += step) {
      int tm_, tn_;
      tile_mn(t, tm_, tn_);
      const int row_b = tn_ * BN + (int)rank * Cfg::BN_OWN;               // of a pair, this CTA's half of the weight rows
      for (int st = 0; st < ns; ++st) {
        if (!mbar_wait_hot_warp(expe_bar(e.s), e.ph ^ 1, abort_flag, a.status, ERR_WAIT_EMPTY)) { ok = false; break; }
        if (elect_one()) {
          const uint32_t dst = exp_base + e.s * Cfg::EXP_STAGE;
          const int nu = units_of(st), x = (st < s_main ? st : st - s_main) * (UNITS * 64);
          const CUtensorMap* const map = st < s_main ? &tm.wp : &tm.wt;
          if constexpr (PAIR) {
            const uint32_t bar = full_lead + 8u * e.s;
            if (rank == 0) mbar_expect_tx(expf_bar(e.s), (uint32_t)(2 * nu * Cfg::B_EXP));
            tma_load_2d_pair(dst, map, bar, x, row_b);
            if (nu == 2) tma_load_2d_pair(dst + Cfg::B_EXP, map, bar, x + 64, row_b);
          } else {
            const uint32_t bar = expw_bar(e.s);
            mbar_expect_tx(bar, (uint32_t)(nu * Cfg::B_EXP));  // boxes are counted whole, zero fill included
            tma_load_2d(dst, map, bar, x, row_b);
            if (nu == 2) tma_load_2d(dst + Cfg::B_EXP, map, bar, x + 64, row_b);
          }
        }
        __syncwarp();
        ++issued;
        e.next();
      }
    }
    if (lane == 0) abort_flag[AB_ISSUED2] = issued;
  } else if (warp == W_MMA) {
    // ------------------------------ UMMA issuer ----------------------------------------------
    if (rank == 0) {
      const uint32_t idesc_h = idesc_dense(ACC_F32, FMT_F16, FMT_F16, TILE_M, BN);
      const uint32_t idesc_bf = idesc_dense(ACC_F32, FMT_BF16, FMT_BF16, TILE_M, BN);
      int use = 0, stages = 0;
      bool ok = true, ready = false;                               // ready: the next stage's barriers are known to be complete
      // loop-invariant pieces of the per-stage operands: barrier addresses are 8 bytes per slot apart, the weight
      // descriptor's low word holds the slot address >> 4, the activation slots are 32 tensor-memory columns apart
      int es = 0;
      uint32_t ph = 0;
      const uint32_t expw0 = expw_bar(0);
      constexpr uint32_t kFullOff = 8u * 2 * GF_EXP_STAGES;      // expw_bar(s) - expf_bar(s)
      constexpr uint32_t kEmptyOff = 8u * GF_EXP_STAGES;         // expw_bar(s) - expe_bar(s)
      const uint64_t bdesc0 = smem_desc_sw128(exp_base);
      const uint32_t bdesc_lo0 = (uint32_t)bdesc0, bdesc_hi = (uint32_t)(bdesc0 >> 32);
      constexpr uint32_t kDescStep = Cfg::EXP_STAGE >> 4;
      const uint32_t a_tmem0 = tmem_base + Cfg::TMEM_A0;
      for (int t = first; t < total_tiles && ok; t += step) {
        const int buf = Cfg::NACC == 2 ? (use & 1) : 0;
        const uint32_t acc_ph = (uint32_t)(Cfg::NACC == 2 ? (use >> 1) & 1 : use & 1);
        if (!mbar_wait_hot_warp(acce_bar(buf), acc_ph ^ 1, abort_flag, a.status, ERR_WAIT_ACC_EMPTY)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d = tmem_base + buf * BN;
        // What this warp does between UMMAs is time the pipe idles, and it has few of them queued: so the next stage's barriers
        // are tested within this one's block (umma_f16_ts_stage): waiting, issuing and looping took 150 + 180 + 100 cycles.
        for (int st = 0; st < ns; ++st) {
          const uint32_t w = expw0 + 8u * es;                      // expf / expe lie at fixed offsets from expw
          // pairs: one barrier per stage covers both operands in both CTAs
          if (!ready && (PAIR ? !mbar_wait_hot_warp(w - kFullOff, ph, abort_flag, a.status, ERR_WAIT_FULL)
                              : !mbar_wait2_hot_warp(w, ph, w - kFullOff, ph, abort_flag, a.status, ERR_WAIT_FULL))) { ok = false; break; }
          tc_fence_after();
          uint32_t a_t = a_tmem0 + (uint32_t)Cfg::A_COLS * es, b_lo = bdesc_lo0 + kDescStep * es;
          if (++es == GF_EXP_STAGES) { es = 0; ph ^= 1u; }
          const uint32_t wn = expw0 + 8u * es;
          uint32_t next = 0u;
          if (elect_one()) {
            const uint32_t idesc = st < s_main ? idesc_h : idesc_bf;
            uint32_t acc = st > 0 ? 1u : 0u;
            if (units_of(st) == 2) {
              if constexpr (PAIR) umma_f16_ts_x4_pair(d, a_t, b_lo, bdesc_hi, idesc, acc);
              else umma_f16_ts_x4(d, a_t, b_lo, bdesc_hi, idesc, acc);
              a_t += 32u;
              b_lo += Cfg::B_EXP >> 4;
              acc = 1u;
            }
            if constexpr (PAIR) next = umma_f16_ts_stage_pair(d, a_t, b_lo, bdesc_hi, idesc, acc, w - kEmptyOff, wn - kFullOff, ph);
            else next = umma_f16_ts_stage(d, a_t, b_lo, bdesc_hi, idesc, acc, w - kEmptyOff, wn, ph, wn - kFullOff);
          }
          ready = __any_sync(0xffffffffu, next != 0u);
          ++stages;
        }
        if (!ok) break;
        if (elect_one()) {
          if constexpr (PAIR) umma_commit_pair_both(accf_bar(buf));
          else umma_commit(accf_bar(buf));
        }
        __syncwarp();
        ++use;
      }
      if (lane == 0) {
        abort_flag[AB_UMMA] = stages;
        abort_flag[AB_ACC] = use;
      }
    }
  }
  } else {
    reg_alloc<Cfg::REGS_EPI>();
    // ------------------------------ epilogue: 8 warps -----------------------------------------
    // warp w: TMEM lane quarter w & 3 (32 rows), half of the columns.  Two steps: the warp's share of the accumulator is
    // read, scaled by rs[m] * cs[n], offset by the bias and rounded to bf16 pairs in registers, and the accumulator is
    // handed back; only then come the activation, the quantiser and the stores.  A 256-wide tile has one accumulator, so
    // everything before the hand-back is time its UMMAs wait: 6200 cycles of a 16900-cycle tile at K = 1152 with the
    // per-column factors loaded from global memory between the reads and activation and stores inside, 2900 with them
    // outside and the factors from shared memory, 1700 with each 16-column piece's loads in flight while the piece before it
    // is worked on (which takes the registers).  The factors come from a table of the warp's own, filled while the UMMAs of
    // the tile still run, as bf16 pairs: cs is a power of two.
    // Stores: bf16 -> the warp's 32 x 32 staging patch in shared memory (64-byte rows, 64-byte swizzle: conflict-free)
    // -> one TMA store, which clips the patch at the edges of y.  A row-per-thread store straight to global memory would
    // put 32 separate 16-byte segments per instruction through the load/store unit that the converter warps depend on.
    const int q = warp & 3, ch = warp >> 2;
    const int trow = q * 32 + lane;
    constexpr int CW = BN / 2;
    const uint32_t stg = smem_u32(stg_area) + warp * 2048;
    const uint32_t stg_row = stg + lane * 64;
    const int stg_sw = (lane >> 1) & 3;
    const uint32_t tab = smem_u32(tab_area) + warp * Cfg::TAB_WARP;
    auto acc_release = [&](int b) {
      if (PAIR && rank != 0) mbar_arrive_cluster_relaxed(map_to_rank(acce_bar(b), 0));
      else mbar_arrive(acce_bar(b));
    };
    const bool qout = BN != 192 && a.q_codes != nullptr;
    auto put_patch = [&](const uint32_t* w16, int col, int row) {     // 32 columns of the warp's 32 rows -> y
      if (lane == 0) bulk_wait_read0();              // the previous patch has left the staging buffer
      __syncwarp();
#pragma unroll
      for (int i = 0; i < 4; ++i)
        gf_sts128(stg_row + (uint32_t)((i ^ stg_sw) << 4), w16[4 * i], w16[4 * i + 1], w16[4 * i + 2], w16[4 * i + 3]);
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        tma_store_2d(&tm.y, stg, col, row);
        bulk_commit_group();
      }
    };
    auto gelu_pairs = [&](uint32_t* w16) {
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w16[e]));
        const __nv_bfloat162 h = __floats2bfloat162_rn(gelu_tanh_bf16(f.x), gelu_tanh_bf16(f.y));
        w16[e] = *reinterpret_cast<const uint32_t*>(&h);
      }
    };
    // Without records a row's power of two comes from its largest chunk scale.  These warps have time while a tile's UMMAs run, so
    // they read the scales one tile ahead and leave 1 / rs for the converters in the tile's slot of a table (see ROW_TILES).  The
    // first tile waits for it: 16-byte loads, eight rows of eight chunks each per warp instruction, 96 chunks in flight.  With
    // 2-byte loads of a row per lane, 24 in flight, every call began with a chain of them: 512 x 12288 x 3072 79.5 -> 63.9 us, 4096 x
    // 4608 x 1152 54.9 -> 50.0, 256 x 1152 x 1152 11.2 -> 10.2.
    int rows_no = 0;
    auto row_powers = [&](int t) {
      int tm_, tn_;
      tile_mn(t, tm_, tn_);
      // this lane: rows r8 .. r8 + 7 of the warp's 32, chunks lane / 4 + 8 i (scales are 16-byte aligned, ldm a multiple of eight)
      const int64_t r8 = (int64_t)tm_ * TILE_M + (int)rank * 128 + q * 32 + (lane & 3) * 8;
      const __nv_bfloat16* const s8 = a.xs + r8;
      uint32_t m[4] = {0u, 0u, 0u, 0u};
#pragma unroll 1
      for (int c0 = lane >> 2; c0 < n_raw; c0 += 96) {
        uint4 v[12];
#pragma unroll
        for (int i = 0; i < 12; ++i) {
          const int c = c0 + 8 * i;
          v[i] = c < n_raw && r8 < a.ldm ? __ldg(reinterpret_cast<const uint4*>(s8 + (int64_t)c * a.ldm)) : make_uint4(0u, 0u, 0u, 0u);
        }
#pragma unroll
        for (int i = 0; i < 12; ++i) {
          m[0] = abs_max_bf16x2(m[0], v[i].x);
          m[1] = abs_max_bf16x2(m[1], v[i].y);
          m[2] = abs_max_bf16x2(m[2], v[i].z);
          m[3] = abs_max_bf16x2(m[3], v[i].w);
        }
      }
      __syncwarp();
#pragma unroll
      for (int o = 4; o < 32; o <<= 1)
#pragma unroll
        for (int i = 0; i < 4; ++i) m[i] = abs_max_bf16x2(m[i], __shfl_xor_sync(0xffffffffu, m[i], o));
      // row `lane` of the 32: half lane % 2 of word (lane / 2) % 4 of the octet lane / 8
      uint32_t mine = 0u;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t v = __shfl_sync(0xffffffffu, m[i], lane >> 3);
        if (((lane >> 1) & 3) == i) mine = v;
      }
      const float smax = __uint_as_float((lane & 1) ? mine & 0xFFFF0000u : mine << 16);
      float rs;
      const float inv = row_inverse_power(smax, rs);
      if (ch == 0) {
        const int rslot = rows_no % Cfg::ROW_TILES;
        gf_sts_f32(smem_u32(row_area) + (uint32_t)(rslot * 128 + trow) * 4, inv);
        __syncwarp();
        if (lane == 0) mbar_arrive(rows_bar(rslot));
      }
      ++rows_no;
      return rs;
    };
    int use = 0;
    bool ok = true;
    float rs_next = 0.f;
    if constexpr (!REC)
      if (first < total_tiles) rs_next = row_powers(first);
    for (int t = first; t < total_tiles && ok; t += step) {
      int tm_, tn_;
      tile_mn(t, tm_, tn_);
      const int m0 = tm_ * TILE_M + (int)rank * 128, n0 = tn_ * BN;
      const int64_t row = (int64_t)m0 + trow;
      const float rs = !REC ? rs_next : (row < a.M) ? __ldg(a.rs + row) : 0.f;
      __syncwarp();                                  // every lane has read the previous tile's table
      for (int i = lane; i < Cfg::PIECES * 8; i += 32) { // one column pair each
        const int64_t col = (int64_t)n0 + ch * CW + 2 * i;
        uint32_t cp = 0u, bp = 0u;
        if (col < a.N) {
          const float2 c = __ldg(reinterpret_cast<const float2*>(a.cs + col));
          cp = __byte_perm(__float_as_uint(c.x), __float_as_uint(c.y), 0x7632);      // powers of two: exact in bf16
          if (a.bias) bp = __ldg(reinterpret_cast<const uint32_t*>(a.bias + col));
        }
        gf_sts64(tab + i * 8, cp, bp);
      }
      if constexpr (!REC)
        if (t + step < total_tiles) rs_next = row_powers(t + step);
      const int buf = Cfg::NACC == 2 ? (use & 1) : 0;
      const uint32_t acc_ph = (uint32_t)(Cfg::NACC == 2 ? (use >> 1) & 1 : use & 1);
      if (!mbar_wait_warp(accf_bar(buf), acc_ph, abort_flag, a.status, ERR_WAIT_ACC_FULL)) { ok = false; break; }
      tc_fence_after();
      ++use;
      const uint32_t tl = tmem_base + ((uint32_t)(q * 32) << 16) + buf * BN + ch * CW;
      uint32_t w[Cfg::PIECES * 8];                    // the output before activation, bf16 pairs
      uint32_t v[2][16];
      uint4 f[2][4];
      auto fetch = [&](int c) {                       // a piece's accumulators and factors
        tmem_ld16(tl + c * 16, v[c & 1]);
#pragma unroll
        for (int e = 0; e < 4; ++e) f[c & 1][e] = gf_lds128(tab + (c * 4 + e) * 16);
      };
      fetch(0);
#pragma unroll
      for (int c = 0; c < Cfg::PIECES; ++c) {
        tmem_wait_ld16(v[c & 1]);
        if (c + 1 < Cfg::PIECES) fetch(c + 1);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const uint4 k = f[c & 1][e];
          w[8 * c + 2 * e] = scale_pair(v[c & 1][4 * e], v[c & 1][4 * e + 1], rs, k.x, k.y);
          w[8 * c + 2 * e + 1] = scale_pair(v[c & 1][4 * e + 2], v[c & 1][4 * e + 3], rs, k.z, k.w);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) acc_release(buf);                // the accumulator is out of TMEM
      if (!qout) {
#pragma unroll
        for (int g = 0; g < CW / 32; ++g) {
          const int64_t col0 = (int64_t)n0 + ch * CW + g * 32;
          if (col0 < a.N) {                            // warp-uniform: otherwise nothing of this patch lies inside y
            if (a.act == 1) gelu_pairs(w + 16 * g);
            put_patch(w + 16 * g, (int)col0, m0 + q * 32);
          }
        }
        continue;
      }
      // ---- quantise-out: every 64 columns of the tile are one group of the following layer ----
#pragma unroll
      for (int k = 0; k < Cfg::PIECES / 4; ++k) {
        const int64_t col0 = (int64_t)n0 + ch * CW + k * 64;
        if (col0 + 64 > a.N) break;                   // padding of the last tile (N is a multiple of 64 here)
        uint32_t* wk = w + 32 * k;                    // the activated output: what the next quantiser sees
        if (a.act == 1) { gelu_pairs(wk); gelu_pairs(wk + 16); }
        if (a.y) {                                    // the bf16 tensor as well, when the caller wants it
          put_patch(wk, (int)col0, m0 + q * 32);
          put_patch(wk + 16, (int)col0 + 32, m0 + q * 32);
        }
        if (row >= a.M) continue;
        if (col0 >= a.q_len) {                        // the following layer's 16-bit channels
          uint4* t4 = reinterpret_cast<uint4*>(a.q_tail + row * a.q_tail_pitch + (col0 - a.q_len));
#pragma unroll
          for (int i = 0; i < 8; ++i) t4[i] = make_uint4(wk[4 * i], wk[4 * i + 1], wk[4 * i + 2], wk[4 * i + 3]);
          continue;
        }
        const int chunk = (int)(col0 >> 6);
        uint4* dst = reinterpret_cast<uint4*>(a.q_codes + row * a.q_row_bytes + (int64_t)chunk * 32);
        GroupParams p;
        if (a.q_mode == DIROTQ_INT4_SYM) {
          const float amax = fmaxf(fmaxf(amax_bf16x16(wk), amax_bf16x16(wk + 8)), fmaxf(amax_bf16x16(wk + 16), amax_bf16x16(wk + 24)));
          p = int_sym_params<true>(amax, -amax, a.q_clip, 7.f);
          const float rcp = __frcp_rn(p.scale);
          dst[0] = int_sym_planar32_packed(wk, rcp, a.q_clip < 1.f);
          dst[1] = int_sym_planar32_packed(wk + 16, rcp, a.q_clip < 1.f);
        } else {
          float mx = -INFINITY, mn = INFINITY;
          minmax_bf16x16(wk, mx, mn);
          minmax_bf16x16(wk + 8, mx, mn);
          minmax_bf16x16(wk + 16, mx, mn);
          minmax_bf16x16(wk + 24, mx, mn);
          p = int_asym_params<true>(mx, mn, a.q_clip, 15.f);
          const float rcp = __frcp_rn(p.scale);
          const bool packs = int_asym_packs(mx, mn, rcp, p.zero);
          dst[0] = int_asym_planar32(wk, p.scale, rcp, p.zero, packs);
          dst[1] = int_asym_planar32(wk + 16, p.scale, rcp, p.zero, packs);
          a.q_zeros[(int64_t)chunk * a.q_ldm + row] = __float2bfloat16_rn(p.zero);
        }
        a.q_scales[(int64_t)chunk * a.q_ldm + row] = __float2bfloat16_rn(p.scale);
      }
    }
    if (lane == 0) bulk_wait_all0();                   // the output is in global memory before the CTA retires
  }
  tc_fence_before();
  __syncthreads();
  if constexpr (PAIR) cluster_sync_all();   // neither CTA retires while the other may still read its shared memory
  const int end_warp = (int)(tid_anew() >> 5);
  uint8_t* const end_bars = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(anew(smem_raw)) + 1023) & ~uintptr_t(1023)) +
                            GF_EXP_STAGES * Cfg::EXP_STAGE + GF_RAW_STAGES * Cfg::RAW_STAGE + Cfg::STG_BYTES + Cfg::TAB_BYTES + Cfg::ROW_BYTES;
  volatile int* const ab = reinterpret_cast<volatile int*>(end_bars + 8 * Cfg::NBARS) + 1;
  if (ab[AB_FLAG]) {                // a wait ran out (in both CTAs of a pair the flag is up)
    regs_even<Cfg::REGS_LAUNCH>(end_warp < GF_EPI_WARPS);
    // bytes that each CTA of a pair fetches for stage q of the kernel-wide sequence
    auto half_of = [&](int q) {
      constexpr int U = Cfg::UNITS;
      const int nm = a.half_chunks ? (a.n_chunks + 1) >> 1 : a.n_chunks, nt = (a.kt + 63) >> 6, sm = (nm + U - 1) / U, st = q % (sm + (nt + U - 1) / U);
      return (uint32_t)(min(U, st < sm ? nm - U * st : nt - U * (st - sm)) * Cfg::B_EXP);
    };
    gf_teardown<BN, A8, PAIR>(end_bars, half_of, a.status);
  }
  if (end_warp == W_MMA) {
    __syncwarp();
    tc_fence_after();
    const uint32_t tmem = *(reinterpret_cast<volatile uint32_t*>(end_bars + 8 * Cfg::NBARS));
    if constexpr (PAIR) tmem_dealloc_pair(tmem, Cfg::TMEM_COLS);
    else tmem_dealloc(tmem, Cfg::TMEM_COLS);
  }
}

// ---------------------------------------------------------------------------------------------------
// Scale preparation, per row (activations: token; weights: output channel): the largest
// chunk scale picks the row's power of two; every chunk scale becomes one 8-byte record
// { (s * 2^24 / rs) twice, -(z * s / rs) twice } of fp16 pairs, ready to be used as packed-FMA operands; the row's 16-bit tail is divided by rs (exact) into its own buffer.
// ---------------------------------------------------------------------------------------------------
template <typename ST> __device__ __forceinline__ float scale_to_float(ST v);
template <> __device__ __forceinline__ float scale_to_float<float>(float v) { return v; }
template <> __device__ __forceinline__ float scale_to_float<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

// Block = ROWS rows x 256 / ROWS chunk phases (thread tid: row tid % ROWS, chunks c = tid / ROWS (mod 256 / ROWS)).
// What this kernel takes is latency: two dependent passes over a few hundred bytes per thread.  So a thread's scales and zero
// points are loaded at once, ahead of the maximum, and kept; and calls of few rows get 16-row blocks (see fold_small_blocks).
template <typename ST, int ROWS>
__device__ __forceinline__ void fold_scales_block(int block, const ST* __restrict__ s, const __nv_bfloat16* __restrict__ z,
                                                  int n_chunks, int64_t rows, int64_t ld_in, uint2* __restrict__ rec,
                                                  int64_t ld_rec, float* __restrict__ rs, const __nv_bfloat16* __restrict__ tail,
                                                  __nv_bfloat16* __restrict__ tail_out, int kt_pitch) {
  constexpr int P = 256 / ROWS;
  __shared__ float part_max[P][ROWS];
  __shared__ float inv_s[ROWS];
  const int lr = threadIdx.x % ROWS, part = threadIdx.x / ROWS;
  const int64_t r0 = (int64_t)block * ROWS;
  const int64_t r = r0 + lr;
  // the tail tile's loads go out first: they do not depend on the scales
  const int units = tail ? kt_pitch / 8 : 0;             // 16-byte units per row
  constexpr int TAIL_IT = 4;
  uint4 tv[TAIL_IT];
  int n_it = 0;
  if (tail) {
#pragma unroll
    for (int it = 0; it < TAIL_IT; ++it) {
      const int i = threadIdx.x + it * 256;
      const int rr = i / units;
      if (i < ROWS * units && r0 + rr < rows) {
        tv[it] = __ldg(reinterpret_cast<const uint4*>(tail + (r0 + rr) * kt_pitch) + (i % units));
        n_it = it + 1;
      }
    }
  }
  constexpr int KEEP = 5;
  float sv[KEEP], zv[KEEP];
#pragma unroll
  for (int k = 0; k < KEEP; ++k) {
    const int c = part + k * P;
    const bool in = r < rows && c < n_chunks;
    sv[k] = in ? scale_to_float<ST>(s[(int64_t)c * ld_in + r]) : 0.f;
    zv[k] = in && z ? __bfloat162float(z[(int64_t)c * ld_in + r]) : 8.f;
  }
  float smax = 0.f;
#pragma unroll
  for (int k = 0; k < KEEP; ++k) smax = fmaxf(smax, fabsf(sv[k]));
  if (r < rows)
    for (int c = part + KEEP * P; c < n_chunks; c += P) smax = fmaxf(smax, fabsf(scale_to_float<ST>(s[(int64_t)c * ld_in + r])));
  part_max[part][lr] = smax;
  __syncthreads();
#pragma unroll
  for (int k = 0; k < P; ++k) smax = fmaxf(smax, part_max[k][lr]);
  float row_pow;
  const float inv = row_inverse_power(smax, row_pow);
  if (part == 0) {
    inv_s[lr] = inv;
    if (r < rows) rs[r] = row_pow;
  }
  auto record = [&](int c, float sc, float zp) { rec[(int64_t)c * ld_rec + r] = chunk_record(sc, zp, inv); };
  if (r < rows) {
#pragma unroll
    for (int k = 0; k < KEEP; ++k)
      if (part + k * P < n_chunks) record(part + k * P, sv[k], zv[k]);
    for (int c = part + KEEP * P; c < n_chunks; c += P)
      record(c, scale_to_float<ST>(s[(int64_t)c * ld_in + r]), z ? __bfloat162float(z[(int64_t)c * ld_in + r]) : 8.f);
  } else if (r < ld_rec) {
    for (int c = part; c < n_chunks; c += P) rec[(int64_t)c * ld_rec + r] = make_uint2(0u, 0u);
  }
  if (tail == nullptr) return;
  __syncthreads();
  auto scale_store = [&](int i, uint4 v) {
    const int rr = i / units, u = i % units;
    const float f = inv_s[rr];
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&v);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float2 x = __bfloat1622float2(h[j]);
      h[j] = __floats2bfloat162_rn(x.x * f, x.y * f);
    }
    *(reinterpret_cast<uint4*>(tail_out + (r0 + rr) * kt_pitch) + u) = v;
  };
#pragma unroll
  for (int it = 0; it < TAIL_IT; ++it)
    if (it < n_it) scale_store(threadIdx.x + it * 256, tv[it]);
  // wide tails (more than 4 x 256 units per block): the rest, load and store in turn
  for (int i = threadIdx.x + TAIL_IT * 256; i < ROWS * units; i += 256) {
    const int rr = i / units;
    if (r0 + rr >= rows) break;
    scale_store(i, __ldg(reinterpret_cast<const uint4*>(tail + (r0 + rr) * kt_pitch) + (i % units)));
  }
}

template <typename ST, int ROWS>
__global__ void __launch_bounds__(256)
fold_scales_kernel(const ST* __restrict__ s, const __nv_bfloat16* __restrict__ z, int n_chunks, int64_t rows, int64_t ld_in,
                   uint2* __restrict__ rec, int64_t ld_rec, float* __restrict__ rs,
                   const __nv_bfloat16* __restrict__ tail, __nv_bfloat16* __restrict__ tail_out, int kt_pitch) {
  pdl_launch_dependents();
  pdl_wait();
  fold_scales_block<ST, ROWS>((int)blockIdx.x, s, z, n_chunks, rows, ld_in, rec, ld_rec, rs, tail, tail_out, kt_pitch);
}

// Weight pre-pass: codes + records -> the fp16 panel [N, n_chunks * 64] the GEMM's weight-tile TMA reads.
// A piece is a word of eight codes and the 16 bytes of the panel it becomes, with the arithmetic and the K
// order of the activation converters (expand_word), so a dot product pairs the right values.  A thread takes kExpandPieces pieces a block's
// width apart, so that a warp reads 128 and writes 512 bytes side by side.  With a thread per chunk of 64 codes, whose stores left a warp as 32 pieces in
// as many lines and whose blocks were half as many as multiprocessors, a panel of 1152 x 1088 cost a call 10 us; now 4 (with the GEMM: 32768
// rows 82.7 -> 75.8, 4096 rows 27.4 -> 19.3, 1024 x 2240 x 2240 26.6 -> 18.4).
// hc != 0 (half chunks: per-head groups of at most 32 channels, whose chunks are half padding): only the first 32 code slots of
// a chunk are expanded and two chunks share one 64-wide stage of the panel, [N, ceil(n_chunks / 2) * 64].
constexpr int kExpandPieces = 4;
__host__ __device__ __forceinline__ int expand_stages(int n_chunks, int hc) { return hc ? (n_chunks + 1) >> 1 : n_chunks; }
static int64_t expand_blocks(int64_t N, int n_chunks, int hc) {
  return (N * expand_stages(n_chunks, hc) * 8 + 256 * kExpandPieces - 1) / (256 * kExpandPieces);
}
__device__ __forceinline__ void expand_weight_panel_block(int block, const uint8_t* __restrict__ wq, int64_t w_row_bytes,
                                                          const uint2* __restrict__ rec, int64_t ld_rec, int64_t N, int n_chunks,
                                                          uint4* __restrict__ panel, int hc) {
  const int n_stage = expand_stages(n_chunks, hc);
  const int64_t total = N * n_stage * 8, p0 = (int64_t)block * (256 * kExpandPieces) + threadIdx.x;
  uint32_t w[kExpandPieces];
  uint2 k[kExpandPieces];
#pragma unroll
  for (int j = 0; j < kExpandPieces; ++j) {
    const int64_t p = p0 + 256 * j, row_stage = p >> 3;
    const int i = (int)p & 7;
    const int64_t n = total <= 0x7fffffffLL ? (int64_t)((uint32_t)row_stage / (uint32_t)n_stage) : row_stage / n_stage;
    const int st = (int)(row_stage - n * n_stage), c = hc ? 2 * st + (i >> 2) : st;
    w[j] = 0u;
    k[j] = make_uint2(0u, 0u);                        // odd chunk count: the last stage's second half is empty
    if (p < total && c < n_chunks) {
      w[j] = __ldg(reinterpret_cast<const uint32_t*>(wq + n * w_row_bytes + (int64_t)c * 32) + (hc ? i & 3 : i));
      k[j] = __ldg(rec + (int64_t)c * ld_rec + n);
    }
  }
#pragma unroll
  for (int j = 0; j < kExpandPieces; ++j) {
    uint32_t y[4];
    expand_word(w[j], 0x00080008u, k[j].x, hmul2_2m4(k[j].x), k[j].y, y);
    if (p0 + 256 * j < total) panel[p0 + 256 * j] = make_uint4(y[0], y[1], y[2], y[3]);
  }
}

__global__ void __launch_bounds__(256)
expand_weight_panel_kernel(const uint8_t* __restrict__ wq, int64_t w_row_bytes, const uint2* __restrict__ rec, int64_t ld_rec,
                           int64_t N, int n_chunks, uint4* __restrict__ panel, int hc) {
  pdl_launch_dependents();
  pdl_wait();
  expand_weight_panel_block((int)blockIdx.x, wq, w_row_bytes, rec, ld_rec, N, n_chunks, panel, hc);
}

// Both per-call preparations of one GEMM in one launch (each alone is a few microseconds of launch and latency):
// blocks [0, fold_blocks) fold the activation scales, the rest expand the weight panel.
struct FoldExpandArgs {
  const __nv_bfloat16* s; const __nv_bfloat16* z; int n_chunks; int64_t rows; int64_t ld_in; uint2* rec; int64_t ld_rec; float* rs;
  const __nv_bfloat16* tail; __nv_bfloat16* tail_out; int kt_pitch;
  const uint8_t* wq; int64_t w_row_bytes; const uint2* w_rec; int64_t ld_wrec; int64_t N; uint4* panel;
  int fold_blocks;
  int hc;
};
template <int ROWS>
__global__ void __launch_bounds__(256) fold_expand_kernel(const FoldExpandArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  if ((int)blockIdx.x < a.fold_blocks)
    fold_scales_block<__nv_bfloat16, ROWS>((int)blockIdx.x, a.s, a.z, a.n_chunks, a.rows, a.ld_in, a.rec, a.ld_rec, a.rs, a.tail,
                                     a.tail_out, a.kt_pitch);
  else
    expand_weight_panel_block((int)blockIdx.x - a.fold_blocks, a.wq, a.w_row_bytes, a.w_rec, a.ld_wrec, a.N, a.n_chunks, a.panel,
                              a.hc);
}

int launch_expand_weight_panel(const uint8_t* wq, int n_chunks, int64_t N, const void* rec, void* panel, cudaStream_t st, int hc) {
  if (N <= 0 || n_chunks <= 0) return DIROTQ_OK;
  return launch_pdl(expand_weight_panel_kernel, dim3((unsigned)expand_blocks(N, n_chunks, hc)), dim3(256), 0, st, wq,
                    (int64_t)n_chunks * 32, reinterpret_cast<const uint2*>(rec), f16_ld_weight(N), N, n_chunks,
                    reinterpret_cast<uint4*>(panel), hc) == cudaSuccess
             ? DIROTQ_OK : DIROTQ_E_CUDA;
}

// Records are read in whole tiles of rows (bulk copies, no bounds handling), so the record arrays are
// padded: activations to 128 rows, weights to 768 (a multiple of every column-tile width).
int64_t f16_ld_act(int64_t M) { return round_up64(M, 128); }
int64_t f16_ld_weight(int64_t N) { return round_up64(N, 768); }

// Rows per block of the folding kernels: 64 keeps whole sectors of scales in a warp, 16 (a 32-byte sector of scales) spread a call
// of fewer than two 64-row blocks per SM over four times as many.  Wide 16-bit tails, which are most of the bytes, want the latter,
// narrow ones the former (us, folding + GEMM of a long sibling call, 16 / 64 rows: 16384 x 2240 x 2240, 320 16-bit channels, 125.3 / 129.0, 8192 x
// 3072 x 3072, 384 of them, 120.1 / 126.4, 18432 rows 236.9 / 239.3; 16384 x 1152 x 1152, 64 of them, 50.3 / 48.6, 18000 rows 51.2 / 49.5, 32768 rows
// 86.5 / 81.4); the line, by rows alone, costs the narrow ones below it 1.7 us.
static bool fold_small_blocks(int64_t ld_rec) { return ld_rec / 64 < 2 * (int64_t)num_sms(); }

int launch_fold_act_scales(const __nv_bfloat16* s, const __nv_bfloat16* z, int n_chunks, int64_t M, int64_t ldm,
                           void* rec, float* rs, const __nv_bfloat16* tail, __nv_bfloat16* tail_out,
                           int kt_pitch, cudaStream_t st) {
  if (M <= 0) return DIROTQ_OK;
  const int64_t ld_rec = f16_ld_act(M);
  const bool small = fold_small_blocks(ld_rec);
  return launch_pdl(small ? fold_scales_kernel<__nv_bfloat16, 16> : fold_scales_kernel<__nv_bfloat16, 64>,
                    dim3((unsigned)(ld_rec / (small ? 16 : 64))), dim3(256), 0, st, s, z, n_chunks, M,
                    ldm, reinterpret_cast<uint2*>(rec), ld_rec, rs, tail, tail_out, kt_pitch) == cudaSuccess
             ? DIROTQ_OK : DIROTQ_E_CUDA;
}

int launch_fold_act_and_expand(const __nv_bfloat16* s, const __nv_bfloat16* z, int n_chunks, int64_t M, int64_t ldm, void* rec,
                               float* rs, const __nv_bfloat16* tail, __nv_bfloat16* tail_out, int kt_pitch, const uint8_t* wq,
                               int64_t N, const void* w_rec, void* panel, cudaStream_t st, int hc) {
  if (M <= 0 || N <= 0) return DIROTQ_OK;
  FoldExpandArgs a;
  a.hc = hc;
  a.s = s; a.z = z; a.n_chunks = n_chunks; a.rows = M; a.ld_in = ldm; a.rec = reinterpret_cast<uint2*>(rec);
  a.ld_rec = f16_ld_act(M); a.rs = rs; a.tail = tail; a.tail_out = tail_out; a.kt_pitch = kt_pitch;
  a.wq = wq; a.w_row_bytes = (int64_t)n_chunks * 32; a.w_rec = reinterpret_cast<const uint2*>(w_rec);
  a.ld_wrec = f16_ld_weight(N); a.N = N; a.panel = reinterpret_cast<uint4*>(panel);
  const bool small = fold_small_blocks(a.ld_rec);
  a.fold_blocks = (int)(a.ld_rec / (small ? 16 : 64));
  const unsigned blocks = (unsigned)a.fold_blocks + (unsigned)expand_blocks(N, n_chunks, hc);
  return launch_pdl(small ? fold_expand_kernel<16> : fold_expand_kernel<64>, dim3(blocks), dim3(256), 0, st, a) == cudaSuccess ? DIROTQ_OK : DIROTQ_E_CUDA;
}

int launch_fold_weight_scales(const float* s, int n_chunks, int64_t N, int64_t ldn, void* rec, float* cs,
                              const __nv_bfloat16* tail, __nv_bfloat16* tail_out, int kt_pitch, cudaStream_t st) {
  if (N <= 0) return DIROTQ_OK;
  const int64_t ld_rec = f16_ld_weight(N);
  fold_scales_kernel<float, 64><<<(unsigned)(ld_rec / 64), 256, 0, st>>>(
      s, nullptr, n_chunks, N, ldn, reinterpret_cast<uint2*>(rec), ld_rec, cs, tail, tail_out, kt_pitch);
  return cudaGetLastError() == cudaSuccess ? DIROTQ_OK : DIROTQ_E_CUDA;
}

template <int BN, int AMODE, bool PAIR, bool REC = false>
static int launch_gf(const GfMaps& tm, const GemmIntF16Args& a, cudaStream_t st) {
  using Cfg = GfCfg<BN, AMODE == 2, PAIR>;
  auto k = gemm_int_f16_kernel<BN, AMODE, PAIR, REC>;
  static PerDeviceOnce attr_once, regs_once;
  if (int rc = set_max_dynamic_smem(attr_once, k, Cfg::SMEM_BYTES)) return rc;
  if (int rc = check_compiled_regs(regs_once, k, Cfg::REGS_LAUNCH)) return rc;
  if constexpr (PAIR) {
    const int64_t tiles = ((a.N + BN - 1) / BN) * ((a.M + 255) / 256);
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(Cfg::THREADS);
    cfg.dynamicSmemBytes = Cfg::SMEM_BYTES;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    // persistent grid: as many pairs as can be resident at once, remembered per device
    static std::atomic<int> resident[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return DIROTQ_E_CUDA;
    int max_pairs = resident[dev].load(std::memory_order_relaxed);
    if (max_pairs <= 0) {
      cfg.gridDim = dim3(2 * (num_sms() / 2));
      cfg.numAttrs = 1;
      if (cudaOccupancyMaxActiveClusters(&max_pairs, k, &cfg) != cudaSuccess || max_pairs <= 0) max_pairs = num_sms() / 2;
      resident[dev].store(max_pairs, std::memory_order_relaxed);
    }
    cfg.gridDim = dim3(2 * (unsigned)(tiles < max_pairs ? tiles : max_pairs));
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, k, tm, a) == cudaSuccess ? DIROTQ_OK : DIROTQ_E_CUDA;
  }
  const int tiles = (int)((a.N + BN - 1) / BN) * (int)((a.M + 127) / 128);
  const int grid = min(tiles, num_sms());
  return launch_pdl(k, dim3(grid), dim3(Cfg::THREADS), Cfg::SMEM_BYTES, st, tm, a) == cudaSuccess ? DIROTQ_OK : DIROTQ_E_CUDA;
}

// Column-tile width.  The persistent grid runs whole rounds of tiles, over 148 CTAs with 128-wide tiles and 74 CTA pairs (256 rows) with
// wider ones.  A round takes 225 / 250 / 320 ns per 64-wide unit of K (128 / 192 / 256 columns) and 1.0 / 1.4 / 1.5 us besides: what a
// stage costs the roles hardly depends on the width, the UMMAs do, and a wide tile's single accumulator has to be handed back.
// Launch, first loads and last epilogue add 4.5 / 5.5 / 6 us.  The smallest sum is taken; measured (us, 128 / 192 / 256 columns): 256 x
// 1152 x 1152 9.4 / 11.1 / 12.7, 1024 x 2240 x 2240 14.3 / 16.8 / 18.9, 4096 x 4608 x 1152 39.3 / 43.8 / 53.3, 3995 x 1152 x 4608 45.5 / 41.0 /
// 37.3, 8192 x 2240 x 2240 75 / 65.5 / 59.4, 32768 x 1152 x 1152 85.6 / 71.7 / 73.3, 4608 x 3072 x 3072 73.8 / 60.6 / 59.4.
// Calls of at most 128 rows would leave half of each pair idle.  The quantise-out epilogue wants whole groups of 64 columns per
// warp: not 192.  DIROTQ_GF_BN overrides.
static int pick_bn_f16(int64_t M, int64_t N, int64_t units, bool qout) {
  if (const char* e = getenv("DIROTQ_GF_BN")) return atoi(e) <= 128 ? 128 : atoi(e) <= 192 && !qout ? 192 : 256;
  if (M <= 128) return 128;
  static const int width[3] = {128, 192, 256}, unit_ns[3] = {225, 250, 320}, tile_ns[3] = {1000, 1400, 1500}, call_ns[3] = {4500, 5500, 6000};
  const int64_t m128 = (M + 127) / 128, m256 = (M + 255) / 256, sms = num_sms();
  int best = 128;
  int64_t best_ns = -1;
  for (int i = 0; i < 3; ++i) {
    if (qout && width[i] == 192) continue;
    const int64_t n = (N + width[i] - 1) / width[i], slots = i ? sms / 2 : sms, rounds = ((i ? m256 : m128) * n + slots - 1) / slots;
    const int64_t ns = rounds * (units * unit_ns[i] + tile_ns[i]) + call_ns[i];
    if (best_ns < 0 || ns < best_ns) { best_ns = ns; best = width[i]; }
  }
  return best;
}

// Column tiles per rasterisation group.  With n fastest over the whole width, the CTAs of one round read every weight
// column tile of the layer; once the fp16 panel no longer sits in L2 next to the activation and output streams (3072 ->
// 12288: 75 MB) those reads go to HBM again on every round.  Groups bound the weight tiles in flight to about 24 MB
// (3072 -> 12288 at 18432 rows: 1325 -> 1169 us, 3072 -> 9216: 927 -> 880, 12288 -> 3072: 1172 -> 1126); layers whose
// panel fits (under 32 MB) keep the plain order, which was 1-2 % faster for them.  DIROTQ_GF_RASTER overrides.
static int pick_raster_f16(int BN, int64_t N, int64_t k_total) {
  if (const char* e = getenv("DIROTQ_GF_RASTER")) return atoi(e);
  const int64_t tile_bytes = (int64_t)BN * k_total * 2, panel_bytes = N * k_total * 2;
  if (panel_bytes <= (32ll << 20) || tile_bytes <= 0) return 0;
  const int64_t g = ((24ll << 20) + tile_bytes / 2) / tile_bytes;
  return (int)(g < 4 ? 4 : g > 16 ? 16 : g);
}

// Whether siblings that share activations without being one GEMM read records (and row powers of two, and a scaled tail) that the
// folding kernel makes once for all of them; other calls read the scales themselves.  The folding kernel is 2-3 us of launch and
// latency, its share of the work in the GEMM four to ten instructions per row and chunk of the converters, which have time for them (us,
// folding kernel + GEMM / GEMM alone, 256 columns: 32768 x 1152 x 3456 199.5 / 197.4, 16384 x 2240 x 2240 120.0 / 113.9, 4608 x 3072 x
// 3072 63.1 / 59.4, x 12288 232.5 / 230.4; before the converters read a raw stage at once the long launches were 2-4 % slower alone).
// For long launches (more than four rounds of 148 tiles) of three siblings the two come out even, and a group keeps its records.
// DIROTQ_GF_BN overrides: 256 takes records, narrower tiles do not.
bool gemm_int_f16_takes_records(int64_t M, int64_t N) {
  if (getenv("DIROTQ_GF_BN")) return pick_bn_f16(M, N, 1, false) == 256;
  return N > 128 && ((M + 127) / 128) * ((N + 255) / 256) > 4 * (int64_t)num_sms();
}

int launch_gemm_int_f16(const GemmIntF16Args& a_in, cudaStream_t st) {
  GemmIntF16Args a = a_in;
  if (a.M <= 0 || a.N <= 0) return DIROTQ_OK;
  if (a.a_mode != DIROTQ_INT4_SYM && a.a_mode != DIROTQ_INT4_ASYM && a.a_mode != DIROTQ_INT8_ASYM) return DIROTQ_E_UNSUPPORTED;
  if ((reinterpret_cast<uintptr_t>(a.bias) & 15) || (reinterpret_cast<uintptr_t>(a.cs) & 15) || (a.N & 7) ||
      (reinterpret_cast<uintptr_t>(a.a_const) & 15) || (reinterpret_cast<uintptr_t>(a.w_panel) & 15) || !a.w_panel)
    return DIROTQ_E_ALIGN;
  const uint64_t n_stage = a.half_chunks ? (uint64_t)((a.n_chunks + 1) / 2) : (uint64_t)a.n_chunks;
  const int64_t k_total = (int64_t)n_stage * 64 + ((a.kt + 63) / 64) * 64;
  const bool rec = a.a_const != nullptr;
  const int BN = rec ? 256 : pick_bn_f16(a.M, a.N, k_total / 64, a.q_codes != nullptr);
  const bool pair = BN > 128;
  if (rec ? !a.rs : !a.xs) return DIROTQ_E_ARG;
  if (a.q_codes) {
    if (a.N % 64 || a.q_len % 64 || a.q_len <= 0 || a.q_len > a.N || a.q_row_bytes < a.q_len / 2 || (a.q_row_bytes & 15) ||
        (a.q_len < a.N && (!a.q_tail || a.q_tail_pitch < a.N - a.q_len || (a.q_tail_pitch & 7) ||
                           (reinterpret_cast<uintptr_t>(a.q_tail) & 15))) ||
        !a.q_scales || (a.q_mode != DIROTQ_INT4_SYM && a.q_mode != DIROTQ_INT4_ASYM) ||
        (a.q_mode == DIROTQ_INT4_ASYM && !a.q_zeros) || (reinterpret_cast<uintptr_t>(a.q_codes) & 15))
      return DIROTQ_E_ARG;
  } else if (!a.y) {
    return DIROTQ_E_ARG;
  }
  GfMaps tm;
  int rc = make_tmap_2d_sw(&tm.xq, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a.xq, (uint64_t)a.x_row_bytes, (uint64_t)a.M,
                           (uint64_t)a.x_row_bytes, 32 * GF_CPS, 128, 32 * GF_CPS);
  if (rc) return rc;
  tm.xs = tm.xz = tm.xq;
  if (!rec) {
    // scales (and zero points): [n_chunks, ldm] bf16, a stage's four chunks of 128 rows in one box
    rc = make_tmap_2d_sw(&tm.xs, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, a.xs, (uint64_t)a.ldm, (uint64_t)a.n_chunks, (uint64_t)a.ldm * 2,
                         128, GF_CPS, 0);
    if (!rc && a.a_mode != DIROTQ_INT4_SYM)
      rc = make_tmap_2d_sw(&tm.xz, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, a.xz, (uint64_t)a.ldm, (uint64_t)a.n_chunks,
                           (uint64_t)a.ldm * 2, 128, GF_CPS, 0);
    if (rc) return rc;
  }
  if (a.raster == 0) a.raster = pick_raster_f16(BN, a.N, k_total);
  rc = make_tmap_2d(&tm.wp, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, a.w_panel, n_stage * 64, (uint64_t)a.N, n_stage * 128, pair ? BN / 2 : BN);
  if (rc) return rc;
  // without an output tensor (quantise-out only) the map is never used: any valid address will do
  rc = make_tmap_2d_sw(&tm.y, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, a.y ? (const void*)a.y : a.w_panel, (uint64_t)a.N, (uint64_t)a.M, (uint64_t)a.N * 2,
                       32, 32, 64);
  if (rc) return rc;
  if (a.kt > 0) {
    rc = make_tmap_2d(&tm.xt, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, a.xt, (uint64_t)a.kt, (uint64_t)a.M, (uint64_t)a.kt_pitch * 2, 128);
    if (rc) return rc;
    rc = make_tmap_2d(&tm.wt, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, a.wt, (uint64_t)a.kt, (uint64_t)a.N, (uint64_t)a.kt_pitch * 2, pair ? BN / 2 : BN);
    if (rc) return rc;
  } else {
    tm.xt = tm.xq;
    tm.wt = tm.wp;
  }
  const int amode = a.a_mode == DIROTQ_INT4_SYM ? 0 : a.a_mode == DIROTQ_INT4_ASYM ? 1 : 2;
  switch (BN * 4 + amode) {
    case 256 * 4 + 0: return rec ? launch_gf<256, 0, true, true>(tm, a, st) : launch_gf<256, 0, true>(tm, a, st);
    case 256 * 4 + 1: return rec ? launch_gf<256, 1, true, true>(tm, a, st) : launch_gf<256, 1, true>(tm, a, st);
    case 256 * 4 + 2: return rec ? launch_gf<256, 2, true, true>(tm, a, st) : launch_gf<256, 2, true>(tm, a, st);
    case 192 * 4 + 0: return launch_gf<192, 0, true>(tm, a, st);
    case 192 * 4 + 1: return launch_gf<192, 1, true>(tm, a, st);
    case 192 * 4 + 2: return launch_gf<192, 2, true>(tm, a, st);
    case 128 * 4 + 0: return launch_gf<128, 0, false>(tm, a, st);
    case 128 * 4 + 1: return launch_gf<128, 1, false>(tm, a, st);
    case 128 * 4 + 2: return launch_gf<128, 2, false>(tm, a, st);
  }
  return DIROTQ_E_ARG;
}

}  // namespace dq
