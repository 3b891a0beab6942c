// Kernel 1: fused rotate + split + quantise.
//
//   x [M, D] bf16  --TMA-->  smem (128-byte swizzle)  --tcgen05.mma kind::f16-->  TMEM fp32
//   TMEM --tcgen05.ld--> registers: round to bf16 (this IS x_rot of the reference's bf16 path),
//   split into the quantised region and the passthrough tail, per-group extrema, scale / zero
//   point, 4-bit (or 8-bit) codes, packed 16-byte stores.  The rotated tensor never touches HBM.
//
// Persistent, warp-specialised: warp 0 = TMA producer, warp 1 = UMMA issuer (owns TMEM),
// warps 2..9 = epilogue (two per TMEM lane quarter, alternating over the 64-column groups).  Two TMEM accumulators of 256 columns let
// the epilogue of tile i overlap the main loop of tile i+1.  Tiles are 128 rows x BN columns of
// the rotated tensor; consecutive tiles share the x row-block, so x and the rotation stay in L2.
//
// Replaces: `x_flat @ self.rotation` + find_params + quantizer (DiRotQ
// dirotq_fused_unrotation_fast.py:69-74), the per-head branch (:76-104) and the stand-alone
// rotation kernels speedup/kernels/{int8,fp8,bf16}_rotation.py.
#include <cstdlib>
#include <cstring>
#include <cuda.h>
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include "layout.cuh"
#include "launchers.cuh"
#include "ptx.cuh"
#include "ptx_pair.cuh"
#include "tma_host.cuh"
#include "quant_math.cuh"

namespace dq {

constexpr int RQ_A_BYTES = 128 * 128;           // 128 rows x 64 bf16
// One CTA per tile: the whole rotation tile (up to 256 rows x 64 bf16) per stage, four stages.  CTA pairs
// (tcgen05 cta_group::2, 256 token rows per pair): each CTA fetches only HALF of the rotation tile -- the tensor core
// reads the other half from the peer's shared memory -- so a stage is 32 KB instead of 48 and six fit.
// UNITS: 64-wide pieces of K per stage.  A stage costs producer and issuer a barrier test of 110 cycles and more, which the UMMAs of
// tiles of at most 128 columns do not hide: two units for those (us, one / two: bf16 4096 x 4608 -> 1152 34.8 / 31.6, rotation of 16384 x 1152 on
// 128 columns 43.8 / 33.6, of 4096 x 1152 13.1 / 12.7; 256 rows, where latencies add up, 7.4 either way).
template <bool PAIR, int UNITS> struct RqStage {
  static constexpr int STAGES = UNITS == 2 ? (PAIR ? 4 : 3) : (PAIR ? 6 : 4);
  static constexpr int B_BYTES = (PAIR ? 128 : 256) / UNITS * 128;
  static constexpr int UNIT_BYTES = RQ_A_BYTES + B_BYTES, STAGE_BYTES = UNITS * UNIT_BYTES;
};
// Epilogue warps per TMEM lane quarter: they take the 64-column chunks (per-head layouts: the heads) of their rows in
// turns.  The NVFP4 epilogue has four scales per chunk to make and is latency-bound, and the per-head
// epilogues wait on several tensor-memory reads per head, so those get more warps.
#ifndef RQ_WPQ_NVFP4
#define RQ_WPQ_NVFP4 4
#endif
#ifndef RQ_WPQ_PERHEAD
#define RQ_WPQ_PERHEAD 4
#endif
constexpr int RQ_TAIL_STAGED = 16;              // high channels per head that go through the staging patch, at most
template <int EPI, bool PAIR = false, int UNITS = 1> struct RqCfg {
  static constexpr int WPQ = (EPI == 2 /* EPI_NVFP4_HIDDEN */) ? RQ_WPQ_NVFP4 : (EPI == 3 || EPI == 4 /* per-head */) ? RQ_WPQ_PERHEAD : 2;
  static constexpr int EPI_WARPS = 4 * WPQ;
  static constexpr int THREADS = (2 + EPI_WARPS) * 32;
  // per epilogue warp: EPI_ROT_ONLY (0) a 32 x 32 bf16 staging patch for its TMA stores, EPI_INT_PERHEAD (3) the high
  // channels of a head of its 32 rows
  static constexpr int STG_WARP = EPI == 0 ? 2048 : EPI == 3 ? 32 * RQ_TAIL_STAGED * 2 : 0;
  static constexpr int STG_BYTES = EPI_WARPS * STG_WARP;
  static constexpr int SMEM_BYTES = RqStage<PAIR, UNITS>::STAGES * RqStage<PAIR, UNITS>::STAGE_BYTES + STG_BYTES + 1024 /*align*/ + 256 /*barriers*/;
};

enum : int { EPI_ROT_ONLY = 0, EPI_INT_HIDDEN = 1, EPI_NVFP4_HIDDEN = 2, EPI_INT_PERHEAD = 3, EPI_NVFP4_PERHEAD = 4 };


// Tile t: row block and column block.  Where the last column block is narrower than the others, a row block's columns start one
// further than those of the row block before, so that a CTA, which takes every gridDim-th tile, meets narrow tiles in turn
// even where the grid and the number of columns have a common factor.
__device__ __forceinline__ void tile_at(const RotArgs& a, int t, int& mt, int& nb) {
  mt = t / a.n_tiles;
  nb = t - mt * a.n_tiles;
  if (a.bn_last != a.BN) {
    nb += mt % a.n_tiles;
    if (nb >= a.n_tiles) nb -= a.n_tiles;
  }
}
__device__ __forceinline__ int tile_width(const RotArgs& a, int nb) { return nb + 1 == a.n_tiles ? a.bn_last : a.BN; }

__device__ __forceinline__ void tile_k_range(const RotArgs& a, int nb, int& kb, int& ke) {
  const int kchunks = (a.K + 63) / 64;
  if (a.band == 0) { kb = 0; ke = kchunks; return; }
  const int n0 = nb * a.BN;
  const int n1 = min(n0 + a.BN, a.g.D);
  const int h0 = n0 / a.band, h1 = (n1 - 1) / a.band;
  kb = (h0 * a.band) / 64;
  ke = min(kchunks, ((h1 + 1) * a.band + 63) / 64);
}

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&h);
}

// 32 bytes of codes of one row: a whole sector in one store where the code buffer starts on a sector (rows are multiples of
// 32 bytes).  Lanes hold different rows, so a store is one request per lane whatever its width.
__device__ __forceinline__ void store_codes32(uint8_t* dst, bool whole, uint4 lo, uint4 hi) {
  if (whole) {
    st_global_32(dst, lo, hi);
  } else {
    reinterpret_cast<uint4*>(dst)[0] = lo;
    reinterpret_cast<uint4*>(dst)[1] = hi;
  }
}

// ---- epilogues: thread = one row of the tile; `taddr` already points at this warp's lanes.
// The 4-bit quantisers stay on the packed bf16 pairs (the scalar form ended a launch 0.2-0.3 us later: 256 x 1152 7.16 -> 6.93 us, 2048
// x 1152 8.42 -> 8.17; launches of many rounds hide either behind the UMMAs).
// Several warps (wpq) share a lane quarter; `turn` counts work items (64-column chunks, heads) across tiles
// and a warp takes the items whose index modulo wpq equals its `half`, which balances odd counts per tile.
template <int MODE>
__device__ __forceinline__ void epi_int_hidden(const RotArgs& a, uint32_t taddr, int64_t row, int n0, int half, uint32_t& turn, int wpq = 2) {
  const ActGeom& g = a.g;
  const bool row_ok = row < a.M, whole = (reinterpret_cast<uintptr_t>(a.codes) & 31) == 0;
  constexpr float maxq = (MODE == MODE_INT4_SYM) ? 7.f : (MODE == MODE_INT4_ASYM ? 15.f : 255.f);
  for (int c0 = 0; c0 < a.BN; c0 += 64) {
    const int col = n0 + c0;
    if (col >= g.D) break;
    if (((turn++) % (uint32_t)wpq) != (uint32_t)half) continue;
    uint32_t r[64];
    __syncwarp();                                 // lanes may have quantised the chunk before in different ways
    tmem_ld32(taddr + c0, r);
    tmem_ld32(taddr + c0 + 32, r + 32);
    tmem_wait_ld();
    // round the fp32 accumulators to bf16 pairs: this IS x_rot of the reference's bf16 forward
    uint32_t xb[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) xb[j] = pack_bf16x2(__uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1]));
    if (a.x_rot && row_ok) {
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (col + 8 * i + 8 <= g.D)
          *reinterpret_cast<uint4*>(a.x_rot + row * g.D + col + 8 * i) = make_uint4(xb[4 * i], xb[4 * i + 1], xb[4 * i + 2], xb[4 * i + 3]);
    }
    if (!a.codes) continue;
    const int nq = max(0, min(64, g.q_len - col));
    if (nq < 64 && row_ok && a.tail) {
      __nv_bfloat16* tr = a.tail + row * g.tail_pitch;
      const int t0 = col - g.q_len;               // tail index of the chunk's first column (may be negative)
      if (nq == 0 && (t0 & 7) == 0 && col + 64 <= g.D) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
          *reinterpret_cast<uint4*>(tr + t0 + 8 * i) = make_uint4(xb[4 * i], xb[4 * i + 1], xb[4 * i + 2], xb[4 * i + 3]);
      } else {
#pragma unroll
        for (int j = 0; j < 64; ++j)
          if (j >= nq && col + j < g.D) tr[t0 + j] = __ushort_as_bfloat16((unsigned short)((j & 1) ? xb[j >> 1] >> 16 : xb[j >> 1]));
      }
    }
    if (nq == 0) continue;
    const int chunk = col >> 6;
    if (nq < 64) {                                // zero padding of the last group takes part in the extrema; its codes: symmetric 0,
#pragma unroll                                    // asymmetric slots meet zero weights
      for (int j = 0; j < 32; ++j) xb[j] &= (2 * j + 1 < nq) ? 0xFFFFFFFFu : ((2 * j < nq) ? 0x0000FFFFu : 0u);
    }
    float mx = -INFINITY, mn = INFINITY;
#pragma unroll
    for (int j = 0; j < 4; ++j) minmax_bf16x16(xb + 8 * j, mx, mn);
    GroupParams p;
    if constexpr (MODE == MODE_INT4_SYM) p = int_sym_params<true>(mx, mn, g.clip, maxq);
    else p = int_asym_params<true>(mx, mn, g.clip, maxq);
    const float rcp = __frcp_rn(p.scale);
    if (!row_ok) continue;
    if constexpr (MODE == MODE_INT4_SYM) {
      const bool clamp = g.clip < 1.f || !(p.scale < INFINITY);      // else no quotient passes 7.03
      store_codes32(a.codes + row * g.code_row_bytes + (int64_t)chunk * 32, whole, int_sym_planar32_packed(xb, rcp, clamp),
                    int_sym_planar32_packed(xb + 16, rcp, clamp));
    } else if constexpr (MODE == MODE_INT4_ASYM) {
      const bool packs = int_asym_packs(mx, mn, rcp, p.zero);
      store_codes32(a.codes + row * g.code_row_bytes + (int64_t)chunk * 32, whole, int_asym_planar32(xb, p.scale, rcp, p.zero, packs),
                    int_asym_planar32(xb + 16, p.scale, rcp, p.zero, packs));
    } else {
      uint8_t* dst = a.codes + row * g.code_row_bytes + (int64_t)chunk * 64;
      const bool packs = int_asym_packs8(mx, mn, rcp, p.zero);
#pragma unroll
      for (int i = 0; i < 2; ++i)
        store_codes32(dst + 32 * i, whole, int_asym_byte16_packed(xb + 16 * i, p.scale, rcp, p.zero, packs),
                      int_asym_byte16_packed(xb + 16 * i + 8, p.scale, rcp, p.zero, packs));
    }
    a.scales[(int64_t)chunk * a.ldm + row] = __float2bfloat16_rn(p.scale);
    if constexpr (MODE != MODE_INT4_SYM) a.zeros[(int64_t)chunk * a.ldm + row] = __float2bfloat16_rn(p.zero);
  }
}

// One 16-column quantisation group at a time (tcgen05.ld x16, a rolled loop over the chunk's four groups):
// the longest epilogue of the kernel stays small in registers and in code, so more warps can share a lane
// quarter and hide each other's latencies.
template <int MODE>
__device__ __forceinline__ void epi_nvfp4_hidden(const RotArgs& a, uint32_t taddr, int64_t row, int n0, int half, uint32_t& turn, int wpq = 2) {
  const ActGeom& g = a.g;
  const bool row_ok = row < a.M;
  const int n_kb64_pad = (g.n_chunks + 3) & ~3;
  const bool short_T = nvfp4_short_tensor_scale(g.T);
  const bool pow2_T = nvfp4_pow2_tensor_scale(g.T);
  for (int c0 = 0; c0 < a.BN; c0 += 64) {
    const int col = n0 + c0;
    if (col >= g.D) break;
    if (((turn++) % (uint32_t)wpq) != (uint32_t)half) continue;
    const int nq = max(0, min(64, g.q_len - col));
    const int chunk = col >> 6;
    uint32_t sfw = 0;
    if constexpr (MODE == MODE_NVFP4_HW) {
      if (nq == 64 && pow2_T && a.codes && !a.x_rot) {
        // a whole chunk under a power-of-two tensor scale: two groups at a time on packed pairs (nvfp4_hw_group)
#pragma unroll 1
        for (int gp = 0; gp < 2; ++gp) {
          uint32_t r[32];
          __syncwarp();                           // lanes may have quantised the groups before in different ways
          tmem_ld32(taddr + c0 + 32 * gp, r);
          tmem_wait_ld();
          uint32_t w[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) w[i] = pack_bf16x2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
          uint2 k0, k1;
          const uint32_t s0 = nvfp4_hw_group(w, g.clip, g.T, k0), s1 = nvfp4_hw_group(w + 8, g.clip, g.T, k1);
          sfw |= (s0 | s1 << 8) << (16 * gp);
          if (row_ok) *reinterpret_cast<uint4*>(a.codes + row * g.code_row_bytes + (int64_t)chunk * 32 + gp * 16) = make_uint4(k0.x, k0.y, k1.x, k1.y);
        }
        if (row_ok) *reinterpret_cast<uint32_t*>(a.sf + sf_offset(row, chunk * 4, n_kb64_pad)) = sfw;
        continue;
      }
    }
#pragma unroll 1
    for (int gi = 0; gi < 4; ++gi) {
      const int gcol = col + 16 * gi;
      if (gcol >= g.D) break;
      uint32_t r[16];
      __syncwarp();
      tmem_ld16(taddr + c0 + 16 * gi, r);
      tmem_wait_ld();
      // the rotated values, rounded to bf16 and packed in pairs: what the quantiser is defined on
      uint32_t w[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) w[i] = pack_bf16x2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
      if (a.x_rot && row_ok) {
#pragma unroll
        for (int i = 0; i < 2; ++i)
          if (gcol + 8 * i + 8 <= g.D)
            *reinterpret_cast<uint4*>(a.x_rot + row * g.D + gcol + 8 * i) = make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
      }
      if (!a.codes) continue;
      const int nvalid = max(0, min(16, nq - 16 * gi));
      if constexpr (MODE == MODE_NVFP4_HW) {
        if (nvalid == 16 && pow2_T) {
          // whole group, power-of-two tensor scale
          uint2 c;
          const uint8_t sb = nvfp4_hw_group(w, g.clip, g.T, c);
          sfw |= (uint32_t)sb << (8 * gi);
          if (row_ok) *reinterpret_cast<uint2*>(a.codes + row * g.code_row_bytes + (int64_t)chunk * 32 + gi * 8) = c;
          continue;
        }
      }
      float v[16];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        v[2 * i] = __uint_as_float(w[i] << 16);
        v[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
      }
      if (nvalid > 0) {
        float amax = 0.f;
#pragma unroll
        for (int j = 0; j < 16; ++j)
          if (j < nvalid) amax = fmaxf(amax, fabsf(v[j]));
        uint32_t lo = 0, hi = 0;
        if constexpr (MODE == MODE_NVFP4_REF) {
          const float sc = nvfp4_ref_scale<true>(amax, g.clip);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            lo |= (j < nvalid ? nvfp4_ref_code<true>(v[j], sc) : 0u) << (4 * j);
            hi |= (8 + j < nvalid ? nvfp4_ref_code<true>(v[8 + j], sc) : 0u) << (4 * j);
          }
          if (row_ok) a.scales[(int64_t)(chunk * 4 + gi) * a.ldm + row] = __float2bfloat16_rn(sc);
        } else {
          float eff = 0.f;
          const uint8_t sb = nvfp4_hw_scale(amax, g.clip, g.T, &eff);
          uint2 c;
          if (nvalid == 16 && eff > 0.f && short_T)
            c = nvfp4_hw_group_fast(v, eff);
          else
            c = nvfp4_hw_group_partial(v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7], v[8], v[9], v[10], v[11], v[12],
                                       v[13], v[14], v[15], nvalid, eff);
          lo = c.x;
          hi = c.y;
          sfw |= (uint32_t)sb << (8 * gi);
        }
        if (row_ok)
          *reinterpret_cast<uint2*>(a.codes + row * g.code_row_bytes + (int64_t)chunk * 32 + gi * 8) = make_uint2(lo, hi);
      } else if (nq > 0 && row_ok) {
        // a group of the chunk that lies wholly in the tail region: its code slots stay zero
        *reinterpret_cast<uint2*>(a.codes + row * g.code_row_bytes + (int64_t)chunk * 32 + gi * 8) = make_uint2(0u, 0u);
      }
      if (nvalid < 16 && row_ok && a.tail) {
        __nv_bfloat16* tr = a.tail + row * g.tail_pitch;
        const int t0 = gcol - g.q_len;
        if (nvalid == 0 && gcol + 16 <= g.D && ((t0 | g.tail_pitch) & 7) == 0) {
          // a group that lies wholly in the 16-bit tail: two 16-byte stores instead of sixteen 2-byte ones
#pragma unroll
          for (int i = 0; i < 2; ++i)
            *reinterpret_cast<uint4*>(tr + t0 + 8 * i) =
                make_uint4(pack_bf16x2(v[8 * i], v[8 * i + 1]), pack_bf16x2(v[8 * i + 2], v[8 * i + 3]),
                           pack_bf16x2(v[8 * i + 4], v[8 * i + 5]), pack_bf16x2(v[8 * i + 6], v[8 * i + 7]));
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (j >= nvalid && gcol + j < g.D) tr[t0 + j] = __float2bfloat16_rn(v[j]);
        }
      }
    }
    if constexpr (MODE == MODE_NVFP4_HW)
      if (a.codes && nq > 0 && row_ok) *reinterpret_cast<uint32_t*>(a.sf + sf_offset(row, chunk * 4, n_kb64_pad)) = sfw;
  }
}

// Per-head layout: head h = tile columns [hh*d, hh*d + d): first d_q quantised as ONE group, last hlen passthrough.
// What bounds it are this epilogue's instructions and, where a head's high channels are an odd number of 2-byte stores, their
// requests (a lane is a row: every store is one request per lane).  So: bf16 pairs throughout, the ragged last block handled with
// masks from the launch's arguments, a whole code sector per store, and odd tails through a patch of shared memory, so that
// consecutive lanes store consecutive channels.  A group of at most two blocks of 32 keeps its words between extrema and codes;
// a longer one reads tensor memory twice.  Us, before and now: 32768 x 16 heads of 72 (9 high) 61.4 / 36.9, 16384 x 70 of 32 (4 high)
// 51.6 / 35.2, in 8 bits 75.4 / 40.6, 18432 x 24 of 128 (16 high) 47.1 / 41.4, NVFP4 63.5 / 49.6; floors by bytes 15 to 25.
// NB: blocks of 32 slots of a group (1, 2; 0 = any number)
template <int MODE, int NB>
__device__ __forceinline__ void perhead_group(const RotArgs& a, uint32_t tcol, int64_t row, bool row_ok, int h, bool whole) {
  const ActGeom& g = a.g;
  constexpr float maxq = (MODE == MODE_INT4_SYM) ? 7.f : (MODE == MODE_INT4_ASYM ? 15.f : 255.f);
  const int nblk = NB ? NB : (g.group + 31) >> 5;
  const bool wide = (g.d & 31) == 0;
  uint32_t pw[NB == 2 ? 32 : 16];
  auto load_block = [&](int b, uint32_t* p) {
    uint32_t r[32];
    __syncwarp();                                 // lanes may have quantised the block before in different ways
    if (wide) {
      tmem_ld32(tcol + 32 * b, r);
    } else {                                      // columns that are only 8-aligned (heads of 72 channels)
      tmem_ld8(tcol + 32 * b, r);
      tmem_ld8(tcol + 32 * b + 8, r + 8);
      tmem_ld8(tcol + 32 * b + 16, r + 16);
      tmem_ld8(tcol + 32 * b + 24, r + 24);
    }
    tmem_wait_ld();
#pragma unroll
    for (int i = 0; i < 16; ++i) p[i] = pack_bf16x2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));   // the rounding of x_rot
  };
  float mx = -INFINITY, mn = INFINITY;
  auto extrema = [&](const uint32_t* p, bool last) {
    if (!last || !a.ragged) {
      minmax_bf16<16>(p, mx, mn);
    } else {
      const uint32_t fill = __byte_perm(p[0], p[0], 0x1010);          // slot 0 of the block (always valid) twice
      uint32_t pm[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) pm[i] = (p[i] & a.pair_mask[i]) | (fill & ~a.pair_mask[i]);
      minmax_bf16<16>(pm, mx, mn);
    }
  };
  if constexpr (NB == 1) {
    load_block(0, pw);
    extrema(pw, true);
  } else if constexpr (NB == 2) {
    load_block(0, pw);
    load_block(1, pw + 16);
    extrema(pw, false);
    extrema(pw + 16, true);
  } else {
#pragma unroll 1
    for (int b = 0; b < nblk; ++b) {
      load_block(b, pw);
      extrema(pw, b + 1 == nblk);
    }
  }
  GroupParams p;
  if constexpr (MODE == MODE_INT4_SYM) p = int_sym_params<true>(mx, mn, g.clip, maxq);
  else p = int_asym_params<true>(mx, mn, g.clip, maxq);
  const float rcp = __frcp_rn(p.scale);
  const uint4 z4 = make_uint4(0u, 0u, 0u, 0u);
  if constexpr (MODE != MODE_INT8_ASYM) {
    const bool packs = MODE == MODE_INT4_SYM ? g.clip < 1.f : int_asym_packs(mx, mn, rcp, p.zero);
    auto codes = [&](const uint32_t* w, bool last) {
      uint4 c;
      if constexpr (MODE == MODE_INT4_SYM) c = int_sym_planar32_packed(w, rcp, packs);
      else c = int_asym_planar32(w, p.scale, rcp, p.zero, packs);
      if (last && a.ragged) c = make_uint4(c.x & a.code_mask[0], c.y & a.code_mask[1], c.z & a.code_mask[2], c.w & a.code_mask[3]);
      return c;
    };
    uint8_t* dst = a.codes + row * g.code_row_bytes + (int64_t)h * g.cpg * 32;
    if constexpr (NB != 0) {
      const uint4 c0 = codes(pw, NB == 1), c1 = NB == 2 ? codes(pw + 16, true) : z4;
      if (row_ok) store_codes32(dst, whole, c0, c1);
    } else {
#pragma unroll 1
      for (int c = 0; c < g.cpg; ++c) {
        load_block(2 * c, pw);
        const uint4 c0 = codes(pw, 2 * c + 1 == nblk);
        uint4 c1 = z4;
        if (2 * c + 1 < nblk) {
          load_block(2 * c + 1, pw);
          c1 = codes(pw, 2 * c + 2 == nblk);
        }
        if (row_ok) store_codes32(dst + 32 * c, whole, c0, c1);
      }
    }
  } else {
    const bool packs = int_asym_packs8(mx, mn, rcp, p.zero);
    uint8_t* dst = a.codes + row * g.code_row_bytes + (int64_t)h * g.cpg * 64;
    auto put = [&](int b, const uint32_t* w, bool last) {
      uint4 c0 = int_asym_byte16_packed(w, p.scale, rcp, p.zero, packs), c1 = int_asym_byte16_packed(w + 8, p.scale, rcp, p.zero, packs);
      if (last && a.ragged) {
        c0 = make_uint4(c0.x & a.code_mask[0], c0.y & a.code_mask[1], c0.z & a.code_mask[2], c0.w & a.code_mask[3]);
        c1 = make_uint4(c1.x & a.code_mask[4], c1.y & a.code_mask[5], c1.z & a.code_mask[6], c1.w & a.code_mask[7]);
      }
      if (row_ok) store_codes32(dst + 32 * b, whole, c0, c1);
    };
    if constexpr (NB != 0) {
      put(0, pw, NB == 1);
      if constexpr (NB == 2) put(1, pw + 16, true);
    } else {
#pragma unroll 1
      for (int b = 0; b < nblk; ++b) {
        load_block(b, pw);
        put(b, pw, b + 1 == nblk);
      }
    }
    if (row_ok)
      for (int b = nblk; b < 2 * g.cpg; ++b) store_codes32(dst + 32 * b, whole, z4, z4);
  }
  if (row_ok) {
    for (int c = 0; c < g.cpg; ++c) {
      a.scales[(int64_t)(h * g.cpg + c) * a.ldm + row] = __float2bfloat16_rn(p.scale);
      if constexpr (MODE != MODE_INT4_SYM) a.zeros[(int64_t)(h * g.cpg + c) * a.ldm + row] = __float2bfloat16_rn(p.zero);
    }
  }
}

template <int MODE>
__device__ __forceinline__ void epi_int_perhead(const RotArgs& a, uint32_t taddr, int64_t row, int lane, int n0, int half, uint32_t& turn,
                                                uint32_t stg) {
  const ActGeom& g = a.g;
  const bool row_ok = row < a.M, whole = (reinterpret_cast<uintptr_t>(a.codes) & 31) == 0;
  constexpr uint32_t WPQ = RqCfg<EPI_INT_PERHEAD>::WPQ;
  const int d = g.d, d_q = g.group;
  const bool staged = g.hlen <= RQ_TAIL_STAGED && ((g.hlen | g.tail_pitch) & 3) != 0;
  int h = n0 / d;
  for (int cb = 0; cb < a.BN && h < g.H; cb += d, ++h) {
    if (((turn++) % WPQ) != (uint32_t)half) continue;
    if (a.x_rot) {
      for (int c8 = 0; c8 < d; c8 += 8) {
        uint32_t r[8];
        tmem_ld8(taddr + cb + c8, r);
        tmem_wait_ld();
        if (row_ok)
          *reinterpret_cast<uint4*>(a.x_rot + row * g.D + n0 + cb + c8) =
              make_uint4(pack_bf16x2(__uint_as_float(r[0]), __uint_as_float(r[1])),
                         pack_bf16x2(__uint_as_float(r[2]), __uint_as_float(r[3])),
                         pack_bf16x2(__uint_as_float(r[4]), __uint_as_float(r[5])),
                         pack_bf16x2(__uint_as_float(r[6]), __uint_as_float(r[7])));
      }
    }
    if (!a.codes) continue;
    if (d_q <= 32) perhead_group<MODE, 1>(a, taddr + cb, row, row_ok, h, whole);
    else if (d_q <= 64) perhead_group<MODE, 2>(a, taddr + cb, row, row_ok, h, whole);
    else perhead_group<MODE, 0>(a, taddr + cb, row, row_ok, h, whole);
    if (!a.tail) continue;
#pragma unroll 1
    for (int c8 = d_q & ~7; c8 < d; c8 += 8) {
      uint32_t r[8];
      __syncwarp();
      tmem_ld8(taddr + cb + c8, r);
      tmem_wait_ld();
      const int t0 = c8 - d_q;                                  // tail index of r[0] within the head (may be negative)
      if (staged) {
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (t0 + j >= 0)
            asm volatile("st.shared.u16 [%0], %1;" ::"r"(stg + (uint32_t)(lane * g.hlen + t0 + j) * 2),
                         "h"(__bfloat16_as_ushort(__float2bfloat16_rn(__uint_as_float(r[j])))) : "memory");
      } else if (row_ok) {
        __nv_bfloat16* tr = a.tail + row * g.tail_pitch + h * g.hlen;
        if (t0 >= 0 && ((t0 | g.hlen | g.tail_pitch) & 7) == 0) {        // a whole, 16-byte aligned octet of tail channels
          *reinterpret_cast<uint4*>(tr + t0) =
              make_uint4(pack_bf16x2(__uint_as_float(r[0]), __uint_as_float(r[1])), pack_bf16x2(__uint_as_float(r[2]), __uint_as_float(r[3])),
                         pack_bf16x2(__uint_as_float(r[4]), __uint_as_float(r[5])), pack_bf16x2(__uint_as_float(r[6]), __uint_as_float(r[7])));
        } else if (t0 == -4 && ((g.hlen | g.tail_pitch) & 3) == 0) {     // the octet's upper half starts the head's tail
          *reinterpret_cast<uint2*>(tr) = make_uint2(pack_bf16x2(__uint_as_float(r[4]), __uint_as_float(r[5])),
                                                     pack_bf16x2(__uint_as_float(r[6]), __uint_as_float(r[7])));
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (t0 + j >= 0) tr[t0 + j] = __float2bfloat16_rn(__uint_as_float(r[j]));
        }
      }
    }
    if (staged) {
      // 32 rows x hlen channels, now consecutive channels by consecutive lanes (e / hlen by multiplication: e < 32 x 16)
      __syncwarp();
      const int64_t row0 = row - lane;
      const uint32_t inv = 65536u / (uint32_t)g.hlen + 1u;
      __nv_bfloat16* const t = a.tail + row0 * g.tail_pitch + h * g.hlen;
#pragma unroll 1
      for (int e = lane; e < 32 * g.hlen; e += 32) {
        const int r = (int)(((uint32_t)e * inv) >> 16);
        uint16_t v;
        asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(stg + (uint32_t)e * 2) : "memory");
        if (row0 + r < a.M) t[r * g.tail_pitch + (e - r * g.hlen)] = __ushort_as_bfloat16(v);
      }
    }
  }
}

// Per-head layout, NVFP4 (hardware recipe): head h = tile columns [hh*d, hh*d + d): its first d - hlen coefficients go to
// code slots h * (d - hlen) .. in blocks of 16 (one UE4M3 scale each, byte-addressed: a head's blocks need not fill a
// scale-factor word), its last hlen to the 16-bit tail.  The GEMM then reads the codes as one hidden-layout row.
__device__ __forceinline__ void epi_nvfp4_perhead(const RotArgs& a, uint32_t taddr, int64_t row, int n0, int half, uint32_t& turn, int wpq = 2) {
  const ActGeom& g = a.g;
  const bool row_ok = row < a.M;
  const int d = g.d, d_q = g.d - g.hlen;
  const int n_kb64_pad = (g.n_chunks + 3) & ~3;
  const bool pow2_T = nvfp4_pow2_tensor_scale(g.T);
  for (int cb = 0; cb < a.BN; cb += d) {
    const int h = (n0 + cb) / d;
    if (h >= g.H) break;
    if (((turn++) % (uint32_t)wpq) != (uint32_t)half) continue;
    if (pow2_T && a.codes && !a.x_rot) {
      // blocks of 16 by nvfp4_hw_group, two at a time from an even block on: 16-byte code stores, two scale bytes
#pragma unroll 1
      for (int c16 = 0; c16 < d_q;) {
        const int slot = h * d_q + c16;                         // first code slot (a multiple of 16)
        uint8_t* dst = a.codes + row * g.code_row_bytes + (slot >> 1);
        uint8_t* sf = a.sf + sf_offset(row, slot >> 4, n_kb64_pad);
        const bool two = !(slot & 16) && c16 + 32 <= d_q;
        uint32_t r[32];
        __syncwarp();                                           // lanes may have quantised the blocks before in different ways
        tmem_ld16(taddr + cb + c16, r);
        if (two) tmem_ld16(taddr + cb + c16 + 16, r + 16);
        tmem_wait_ld();
        uint32_t w[16];
#pragma unroll
        for (int i = 0; i < 16; ++i)
          if (i < 8 || two) w[i] = pack_bf16x2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
        uint2 k0, k1;
        const uint32_t s0 = nvfp4_hw_group(w, g.clip, g.T, k0);
        if (two) {
          const uint32_t s1 = nvfp4_hw_group(w + 8, g.clip, g.T, k1);
          if (row_ok) {
            *reinterpret_cast<uint4*>(dst) = make_uint4(k0.x, k0.y, k1.x, k1.y);
            *reinterpret_cast<uint16_t*>(sf) = (uint16_t)(s0 | s1 << 8);
          }
        } else if (row_ok) {
          *reinterpret_cast<uint2*>(dst) = k0;
          *sf = (uint8_t)s0;
        }
        c16 += two ? 32 : 16;
      }
    }
    const int c_rest = pow2_T && a.codes && !a.x_rot ? d_q : 0;
#pragma unroll 1
    for (int c16 = c_rest; c16 < d; c16 += 16) {
      uint32_t r[16];
      __syncwarp();
      tmem_ld16(taddr + cb + c16, r);
      tmem_wait_ld();
      uint32_t w[8];                       // the rotated values, rounded to bf16 and packed in pairs
#pragma unroll
      for (int i = 0; i < 8; ++i) w[i] = pack_bf16x2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
      if (!row_ok) continue;
      if (a.x_rot) {
        uint4* xr = reinterpret_cast<uint4*>(a.x_rot + row * g.D + n0 + cb + c16);
        xr[0] = make_uint4(w[0], w[1], w[2], w[3]);
        xr[1] = make_uint4(w[4], w[5], w[6], w[7]);
      }
      if (!a.codes) continue;
      if (c16 < d_q) {
        const int slot = h * d_q + c16;                       // first code slot of this block (a multiple of 16)
        uint8_t sb;
        uint2 c;
        if (pow2_T) {
          sb = nvfp4_hw_group(w, g.clip, g.T, c);
        } else {
          float eff = 0.f;
          float v[16];
          float amax = 0.f;
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            v[2 * i] = __uint_as_float(w[i] << 16);
            v[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
            amax = fmaxf(amax, fmaxf(fabsf(v[2 * i]), fabsf(v[2 * i + 1])));
          }
          sb = nvfp4_hw_scale(amax, g.clip, g.T, &eff);
          c = nvfp4_hw_group_partial(v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7], v[8], v[9], v[10], v[11], v[12], v[13],
                                     v[14], v[15], 16, eff);
        }
        *reinterpret_cast<uint2*>(a.codes + row * g.code_row_bytes + (slot >> 1)) = c;
        a.sf[sf_offset(row, slot >> 4, n_kb64_pad)] = sb;
      } else {
        __nv_bfloat16* tr = a.tail + row * g.tail_pitch + h * g.hlen + (c16 - d_q);
        const int left = d - c16;                             // 16, or fewer at the end of a head whose tail is no multiple of 16
        if (left >= 16 && (((h * g.hlen + c16 - d_q) | g.tail_pitch) & 7) == 0) {
          reinterpret_cast<uint4*>(tr)[0] = make_uint4(w[0], w[1], w[2], w[3]);
          reinterpret_cast<uint4*>(tr)[1] = make_uint4(w[4], w[5], w[6], w[7]);
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (j < left) tr[j] = __ushort_as_bfloat16((unsigned short)((j & 1) ? (w[j >> 1] >> 16) : (w[j >> 1] & 0xFFFFu)));
        }
      }
    }
    // code slots between the last head's blocks and the end of the last 64-slot chunk: zero codes under zero scales
    if (row_ok && a.codes && h == g.H - 1) {
      for (int slot = g.q_len; slot < g.k_pad; slot += 16)
        *reinterpret_cast<uint2*>(a.codes + row * g.code_row_bytes + (slot >> 1)) = make_uint2(0u, 0u);
    }
  }
}

// Plain GEMM epilogue: y[M, N] = acc (+ bias) as bf16; used for the stand-alone rotation and for
// the bf16 GEMM behind the W4A16 layer.  32 columns at a time: tcgen05.ld -> + bias -> bf16 -> the warp's 32 x 32
// staging patch in shared memory (64-byte rows, 64-byte swizzle) -> one TMA store, which clips the patch at the
// edges of y.  (A row-per-thread store straight to global memory puts 32 separate 16-byte segments per
// instruction through the load/store unit.)
__device__ __forceinline__ void epi_rot_only(const RotArgs& a, const CUtensorMap* tm_y, uint32_t stg, uint32_t taddr, int row0,
                                             int lane, int n0, int half, uint32_t& turn, int wpq = 2) {
  const ActGeom& g = a.g;
  const uint32_t stg_row = stg + lane * 64;
  const int sw = (lane >> 1) & 3;
  for (int c0 = 0; c0 < a.BN; c0 += 32) {
    const int col = n0 + c0;
    if (col >= g.D) break;
    if (((turn++) % (uint32_t)wpq) != (uint32_t)half) continue;
    uint32_t r[32];
    tmem_ld32(taddr + c0, r);
    tmem_wait_ld();
    if (lane == 0) bulk_wait_read0();              // the previous patch has left the staging buffer
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float f[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(r[8 * i + e]);
      if (a.bias && col + 8 * i + 8 <= g.D) {
        const uint4 bb = __ldg(reinterpret_cast<const uint4*>(a.bias + col + 8 * i));
        const __nv_bfloat162* bh = reinterpret_cast<const __nv_bfloat162*>(&bb);
#pragma unroll
        for (int e2 = 0; e2 < 4; ++e2) {
          const float2 b2 = __bfloat1622float2(bh[e2]);
          f[2 * e2] += b2.x;
          f[2 * e2 + 1] += b2.y;
        }
      }
      asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(stg_row + (uint32_t)((i ^ sw) << 4)),
                   "r"(pack_bf16x2(f[0], f[1])), "r"(pack_bf16x2(f[2], f[3])), "r"(pack_bf16x2(f[4], f[5])),
                   "r"(pack_bf16x2(f[6], f[7]))
                   : "memory");
    }
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0 && row0 < a.M) {
      tma_store_2d(tm_y, stg, col, row0);
      bulk_commit_group();
    }
  }
}

// PAIR: clusters of two CTAs share one 256-row tile through tcgen05.mma.cta_group::2 (each CTA its own 128 token
// rows and half of the rotation tile); completions of both CTAs' loads are counted on the leader's full barrier, the
// leader commits to both CTAs' empty / accumulator-full barriers, epilogue warps of both arrive on the leader's
// accumulator-empty barrier (the peer's arrivals carry no memory ordering: their payload is tensor memory).
template <int EPI, int MODE, bool PAIR, int UNITS>
__global__ void __launch_bounds__(RqCfg<EPI>::THREADS, 1)
rotate_quant_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_u,
                    const __grid_constant__ CUtensorMap tm_y, const RotArgs a) {
  using Stage = RqStage<PAIR, UNITS>;
  constexpr int RQ_STAGES = Stage::STAGES, RQ_STAGE_BYTES = Stage::STAGE_BYTES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* stg_area = smem + RQ_STAGES * RQ_STAGE_BYTES;                  // 1024-byte aligned
  uint64_t* bars = reinterpret_cast<uint64_t*>(stg_area + RqCfg<EPI>::STG_BYTES);
  static_assert((2 * RQ_STAGES + 4) * 8 + 4 + AB_WORDS * 4 <= 256, "barrier area");
  // bars[0..S) full, [S..2S) empty, [2S..2S+2) acc_full, [2S+2..2S+4) acc_empty
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * RQ_STAGES + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = PAIR ? cluster_ctarank() : 0u;      // 0 = leader (issues the UMMAs)
  const uint32_t bar0 = smem_u32(bars);
  auto full_bar = [&](int s) { return bar0 + 8u * s; };
  auto empty_bar = [&](int s) { return bar0 + 8u * (RQ_STAGES + s); };
  auto accf_bar = [&](int b) { return bar0 + 8u * (2 * RQ_STAGES + b); };
  auto acce_bar = [&](int b) { return bar0 + 8u * (2 * RQ_STAGES + 2 + b); };
  const uint32_t abort_addr = bar0 + 8u * (2 * RQ_STAGES + 4) + 4u;

  if (threadIdx.x == 0) {
    for (int s = 0; s < RQ_STAGES; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(accf_bar(b), 1); mbar_init(acce_bar(b), (PAIR ? 2 : 1) * RqCfg<EPI>::EPI_WARPS); }
    abort_init(abort_flag, a.wait_limit_k, PAIR ? map_to_rank(abort_addr, rank ^ 1) : 0u);
    fence_mbar_init();
    prefetch_tmap(&tm_x);
    prefetch_tmap(&tm_u);
  }
  if (warp == 1) {
    if constexpr (PAIR) tmem_alloc_pair(smem_u32(tmem_slot), 512);
    else tmem_alloc(smem_u32(tmem_slot), 512);
  }
  tc_fence_before();
  __syncthreads();
  if constexpr (PAIR) cluster_sync_all();   // both CTAs' barriers exist before anything arrives on them remotely
  tc_fence_after();
  pdl_launch_dependents();
  pdl_wait();                       // whatever produced x (and last used the output buffers) has completed
  const uint32_t tmem_base = *tmem_slot;
  // tiles: (128-row block, column block), or (256-row pair block, column block) walked by clusters
  const int total_tiles = (PAIR ? (a.m_tiles + 1) / 2 : a.m_tiles) * a.n_tiles;
  const int first = PAIR ? (int)cluster_id_x() : (int)blockIdx.x, step = PAIR ? (int)cluster_count_x() : (int)gridDim.x;
  const int bn_own = PAIR ? a.BN / 2 : a.BN;                 // rotation-tile rows this CTA fetches
  const uint32_t smem_base = smem_u32(smem), stage_tx = UNITS * (RQ_A_BYTES + bn_own * 128);   // a CTA's bytes per stage

  if (warp == 0) {
    int s = 0;
    uint32_t ph = 0;
    int issued = 0;
    bool ok = true;
    for (int t = first; t < total_tiles && ok; t += step) {
      int mt, nb;
      tile_at(a, t, mt, nb);
      const int mb = PAIR ? 2 * mt + (int)rank : mt;
      const int row_u = nb * a.BN + (int)rank * (tile_width(a, nb) >> 1);   // of a pair, each CTA fetches half of the tile's rows
      int kb, ke;
      tile_k_range(a, nb, kb, ke);
      for (int kc = kb; kc < ke; kc += UNITS) {
        if (!mbar_wait_hot_warp(empty_bar(s), ph ^ 1, abort_flag, a.status, ERR_WAIT_EMPTY)) { ok = false; break; }
        if (elect_one()) {
          const uint32_t sa = smem_base + s * RQ_STAGE_BYTES, fb = PAIR ? map_to_rank(full_bar(s), 0) : full_bar(s);
          if (rank == 0) mbar_expect_tx(full_bar(s), (PAIR ? 2u : 1u) * stage_tx);
#pragma unroll
          for (int u = 0; u < UNITS; ++u) {
            const int x = (UNITS == 1 ? kc : min(kc + u, ke - 1)) * 64;    // past the last unit: the last one again, which no UMMA reads
            const uint32_t su = sa + u * Stage::UNIT_BYTES;
            if constexpr (PAIR) {
              tma_load_2d_pair(su, &tm_x, fb, x, mb * 128);
              tma_load_2d_pair(su + RQ_A_BYTES, &tm_u, fb, x, row_u);
            } else {
              tma_load_2d(su, &tm_x, fb, x, mb * 128);
              tma_load_2d(su + RQ_A_BYTES, &tm_u, fb, x, row_u);
            }
          }
        }
        __syncwarp();
        ++issued;
        if (++s == RQ_STAGES) { s = 0; ph ^= 1; }
      }
    }
    if (lane == 0) abort_flag[AB_ISSUED] = issued;
  } else if (warp == 1) {
    if (rank == 0) {
      int s = 0, buf = 0, stages = 0, accs = 0;
      uint32_t ph = 0, aph = 0;
      bool ok = true, ready = false;                       // ready: the next stage is known to be full
      const uint64_t op_d0 = smem_desc_sw128(smem_base);
      const uint32_t op_lo0 = (uint32_t)op_d0, op_hi = (uint32_t)(op_d0 >> 32);
      for (int t = first; t < total_tiles && ok; t += step) {
        int mt, nb;
        tile_at(a, t, mt, nb);
        const uint32_t idesc = idesc_dense(ACC_F32, FMT_BF16, FMT_BF16, PAIR ? 256 : 128, (uint32_t)tile_width(a, nb));
        int kb, ke;
        tile_k_range(a, nb, kb, ke);
        if (!mbar_wait_hot_warp(acce_bar(buf), aph ^ 1, abort_flag, a.status, ERR_WAIT_ACC_EMPTY)) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + buf * 256;
        for (int kc = kb; kc < ke; kc += UNITS) {
          if (!ready && !mbar_wait_hot_warp(full_bar(s), ph, abort_flag, a.status, ERR_WAIT_FULL)) { ok = false; break; }
          tc_fence_after();
          // descriptors from loop-invariant words; the stage's four UMMAs, their commit and a test of the next stage's barrier in
          // one block (what this warp does between UMMAs is time the tensor pipe idles)
          uint32_t a_lo = op_lo0 + (uint32_t)s * (RQ_STAGE_BYTES >> 4), acc = kc > kb ? 1u : 0u;
          const uint32_t done = empty_bar(s);
          if (++s == RQ_STAGES) { s = 0; ph ^= 1; }
          uint32_t next = 0u;
          if (elect_one()) {
            if (UNITS == 2 && kc + 2 <= ke) {
              if constexpr (PAIR) umma_f16_ss_x4_pair(d_tmem, a_lo, a_lo + (RQ_A_BYTES >> 4), op_hi, idesc, acc);
              else umma_f16_ss_x4(d_tmem, a_lo, a_lo + (RQ_A_BYTES >> 4), op_hi, idesc, acc);
              a_lo += Stage::UNIT_BYTES >> 4;
              acc = 1u;
            }
            if constexpr (PAIR) next = umma_f16_ss_stage_pair(d_tmem, a_lo, a_lo + (RQ_A_BYTES >> 4), op_hi, idesc, acc, done, full_bar(s), ph);
            else next = umma_f16_ss_stage(d_tmem, a_lo, a_lo + (RQ_A_BYTES >> 4), op_hi, idesc, acc, done, full_bar(s), ph);
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
        ++accs;
        buf ^= 1;
        if (buf == 0) aph ^= 1;
      }
      if (lane == 0) {
        abort_flag[AB_UMMA] = stages;
        abort_flag[AB_ACC] = accs;
      }
    }
  } else {
    const int q = warp & 3, half = (warp - 2) >> 2;
    int buf = 0;
    uint32_t aph = 0, turn = 0;
    const uint32_t acce_leader = PAIR ? map_to_rank(acce_bar(0), 0) : 0u;
    for (int t = first; t < total_tiles; t += step) {
      int mt, nb;
      tile_at(a, t, mt, nb);
      const int mb = PAIR ? 2 * mt + (int)rank : mt;
      if (!mbar_wait_warp(accf_bar(buf), aph, abort_flag, a.status, ERR_WAIT_ACC_FULL)) break;
      tc_fence_after();
      const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + buf * 256;
      const int64_t row = (int64_t)mb * 128 + q * 32 + lane;
      const int n0 = nb * a.BN;
      if constexpr (EPI == EPI_ROT_ONLY)
        epi_rot_only(a, &tm_y, smem_u32(stg_area) + (warp - 2) * RqCfg<EPI>::STG_WARP, taddr, mb * 128 + q * 32, lane, n0, half, turn);
      else if constexpr (EPI == EPI_INT_HIDDEN) epi_int_hidden<MODE>(a, taddr, row, n0, half, turn);
      else if constexpr (EPI == EPI_NVFP4_HIDDEN) epi_nvfp4_hidden<MODE>(a, taddr, row, n0, half, turn, RqCfg<EPI>::WPQ);
      else if constexpr (EPI == EPI_NVFP4_PERHEAD) epi_nvfp4_perhead(a, taddr, row, n0, half, turn, RqCfg<EPI>::WPQ);
      else epi_int_perhead<MODE>(a, taddr, row, lane, n0, half, turn, smem_u32(stg_area) + (warp - 2) * RqCfg<EPI>::STG_WARP);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (PAIR && rank != 0) mbar_arrive_cluster_relaxed(acce_leader + 8u * buf);
        else mbar_arrive(acce_bar(buf));
      }
      buf ^= 1;
      if (buf == 0) aph ^= 1;
    }
    if constexpr (EPI == EPI_ROT_ONLY)
      if (lane == 0) bulk_wait_all0();                 // the output is in global memory before the CTA retires
  }
  tc_fence_before();
  __syncthreads();
  if constexpr (PAIR) cluster_sync_all();   // neither CTA retires while the other may still read its shared memory
  if (abort_flag[AB_FLAG]) {        // a wait ran out (in both CTAs of a pair the flag is up): await what is in flight
    if (warp == 0 && lane == 0) {
      const int own = abort_flag[AB_ISSUED];
      if constexpr (PAIR) {
        const int peer = ld_cluster_s32(map_to_rank(abort_addr + 4u * AB_ISSUED, rank ^ 1));
        if (rank == 0) drain_pair_ring(full_bar, RQ_STAGES, own, peer, max(own, peer), [&](int) -> uint32_t { return stage_tx; }, a.status);
      } else {
        drain_ring(full_bar, RQ_STAGES, own, a.status);
      }
    }
    if (warp == 1 && lane == 0) {                       // in both CTAs of a pair, where the leader's commits arrive
      int stages = abort_flag[AB_UMMA], accs = abort_flag[AB_ACC];
      if constexpr (PAIR) {
        const uint32_t lead = map_to_rank(abort_addr, 0);
        stages = ld_cluster_s32(lead + 4u * AB_UMMA);
        accs = ld_cluster_s32(lead + 4u * AB_ACC);
      }
      drain_ring(empty_bar, RQ_STAGES, stages, a.status);
      drain_ring(accf_bar, 2, accs, a.status);
    }
    __syncwarp();
    __syncthreads();
    if constexpr (PAIR) cluster_sync_all();
  }
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    if constexpr (PAIR) tmem_dealloc_pair(tmem_base, 512);
    else tmem_dealloc(tmem_base, 512);
  }
}

// ---- host side ----------------------------------------------------------------------------------
int num_sms() {
  // per device: a process may drive GPUs of different sizes
  static std::atomic<int> cache[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  int n = cache[dev].load(std::memory_order_relaxed);
  if (n <= 0) {
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    cache[dev].store(n, std::memory_order_relaxed);
  }
  return n;
}

template <int EPI, int MODE, bool PAIR, int UNITS>
static int launch_rq_impl(const CUtensorMap& tx, const CUtensorMap& tu, const CUtensorMap& ty, const RotArgs& a, cudaStream_t st) {
  using Cfg = RqCfg<EPI, PAIR, UNITS>;
  auto k = rotate_quant_kernel<EPI, MODE, PAIR, UNITS>;
  static PerDeviceOnce attr_once;
  if (int rc = set_max_dynamic_smem(attr_once, k, Cfg::SMEM_BYTES)) return rc;
  if constexpr (!PAIR) {
    const int grid = min(a.m_tiles * a.n_tiles, num_sms());
    return launch_pdl(k, dim3(grid), dim3(Cfg::THREADS), Cfg::SMEM_BYTES, st, tx, tu, ty, a) == cudaSuccess ? DIROTQ_OK : DIROTQ_E_CUDA;
  } else {
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
    const int tiles = ((a.m_tiles + 1) / 2) * a.n_tiles;
    cfg.gridDim = dim3(2 * min(tiles, max_pairs));
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, k, tx, tu, ty, a) == cudaSuccess ? DIROTQ_OK : DIROTQ_E_CUDA;
  }
}

// tu_pair: the rotation's tensor map with a box of BN / 2 rows (what one CTA of a pair fetches); used when the call
// has more than one 128-row block (DIROTQ_ROTATE_TILE = single | pair forces one form: measurements, tests).
template <int EPI, int MODE>
static int launch_rq(const CUtensorMap& tx, const CUtensorMap& tu, const CUtensorMap& tu_pair, const RotArgs& a, cudaStream_t st) {
  CUtensorMap ty = tx;                                 // only the plain-GEMM epilogue stores through a tensor map
  if constexpr (EPI == EPI_ROT_ONLY) {
    if ((a.g.D & 7) || (reinterpret_cast<uintptr_t>(a.x_rot) & 15)) return DIROTQ_E_ALIGN;
    int rc = make_tmap_2d_sw(&ty, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, a.x_rot, (uint64_t)a.g.D, (uint64_t)a.M,
                             (uint64_t)a.g.D * 2, 32, 32, 64);
    if (rc) return rc;
  }
  bool pair = a.m_tiles >= 2 && (a.BN / 2) % 8 == 0;
  if (const char* e = getenv("DIROTQ_ROTATE_TILE")) {
    if (!strcmp(e, "single")) pair = false;
    else if (!strcmp(e, "pair")) pair = (a.BN / 2) % 8 == 0;
  }
  if constexpr (EPI == EPI_ROT_ONLY || EPI == EPI_INT_HIDDEN || EPI == EPI_NVFP4_HIDDEN)
    if (a.BN <= 128 && a.band == 0)
      return pair ? launch_rq_impl<EPI, MODE, true, 2>(tx, tu_pair, ty, a, st) : launch_rq_impl<EPI, MODE, false, 2>(tx, tu, ty, a, st);
  return pair ? launch_rq_impl<EPI, MODE, true, 1>(tx, tu_pair, ty, a, st) : launch_rq_impl<EPI, MODE, false, 1>(tx, tu, ty, a, st);
}

// The last column of tiles is only as wide as D needs, rounded up to 64 (1152 columns were five tiles of 256, and are four and a
// half): 32768 x 1152 63.9 -> 62.3 us, 32768 x 4608 -> 1152 in bf16 246 -> 242.  The shared-memory pipe, which the operands
// pass twice, keeps the gain below the UMMAs saved.
static int last_width(int D, int bn) {
  const int w = ((D % bn) + 63) & ~63;
  return w == 0 || w > bn ? bn : w;
}
// Picks the N tile.  Per-head layouts: a whole number of heads (and a multiple of 16 for the UMMA shape).  Hidden layouts and
// plain GEMMs: the persistent grid runs whole rounds over 74 CTA pairs; a round takes 190 / 255 / 335 ns per 64-wide unit of K (128 / 192 /
// 256 columns) and 0.25 / 0.9 / 0.4 us besides, a call 5.3 / 4.6 / 5.8 us, and a tile of the last column saves 0.44 of the columns it
// lacks.  The smallest sum is taken; measured (us, 128 / 192 / 256): rotation of 4096 x 1152 12.7 / 14.3 / 16.8, 6000 x 1152 16.0 / 15.6 /
// 18.0, 16384 x 1152 33.6 / 33.6 / 35.2, 32768 x 1152 66.4 / 61.9 / 61.4, 2048 x 2240 19.3 / 24.2 / 18.8, 4096 x 2240 32.8 / 33.6 / 30.7, 4608 x 3072
// 59.0 / 55.7 / 56.9, 16384 x 3072 214 / 201 / 198; bf16 4096 x 4608 -> 1152 31.9 / 40.1 / 49.6, 32768 rows 254 / 237 / 241, 1024 x 12288 ->
// 3072 77.8 / 56.1 / 70.0.
int pick_bn(const ActGeom& g, int64_t M, int64_t K) {
  if (g.H > 0) {
    int best = 0;
    for (int k = 1; k * g.d <= 256; ++k)
      if ((k * g.d) % 16 == 0) best = k * g.d;
    return best;
  }
  static const int width[3] = {128, 192, 256}, unit_ns[3] = {190, 255, 335}, tile_ns[3] = {250, 900, 400}, call_ns[3] = {5300, 4600, 5800};
  const int64_t m_pairs = (M + 255) / 256, pairs = num_sms() / 2, units = (K + 63) / 64;
  int best = 128;
  int64_t best_ns = -1;
  for (int i = 0; i < 3; ++i) {
    const int64_t n_tiles = ceil_div(g.D, width[i]), rounds = (m_pairs * n_tiles + pairs - 1) / pairs;
    const int64_t lacks = width[i] - last_width(g.D, width[i]);
    const int64_t ns = rounds * (units * unit_ns[i] + tile_ns[i]) + call_ns[i] - rounds / n_tiles * units * unit_ns[i] * lacks * 44 / (100 * width[i]);
    if (best_ns < 0 || ns < best_ns) { best_ns = ns; best = width[i]; }
  }
  return best;
}

static void ragged_masks(const ActGeom& g, RotArgs& a) {
  const int nv = g.group & 31;
  a.ragged = nv != 0;
  for (int j = 0; j < 32 && nv; ++j) {
    if (j >= nv) continue;
    a.pair_mask[j >> 1] |= 0xFFFFu << (16 * (j & 1));
    if (g.mode == DIROTQ_INT8_ASYM) a.code_mask[j >> 2] |= 0xFFu << (8 * (j & 3));
    else a.code_mask[(j & 15) >> 2] |= (j < 16 ? 0xFu : 0xF0u) << (8 * (j & 3));
  }
}

int launch_rotate_quantize(const ActGeom& g, const void* x, const void* rot_t, int64_t M, RotArgs a, cudaStream_t st) {
  if (M <= 0) return DIROTQ_OK;
  a.g = g;
  a.M = M;
  a.K = g.D;
  a.bias = nullptr;
  a.ldm = ld_rows(M);
  const bool rot_only = a.codes == nullptr;
  if (rot_only && !a.x_rot) return DIROTQ_E_ARG;
  // The rotation-only epilogue stores whole 32-column patches, so it takes the tile widths of the hidden layouts even
  // under a per-head rotation (whose whole-head widths, 144 for 72-wide heads, are not multiples of 32); the K range of
  // a tile follows the heads its columns touch either way.
  ActGeom g_tile = g;
  if (rot_only) g_tile.H = 0;
  a.BN = pick_bn(g_tile, M, g.D);
  if (a.BN <= 0) return DIROTQ_E_UNSUPPORTED;
  a.n_tiles = ceil_div(g.D, a.BN);
  a.bn_last = last_width(g.D, a.BN);
  a.m_tiles = (int)((M + 127) / 128);
  a.band = g.H > 0 ? g.d : 0;
  if (!rot_only && g.H > 0) {
    // 32-column TMEM reads of a head's group must stay inside the head
    if (((g.group + 31) / 32) * 32 > g.d) return DIROTQ_E_UNSUPPORTED;
    ragged_masks(g, a);
  }
  if (!rot_only && g.H == 0 && !is_nvfp4(g.mode) && g.group != 64) return DIROTQ_E_UNSUPPORTED;
  if (!rot_only && g.per_token) return DIROTQ_E_UNSUPPORTED;     // a row's scale needs the whole rotated row: rotate, then quantise
  CUtensorMap tx, tu;
  int rc = make_tmap_2d(&tx, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, x, (uint64_t)g.D, (uint64_t)M, (uint64_t)g.D * 2, 128);
  if (rc) return rc;
  rc = make_tmap_2d(&tu, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, rot_t, (uint64_t)g.D, (uint64_t)g.D, (uint64_t)g.D * 2,
                    (uint32_t)a.BN);
  if (rc) return rc;
  CUtensorMap tu2 = tu;
  if ((a.BN / 2) % 8 == 0) {
    rc = make_tmap_2d(&tu2, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, rot_t, (uint64_t)g.D, (uint64_t)g.D, (uint64_t)g.D * 2,
                      (uint32_t)(a.BN / 2));
    if (rc) return rc;
  }
  if (rot_only) return launch_rq<EPI_ROT_ONLY, 0>(tx, tu, tu2, a, st);
  if (g.H > 0) {
    switch (g.mode) {
      case DIROTQ_INT4_SYM: return launch_rq<EPI_INT_PERHEAD, MODE_INT4_SYM>(tx, tu, tu2, a, st);
      case DIROTQ_INT4_ASYM: return launch_rq<EPI_INT_PERHEAD, MODE_INT4_ASYM>(tx, tu, tu2, a, st);
      case DIROTQ_INT8_ASYM: return launch_rq<EPI_INT_PERHEAD, MODE_INT8_ASYM>(tx, tu, tu2, a, st);
      case DIROTQ_NVFP4_HW: return launch_rq<EPI_NVFP4_PERHEAD, MODE_NVFP4_HW>(tx, tu, tu2, a, st);
      default: return DIROTQ_E_UNSUPPORTED;
    }
  }
  switch (g.mode) {
    case DIROTQ_INT4_SYM: return launch_rq<EPI_INT_HIDDEN, MODE_INT4_SYM>(tx, tu, tu2, a, st);
    case DIROTQ_INT4_ASYM: return launch_rq<EPI_INT_HIDDEN, MODE_INT4_ASYM>(tx, tu, tu2, a, st);
    case DIROTQ_INT8_ASYM: return launch_rq<EPI_INT_HIDDEN, MODE_INT8_ASYM>(tx, tu, tu2, a, st);
    case DIROTQ_NVFP4_REF: return launch_rq<EPI_NVFP4_HIDDEN, MODE_NVFP4_REF>(tx, tu, tu2, a, st);
    case DIROTQ_NVFP4_HW: return launch_rq<EPI_NVFP4_HIDDEN, MODE_NVFP4_HW>(tx, tu, tu2, a, st);
  }
  return DIROTQ_E_UNSUPPORTED;
}

// y[M, N] = x[M, K] @ w_t[N, K]^T (+ bias), all bf16, fp32 accumulation on tcgen05.
int launch_gemm_bf16(const void* x, const void* w_t, int64_t M, int64_t N, int64_t K, const void* bias, void* y,
                     int* status, cudaStream_t st) {
  if (M <= 0) return DIROTQ_OK;
  if (N % 8 || K % 8) return DIROTQ_E_UNSUPPORTED;
  RotArgs a{};
  a.g = ActGeom{};
  a.g.D = (int)N;
  a.M = M;
  a.K = (int)K;
  a.ldm = ld_rows(M);
  a.BN = pick_bn(a.g, M, K);
  a.n_tiles = ceil_div((int)N, a.BN);
  a.bn_last = last_width((int)N, a.BN);
  a.m_tiles = (int)((M + 127) / 128);
  a.band = 0;
  a.x_rot = static_cast<__nv_bfloat16*>(y);
  a.bias = static_cast<const __nv_bfloat16*>(bias);
  a.status = status;
  a.wait_limit_k = wait_limit_k();
  CUtensorMap tx, tu;
  int rc = make_tmap_2d(&tx, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, x, (uint64_t)K, (uint64_t)M, (uint64_t)K * 2, 128);
  if (rc) return rc;
  rc = make_tmap_2d(&tu, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, w_t, (uint64_t)K, (uint64_t)N, (uint64_t)K * 2, (uint32_t)a.BN);
  if (rc) return rc;
  CUtensorMap tu2;
  rc = make_tmap_2d(&tu2, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, w_t, (uint64_t)K, (uint64_t)N, (uint64_t)K * 2, (uint32_t)(a.BN / 2));
  if (rc) return rc;
  return launch_rq<EPI_ROT_ONLY, 0>(tx, tu, tu2, a, st);
}

}  // namespace dq
