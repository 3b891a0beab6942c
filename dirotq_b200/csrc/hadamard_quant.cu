// Front end of a Hadamard layer in one pass: transform of the leading n channels (hadamard.cu's arithmetic, stage by stage, so
// bit-identical to it and to the reference's butterflies), quantisation of exactly those channels (quantize.cu's arithmetic on
// the bf16-rounded result), the other channels copied to the 16-bit operand.  Reads each input once and writes codes: the
// separate kernels write the transformed tensor and read it back.
//
// A warp owns 32 blocks of B channels, one block a lane: one row of 4096 (B = 128) or 2048 (B = 64), two rows of 1024.  The
// stages inside a block are register arithmetic; then the 32 lanes trade blocks for columns through shared memory, 64 columns
// of every block at a time, and the remaining stages run over the blocks of a row, on pairs of neighbouring columns.  One
// exchange instead of two, no barrier beyond the warp's, and packed fp32 pairs (add / sub .f32x2) for all but one stage.  The
// bf16 result goes through the same buffer once more, so that a lane quantises whole 64-channel chunks without shuffles and
// writes their codes as full sectors.  The next row arrives by asynchronous copies meanwhile.  All buffers have their blocks
// 16 bytes further apart than their length: every access below is free of bank conflicts.
//
// Bound by instruction issue and the shared-memory pipe together (n = 4096, 18432 rows: 53 % of issue slots, 60 % of the
// pipe's wavefronts, 31 % of DRAM); 12 warps of 168 registers a multiprocessor, 16 of 128 for the shorter rows.  Transform and
// quantiser, separate launches -> this one, us, for 4-bit symmetric / asymmetric / 8-bit / NVFP4 codes:
//   4096 rows, n = 1024 of 1152    10.4 ->  6.6   10.9 ->  7.1   11.6 ->  7.7   13.3 ->  6.9
//              n = 2048 of 2240    18.1 -> 12.1   19.3 -> 13.2   20.0 -> 15.0   19.8 -> 12.9
//              n = 4096 of 4608    33.7 -> 20.2   36.0 -> 23.9   37.7 -> 26.9   34.5 -> 21.8
//   18432 rows, n = 4096            141 -> 80      150 -> 93      161 -> 105     158 -> 80
//   256 rows, n = 1024              5.7 ->  3.4    6.0 ->  3.7    6.3 ->  4.5    6.3 ->  3.6
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include "layout.cuh"
#include "launchers.cuh"
#include "ptx.cuh"
#include "quant_math.cuh"

namespace dq {

template <int LOGN>
struct HqCfg {
  static constexpr int N = 1 << LOGN;
  static constexpr int L = LOGN >= 11 ? 32 : N / 64;      // lanes per row
  static constexpr int B = N / L;                         // channels per lane
  static constexpr int ROWS = 32 / L;                     // rows per warp
  static constexpr int HALVES = B / 64;                   // exchanges of 64 columns
  static constexpr int COLS = 64 / L;                     // columns per lane and exchange
  static constexpr int IN_PITCH = 2 * B + 16;             // bytes between blocks of bf16 values
  static constexpr int XCH_PITCH = 64 * 4 + 16;           // ... and of fp32 columns
  static constexpr int IN_BYTES = 32 * IN_PITCH, XCH_BYTES = 32 * XCH_PITCH, FLIP_BYTES = L * IN_PITCH;
  static constexpr int WARPS = B == 128 ? 12 : 16;        // 168 or 128 registers a thread
  static constexpr int SMEM = FLIP_BYTES + WARPS * (IN_BYTES + XCH_BYTES);
  static_assert(B == 64 || B == 128, "blocks of one or two chunks");
  static_assert(XCH_BYTES >= 32 * IN_PITCH, "the bf16 result passes through the exchange buffer");
  static_assert(SMEM <= 227 * 1024, "one block per multiprocessor");
};

__device__ __forceinline__ uint64_t pair_f32(uint32_t lo, uint32_t hi) { return ((uint64_t)hi << 32) | lo; }
__device__ __forceinline__ void butterfly2(uint64_t& p, uint64_t& q) {
  uint64_t s, d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(s) : "l"(p), "l"(q));
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(p), "l"(q));
  p = s;
  q = d;
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ uint4 lds128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void sts128(uint32_t a, uint4 v) {
  asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(a), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

// One chunk of 64 channels as packed pairs -> its codes, scale and zero point (quantize.cu: packed_path, groups of 64; for
// NVFP4 the whole-chunk path).
template <int MODE>
__device__ __forceinline__ void quantise_chunk(const QuantArgs& a, const uint32_t* w, int64_t row, int chunk, int n_kb64_pad) {
  const ActGeom& g = a.g;
  if constexpr (MODE == MODE_NVFP4_HW) {
    uint2 c[4];
    uint32_t sfw = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) sfw |= (uint32_t)nvfp4_hw_group(w + 8 * i, g.clip, g.T, c[i]) << (8 * i);
    st_global_32(a.codes + row * g.code_row_bytes + (int64_t)chunk * 32, make_uint4(c[0].x, c[0].y, c[1].x, c[1].y),
                 make_uint4(c[2].x, c[2].y, c[3].x, c[3].y));
    *reinterpret_cast<uint32_t*>(a.sf + sf_offset(row, chunk * 4, n_kb64_pad)) = sfw;
  } else {
    constexpr float maxq = MODE == MODE_INT4_SYM ? 7.f : (MODE == MODE_INT4_ASYM ? 15.f : 255.f);
    float mx = -INFINITY, mn = INFINITY;
    GroupParams p;
    if constexpr (MODE == MODE_INT4_SYM) {
#pragma unroll
      for (int i = 0; i < 4; ++i) mx = fmaxf(mx, amax_bf16x16(w + 8 * i));
      mn = -mx;
      p = int_sym_params<true>(mx, mn, g.clip, maxq);
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) minmax_bf16x16(w + 8 * i, mx, mn);
      p = int_asym_params<true>(mx, mn, g.clip, maxq);
    }
    const float rcp = __frcp_rn(p.scale);
    if constexpr (MODE == MODE_INT8_ASYM) {
      uint8_t* dst = a.codes + row * g.code_row_bytes + (int64_t)chunk * 64;
      const bool packs = int_asym_packs8(mx, mn, rcp, p.zero);
#pragma unroll
      for (int i = 0; i < 2; ++i)
        st_global_32(dst + 32 * i, int_asym_byte16_packed(w + 16 * i, p.scale, rcp, p.zero, packs),
                     int_asym_byte16_packed(w + 16 * i + 8, p.scale, rcp, p.zero, packs));
    } else {
      uint4 c[2];
#pragma unroll
      for (int i = 0; i < 2; ++i)
        c[i] = MODE == MODE_INT4_SYM ? int_sym_planar32_packed(w + 16 * i, rcp, g.clip < 1.f)
                                     : int_asym_planar32(w + 16 * i, p.scale, rcp, p.zero, int_asym_packs(mx, mn, rcp, p.zero));
      st_global_32(a.codes + row * g.code_row_bytes + (int64_t)chunk * 32, c[0], c[1]);
    }
    a.scales[(int64_t)chunk * a.ldm + row] = __float2bfloat16_rn(p.scale);
    if constexpr (MODE != MODE_INT4_SYM) a.zeros[(int64_t)chunk * a.ldm + row] = __float2bfloat16_rn(p.zero);
  }
}

// Eight pairs times 1 / sqrt(n), rounded to bf16 as the reference rounds the fp32 quotient v / sqrt(n).  EXACT (n a power of
// four): a scaling.  Else the product q = v fl(1 / sqrt(n)) stands for the quotient d = fl(v / sqrt(n)): the reciprocal, the
// product and the quotient are each off by a factor within 1 +- 2^-24, so q and d are at most three units in the last place of
// fp32 apart (two among subnormal results), and both round to the same bf16 value unless q lies within that of the middle
// between two of them, 0x8000 in its low half.  Then, for one value in 7000, the division itself decides.
template <bool EXACT>
__device__ __forceinline__ void normalise8(const uint64_t* s, float norm, float inv_norm, uint32_t* o) {
  const uint64_t inv2 = twice_f32(inv_norm);
  uint32_t nearest = 0xFFFFFFFFu;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const uint64_t m = mul_f32x2((uint32_t)s[i], (uint32_t)(s[i] >> 32), inv2);
    const uint32_t m0 = (uint32_t)m, m1 = (uint32_t)(m >> 32);
    if constexpr (!EXACT) nearest = min(nearest, min(m0 * 65536u - 0x7FFC0000u, m1 * 65536u - 0x7FFC0000u));
    const __nv_bfloat162 b = __floats2bfloat162_rn(__uint_as_float(m0), __uint_as_float(m1));
    o[i] = *reinterpret_cast<const uint32_t*>(&b);
  }
  if constexpr (!EXACT) {
    if (nearest <= 0x00080000u) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const __nv_bfloat162 b = __floats2bfloat162_rn(__fdiv_rn(__uint_as_float((uint32_t)s[i]), norm),
                                                       __fdiv_rn(__uint_as_float((uint32_t)(s[i] >> 32)), norm));
        o[i] = *reinterpret_cast<const uint32_t*>(&b);
      }
    }
  }
}

template <int LOGN, int MODE>
__global__ void __launch_bounds__(HqCfg<LOGN>::WARPS * 32, 1)
hadamard_quant_kernel(const QuantArgs a, const __nv_bfloat16* __restrict__ flips, float norm, float inv_norm) {
  using C = HqCfg<LOGN>;
  constexpr int B = C::B, L = C::L, THREADS = C::WARPS * 32;
  extern __shared__ __align__(16) uint8_t hq_smem[];
  const ActGeom& g = a.g;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int l = lane % L, rr = lane / L;
  const uint32_t flip_s = smem_u32(hq_smem), in_s = flip_s + C::FLIP_BYTES + warp * (C::IN_BYTES + C::XCH_BYTES),
                 xch_s = in_s + C::IN_BYTES;
  const int64_t units = (a.M + C::ROWS - 1) / C::ROWS, step = (int64_t)gridDim.x * C::WARPS;
  const int n_kb64_pad = (g.n_chunks + 3) & ~3;
  const int per_row = a.tail ? g.tail_pitch >> 3 : 0;     // 16-byte pieces of the channels that keep 16 bits

  auto fetch = [&](int64_t u) {                           // the rows of unit u, each piece of 8 channels to its block's place
#pragma unroll
    for (int k = 0; k < B / 8; ++k) {
      const int p = 32 * k + lane, r = p / (C::N / 8);
      const int64_t row = u * C::ROWS + r;
      if (row < a.M)
        cp_async16(in_s + (p / (B / 8)) * C::IN_PITCH + 16 * (p % (B / 8)), a.x + row * a.x_pitch + 8 * (p - r * (C::N / 8)));
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto tail_piece = [&](int64_t u, int i, int64_t& at) {  // piece i of the unit's rows: its value, and its place or -1
    const int r = C::ROWS == 1 ? 0 : i / per_row, t = (i - r * per_row) * 8;
    const int64_t row = u * C::ROWS + r;
    at = r < C::ROWS && i < C::ROWS * per_row && row < a.M ? row * g.tail_pitch + t : -1;
    if (at < 0 || t >= g.tail_total) return make_uint4(0u, 0u, 0u, 0u);
    return __ldg(reinterpret_cast<const uint4*>(a.x + row * a.x_pitch + g.q_len + t));
  };

  pdl_launch_dependents();
  pdl_wait();
  int64_t u = (int64_t)warp * gridDim.x + blockIdx.x;     // neighbouring units on different multiprocessors: short calls spread
  if (u < units) fetch(u);
  if (flips) {
    for (int p = threadIdx.x; p < C::N / 8; p += THREADS)
      sts128(flip_s + (p / (B / 8)) * C::IN_PITCH + 16 * (p % (B / 8)), __ldg(reinterpret_cast<const uint4*>(flips) + p));
  }
  __syncthreads();

  for (; u < units; u += step) {
    uint64_t v[B / 2];                                    // v[i]: values i and i + B / 2 of the lane's block
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
#pragma unroll
    for (int q = 0; q < B / 16; ++q) {
      const uint32_t at = 16 * q, far = at + B;
      const uint4 x0 = lds128(in_s + lane * C::IN_PITCH + at), x1 = lds128(in_s + lane * C::IN_PITCH + far);
      uint32_t w0[4] = {x0.x, x0.y, x0.z, x0.w}, w1[4] = {x1.x, x1.y, x1.z, x1.w};
      if (flips) {                                        // the product with +-1 is taken in bf16, as the reference does
        const uint4 f0 = lds128(flip_s + l * C::IN_PITCH + at), f1 = lds128(flip_s + l * C::IN_PITCH + far);
        const uint32_t g0[4] = {f0.x, f0.y, f0.z, f0.w}, g1[4] = {f1.x, f1.y, f1.z, f1.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const __nv_bfloat162 p0 = __hmul2(*reinterpret_cast<const __nv_bfloat162*>(&w0[i]), *reinterpret_cast<const __nv_bfloat162*>(&g0[i]));
          const __nv_bfloat162 p1 = __hmul2(*reinterpret_cast<const __nv_bfloat162*>(&w1[i]), *reinterpret_cast<const __nv_bfloat162*>(&g1[i]));
          w0[i] = *reinterpret_cast<const uint32_t*>(&p0);
          w1[i] = *reinterpret_cast<const uint32_t*>(&p1);
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        v[8 * q + 2 * i] = pair_f32(w0[i] << 16, w1[i] << 16);
        v[8 * q + 2 * i + 1] = pair_f32(w0[i] & 0xFFFF0000u, w1[i] & 0xFFFF0000u);
      }
    }
    __syncwarp();                                         // every lane's values are in registers: the next rows may come
    if (u + step < units) fetch(u + step);

    // stages h = 1 .. B / 2, the last one inside the pairs
#pragma unroll
    for (int h = 1; h < B / 2; h <<= 1)
#pragma unroll
      for (int i = 0; i < B / 2; ++i)
        if ((i & h) == 0) butterfly2(v[i], v[i + h]);
#pragma unroll
    for (int i = 0; i < B / 2; ++i) {
      const float p = __uint_as_float((uint32_t)v[i]), q = __uint_as_float((uint32_t)(v[i] >> 32));
      v[i] = pair_f32(__float_as_uint(__fadd_rn(p, q)), __float_as_uint(__fsub_rn(p, q)));
    }

    // stages over the blocks of a row, 64 columns of every block at a time
    uint32_t o[C::HALVES][32];                            // bf16 pairs: word (block of the row, pair of the lane's columns)
#pragma unroll
    for (int hf = 0; hf < C::HALVES; ++hf) {
      auto value = [&](int c) {                           // value c of this half
        const int i = 64 * hf + c;
        return i < B / 2 ? (uint32_t)v[i % (B / 2)] : (uint32_t)(v[i % (B / 2)] >> 32);
      };
#pragma unroll
      for (int c = 0; c < 64; c += 4)
        sts128(xch_s + lane * C::XCH_PITCH + 4 * c, make_uint4(value(c), value(c + 1), value(c + 2), value(c + 3)));
      __syncwarp();
      uint64_t s[32];
#pragma unroll
      for (int j = 0; j < L; ++j) {
        const uint32_t at = xch_s + (rr * L + j) * C::XCH_PITCH + 4 * C::COLS * l;
        if constexpr (C::COLS == 2) {
          asm volatile("ld.shared.b64 %0, [%1];" : "=l"(s[j]) : "r"(at) : "memory");
        } else {
          asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(s[2 * j]), "=l"(s[2 * j + 1]) : "r"(at) : "memory");
        }
      }
      __syncwarp();
#pragma unroll
      for (int h = C::COLS / 2; h < 32; h <<= 1)
#pragma unroll
        for (int i = 0; i < 32; ++i)
          if ((i & h) == 0) butterfly2(s[i], s[i + h]);
#pragma unroll
      for (int i = 0; i < 32; i += 8) normalise8<LOGN % 2 == 0>(s + i, norm, inv_norm, o[hf] + i);
    }
#pragma unroll
    for (int hf = 0; hf < C::HALVES; ++hf)
#pragma unroll
      for (int j = 0; j < L; ++j) {
        const uint32_t at = xch_s + (rr * L + j) * C::IN_PITCH + 2 * (64 * hf + C::COLS * l);
        if constexpr (C::COLS == 2) {
          asm volatile("st.shared.b32 [%0], %1;" ::"r"(at), "r"(o[hf][j]) : "memory");
        } else {
          asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(at), "r"(o[hf][2 * j]), "r"(o[hf][2 * j + 1]) : "memory");
        }
      }
    __syncwarp();

    // the 16-bit channels pass through while the chunks are quantised
    int64_t t_at[2] = {-1, -1};
    uint4 t_val[2];
    if (per_row) {
#pragma unroll
      for (int k = 0; k < 2; ++k) t_val[k] = tail_piece(u, 32 * k + lane, t_at[k]);
    }
    const int64_t row = u * C::ROWS + rr;
#pragma unroll 1
    for (int c = 0; c < C::HALVES; ++c) {
      uint32_t w[32];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const uint4 q = lds128(xch_s + lane * C::IN_PITCH + 128 * c + 16 * i);
        w[4 * i] = q.x; w[4 * i + 1] = q.y; w[4 * i + 2] = q.z; w[4 * i + 3] = q.w;
      }
      if (row < a.M) quantise_chunk<MODE>(a, w, row, l * C::HALVES + c, n_kb64_pad);
    }
    if (per_row) {
#pragma unroll
      for (int k = 0; k < 2; ++k)
        if (t_at[k] >= 0) *reinterpret_cast<uint4*>(a.tail + t_at[k]) = t_val[k];
      for (int i = 64 + lane; i < C::ROWS * per_row; i += 32) {
        const uint4 val = tail_piece(u, i, t_at[0]);
        if (t_at[0] >= 0) *reinterpret_cast<uint4*>(a.tail + t_at[0]) = val;
      }
    }
    __syncwarp();                                         // the chunks are read: the buffer takes the next rows' columns
  }
}

template <int LOGN, int MODE>
static int launch_hq(const QuantArgs& a, const void* flips, cudaStream_t st) {
  using C = HqCfg<LOGN>;
  static PerDeviceOnce once;
  const auto k = hadamard_quant_kernel<LOGN, MODE>;
  if (const int rc = set_max_dynamic_smem(once, k, C::SMEM)) return rc;
  const float norm = sqrtf((float)C::N);
  const int64_t units = (a.M + C::ROWS - 1) / C::ROWS;
  const int grid = (int)(units < num_sms() ? units : num_sms());
  return launch_pdl(k, dim3(grid), dim3(C::WARPS * 32), C::SMEM, st, a, static_cast<const __nv_bfloat16*>(flips), norm,
                    1.f / norm) == cudaSuccess ? DIROTQ_OK : DIROTQ_E_CUDA;
}

template <int LOGN>
static int launch_hq_mode(const QuantArgs& a, const void* flips, cudaStream_t st) {
  switch (a.g.mode) {
    case DIROTQ_INT4_SYM: return launch_hq<LOGN, MODE_INT4_SYM>(a, flips, st);
    case DIROTQ_INT4_ASYM: return launch_hq<LOGN, MODE_INT4_ASYM>(a, flips, st);
    case DIROTQ_INT8_ASYM: return launch_hq<LOGN, MODE_INT8_ASYM>(a, flips, st);
    default: return launch_hq<LOGN, MODE_NVFP4_HW>(a, flips, st);
  }
}

// Transforms of one or two 64-channel chunks a lane that cover exactly the quantised channels, in the formats of which
// quantize.cu has a packed path.  (Shorter ones are launch-bound and have rows of less than 16 lanes; 8192 would take 256 values
// a lane.)  A warp that has its multiprocessor to itself takes about 5 us for a row of 4096, more than both separate kernels
// with 256 threads a row (16 rows, 4-bit symmetric / 8-bit: 5.8 / 7.3 us against 4.8 / 5.3; 64 rows 5.8 / 7.7 against 5.8 / 6.6);
// with more rows than multiprocessors it is the faster one (150 rows: 5.3 / 7.4 against 7.3 / 8.2).
bool hadamard_quant_covers(const ActGeom& g, int n, int64_t M) {
  if (n != 1024 && n != 2048 && n != 4096) return false;
  if (n == 4096 && M <= num_sms()) return false;
  if (g.H != 0 || g.per_token || g.q_len != n || g.tail_total % 8 || g.tail_pitch % 8) return false;
  if (g.mode == DIROTQ_NVFP4_HW) {
    uint32_t t;
    memcpy(&t, &g.T, 4);
    return (t & 0x7FFFFFu) == 0u;                         // quantize.cu's packed path: a power-of-two tensor scale
  }
  return g.mode != DIROTQ_NVFP4_REF && g.group == 64;
}

int launch_hadamard_quant(const QuantArgs& a, int n, const void* flips, cudaStream_t st) {
  if (a.M <= 0) return DIROTQ_OK;
  if (!hadamard_quant_covers(a.g, n, a.M)) return DIROTQ_E_UNSUPPORTED;
  switch (n) {
    case 1024: return launch_hq_mode<10>(a, flips, st);
    case 2048: return launch_hq_mode<11>(a, flips, st);
    default: return launch_hq_mode<12>(a, flips, st);
  }
}

}  // namespace dq
