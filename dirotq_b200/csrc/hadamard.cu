// Walsh-Hadamard front end of the layers the reference rotates with a randomised Hadamard transform
// instead of a dense PCA rotation (DiRotQ dirotq_fused_unrotation_fast.py:106-128, utils/hadamard_utils.py:56-80):
//   y[:, :n] = FWHT(x[:, :n] * flips) / sqrt(n)   (fp32 butterflies, stage order h = 1, 2, 4, ...)
//   y[:, n:] = x[:, n:]
// Every output is produced by the same sequence of fp32 additions as the reference's butterfly, so the
// result is bit-identical to it; the quantiser then runs on y.  HBM-bound: 2 D bytes in, 2 D bytes out per row.
//
// n / 16 threads per row (several rows per CTA when that is fewer than 256), 16 values per thread in registers.  Four
// stages at a time are register arithmetic: in pass p a thread holds the 16 values whose indices differ only in bits
// 4p .. 4p+3, so the stages h = 2^(4p) .. 2^(4p+3) need no exchange; between passes the values trade places through
// shared memory (rows of 16 floats padded to 17: conflict-free in the first two passes; in a third, whose lanes reach over
// two rows, lanes 0 and 31 share a bank).  A thread writes only
// the positions it read, so one barrier per exchange is enough.  4096 rows x 4608 channels, n = 4096: 98 -> 21 us (one
// barrier pair and one shared-memory round trip per stage, with the butterfly's index arithmetic, before).
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include "layout.cuh"
#include "launchers.cuh"
#include "ptx.cuh"

namespace dq {

template <int BITS, int STRIDE>
__device__ __forceinline__ void fwht_stages(float* v) {      // BITS stages over register distances STRIDE, 2 STRIDE, ...
#pragma unroll
  for (int s = 0; s < BITS; ++s) {
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const int h = STRIDE << s;
      if ((i & h) == 0) {
        const float p = v[i], q = v[i + h];
        v[i] = __fadd_rn(p, q);
        v[i + h] = __fsub_rn(p, q);
      }
    }
  }
}

// A row of 16 or 32 transformed channels has one or two threads, 256 or 128 rows share a block, and the rest of a row is as
// wide as ever: blocks of their own copy it (1152 channels, n = 16: 54 -> 2 us for 256 rows, 85 -> 26 for 32768).  Longer
// transforms copy theirs in passing, which the loads of the transform hide (n = 8192 of 12288 channels, 32768 rows: 415 us,
// 473 with blocks of their own; from n = 128 to 512 the two differ by a microsecond either way).
constexpr bool copy_blocks_of(int logn) { return logn <= 5; }

template <int LOGN>
__global__ void __launch_bounds__(LOGN == 13 ? 512 : 256)
hadamard_low_kernel(const __nv_bfloat16* __restrict__ x, int64_t M, int D, const __nv_bfloat16* __restrict__ flips,
                    float inv_norm_is_exact, float norm, __nv_bfloat16* __restrict__ y, int fwht_blocks, int copy_rows) {
  constexpr int N = 1 << LOGN, T = N / 16, THREADS = LOGN == 13 ? 512 : 256, ROWS = THREADS / T;
  constexpr int FULL = LOGN / 4, REM = LOGN % 4;              // passes of four stages, stages of the last pass
  __shared__ float sh[(FULL > 1 || REM) ? ROWS * T * 17 : 1];
  if constexpr (copy_blocks_of(LOGN)) {
    if ((int)blockIdx.x >= fwht_blocks) {                     // untouched channels of copy_rows rows
      const int per = (D - N) >> 3;                           // 16-byte units per row
      const int64_t r0 = (int64_t)((int)blockIdx.x - fwht_blocks) * copy_rows;
      pdl_launch_dependents();
      pdl_wait();
      for (int i = threadIdx.x; i < copy_rows * per; i += THREADS) {
        const int r = i / per;
        if (r0 + r >= M) break;
        const int64_t at = (r0 + r) * D + N + 8 * (i - r * per);
        *reinterpret_cast<uint4*>(y + at) = *reinterpret_cast<const uint4*>(x + at);
      }
      return;
    }
  }
  const int t = threadIdx.x % T, lr = threadIdx.x / T;
  const int64_t row = (int64_t)blockIdx.x * ROWS + lr;
  const bool ok = row < M;
  const __nv_bfloat16* xr = x + row * D;
  __nv_bfloat16* yr = y + row * D;
  float* s = sh + lr * (T * 17);
  pdl_launch_dependents();
  pdl_wait();
  float v[16];
  if (ok) {
    const uint4 a = *reinterpret_cast<const uint4*>(xr + 16 * t), b = *reinterpret_cast<const uint4*>(xr + 16 * t + 8);
    uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    if (flips) {                        // the product with +-1 is taken in bf16, as the reference does
      const uint4 fa = __ldg(reinterpret_cast<const uint4*>(flips + 16 * t)), fb = __ldg(reinterpret_cast<const uint4*>(flips + 16 * t + 8));
      const uint32_t f[8] = {fa.x, fa.y, fa.z, fa.w, fb.x, fb.y, fb.z, fb.w};
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const __nv_bfloat162 p = __hmul2(*reinterpret_cast<const __nv_bfloat162*>(&w[j]), *reinterpret_cast<const __nv_bfloat162*>(&f[j]));
        w[j] = *reinterpret_cast<const uint32_t*>(&p);
      }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      v[2 * j] = __uint_as_float(w[j] << 16);
      v[2 * j + 1] = __uint_as_float(w[j] & 0xFFFF0000u);
    }
  } else {
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = 0.f;
  }
  fwht_stages<4, 1>(v);
  if constexpr (FULL > 1 || REM) {
#pragma unroll
    for (int j = 0; j < 16; ++j) s[17 * t + j] = v[j];
  }
#pragma unroll
  for (int p = 1; p < FULL; ++p) {                            // indices differing in bits 4p .. 4p+3
    __syncthreads();
    const int base = ((t >> (4 * p)) << (4 * p + 4)) + (t & ((1 << (4 * p)) - 1));
    float* sp = s + 17 * (base >> 4) + (base & 15);
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = sp[17 * (j << (4 * p - 4))];
    fwht_stages<4, 1>(v);
    if (p + 1 < FULL || REM) {
#pragma unroll
      for (int j = 0; j < 16; ++j) sp[17 * (j << (4 * p - 4))] = v[j];
    }
  }
  // last pass of REM stages: COLS neighbouring columns at each of 2^REM distances of N >> REM
  constexpr int COLS = 16 >> REM;
  if constexpr (REM > 0) {
    __syncthreads();
    const int base = COLS * t;
#pragma unroll
    for (int j = 0; j < (1 << REM); ++j)
#pragma unroll
      for (int c = 0; c < COLS; ++c) v[COLS * j + c] = s[17 * ((base >> 4) + j * (T >> REM)) + (base & 15) + c];
    fwht_stages<REM, COLS>(v);
  }
  // normalise (IEEE division by sqrt(n), exact scaling when n is a power of four) and store
  if (ok) {
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = inv_norm_is_exact != 0.f ? v[j] * inv_norm_is_exact : __fdiv_rn(v[j], norm);
    if constexpr (REM == 0 && FULL > 1) {
      constexpr int P = 4 * (FULL - 1);
#pragma unroll
      for (int j = 0; j < 16; ++j) yr[t + (j << P)] = __float2bfloat16_rn(v[j]);     // 64 bytes per warp and store
    } else {
      uint32_t w[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const __nv_bfloat162 hh = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
        w[j] = *reinterpret_cast<const uint32_t*>(&hh);
      }
      if constexpr (REM == 0) {                               // N == 16
        *reinterpret_cast<uint4*>(yr) = make_uint4(w[0], w[1], w[2], w[3]);
        *reinterpret_cast<uint4*>(yr + 8) = make_uint4(w[4], w[5], w[6], w[7]);
      } else if constexpr (REM == 1) {
#pragma unroll
        for (int j = 0; j < 2; ++j)
          *reinterpret_cast<uint4*>(yr + 8 * t + j * (N >> 1)) = make_uint4(w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]);
      } else if constexpr (REM == 2) {
#pragma unroll
        for (int j = 0; j < 4; ++j) *reinterpret_cast<uint2*>(yr + 4 * t + j * (N >> 2)) = make_uint2(w[2 * j], w[2 * j + 1]);
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) *reinterpret_cast<uint32_t*>(yr + 2 * t + j * (N >> 3)) = w[j];
      }
    }
    // untouched channels
    if constexpr (!copy_blocks_of(LOGN))
      for (int c = N + 8 * t; c < D; c += 8 * T) *reinterpret_cast<uint4*>(yr + c) = *reinterpret_cast<const uint4*>(xr + c);
  }
}

template <int LOGN>
static int launch_fwht(const void* x, int64_t M, int D, const void* flips, void* y, cudaStream_t st) {
  constexpr int THREADS = LOGN == 13 ? 512 : 256, ROWS = THREADS / ((1 << LOGN) / 16);
  const float norm = sqrtf((float)(1 << LOGN));
  const float inv_exact = (LOGN % 2 == 0) ? 1.f / norm : 0.f;     // power of four: the division is an exact scaling
  const int64_t fwht_blocks = (M + ROWS - 1) / ROWS;
  const int per = (D - (1 << LOGN)) / 8;                      // 16-byte units to copy per row, four per thread and block
  const int copy_rows = per > 0 && per < 4 * THREADS ? 4 * THREADS / per : 1;
  const int64_t copy_blocks = copy_blocks_of(LOGN) && per > 0 ? (M + copy_rows - 1) / copy_rows : 0;
  if (fwht_blocks + copy_blocks > 0x7fffffff) return DIROTQ_E_TOO_LARGE;
  return launch_pdl(hadamard_low_kernel<LOGN>, dim3((unsigned)(fwht_blocks + copy_blocks)), dim3(THREADS), 0, st,
                    static_cast<const __nv_bfloat16*>(x), M, D, static_cast<const __nv_bfloat16*>(flips), inv_exact, norm,
                    static_cast<__nv_bfloat16*>(y), (int)fwht_blocks, copy_rows) == cudaSuccess
             ? DIROTQ_OK : DIROTQ_E_CUDA;
}

int launch_hadamard_low(const void* x, int64_t M, int D, int n, const void* flips, void* y, cudaStream_t st) {
  if (M <= 0) return DIROTQ_OK;
  if (n < 16 || n > 8192 || (n & (n - 1)) || n > D || D % 8) return DIROTQ_E_UNSUPPORTED;
  switch (n) {
    case 16: return launch_fwht<4>(x, M, D, flips, y, st);
    case 32: return launch_fwht<5>(x, M, D, flips, y, st);
    case 64: return launch_fwht<6>(x, M, D, flips, y, st);
    case 128: return launch_fwht<7>(x, M, D, flips, y, st);
    case 256: return launch_fwht<8>(x, M, D, flips, y, st);
    case 512: return launch_fwht<9>(x, M, D, flips, y, st);
    case 1024: return launch_fwht<10>(x, M, D, flips, y, st);
    case 2048: return launch_fwht<11>(x, M, D, flips, y, st);
    case 4096: return launch_fwht<12>(x, M, D, flips, y, st);
    default: return launch_fwht<13>(x, M, D, flips, y, st);
  }
}

}  // namespace dq
