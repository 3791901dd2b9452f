// prep.cuh -- operand preparation kernels (HBM-bound, one pass each).
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <type_traits>

#include "common.cuh"

namespace simd2 {

// B'[p][2j+e] = B[2p+e][j] for 2p+e < K and j < N, else `pad`.
// B' has Kp/2 rows of 2*Np floats (Kp, Np are the padded sizes); a float4 of
// B' is (B[2p][j], B[2p+1][j], B[2p][j+1], B[2p+1][j+1]).
// A thread fills 4 columns (two float4 stores); B with 16-byte aligned rows is
// read with one float4 load per k row where the 4 columns are in range.
__global__ void interleave_pairs_kernel(const float* __restrict__ B, long long ldb, int K, int N,
                                        float* __restrict__ Bp, int Kp, int Np, float pad,
                                        const int* gate = nullptr) {
  if (gate && *gate == 0) return;
  const long long quads = Np / 4;
  const long long total = (long long)(Kp / 2) * quads;
  const bool vec = (ldb % 4 == 0) && (reinterpret_cast<uintptr_t>(B) % 16 == 0);
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    const int p = (int)(t / quads);
    const int j = (int)(t - (long long)p * quads) * 4;
    float x[2][4];
#pragma unroll
    for (int r = 0; r < 2; r++) {
      const int k = 2 * p + r;
      if (vec && k < K && j + 4 <= N) {
        const float4 u = __ldg(reinterpret_cast<const float4*>(B + (long long)k * ldb + j));
        x[r][0] = u.x, x[r][1] = u.y, x[r][2] = u.z, x[r][3] = u.w;
        continue;
      }
#pragma unroll
      for (int e = 0; e < 4; e++) x[r][e] = (k < K && j + e < N) ? B[(long long)k * ldb + j + e] : pad;
    }
    float4* o = reinterpret_cast<float4*>(Bp) + 2 * t;
    o[0] = make_float4(x[0][0], x[1][0], x[0][1], x[1][1]);
    o[1] = make_float4(x[0][2], x[1][2], x[0][3], x[1][3]);
  }
}

// Dense copy of A into an [M][Kp] float panel (row pitch Kp), padding k >= K
// with `pad`, for an A whose rows are not 16-byte aligned for TMA.
__global__ void pack_rows_kernel(const float* __restrict__ A, long long lda, int M, int K, float* __restrict__ Ap,
                                 int Kp, float pad, const int* gate = nullptr) {
  if (gate && *gate == 0) return;
  const long long total = (long long)M * Kp;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(t / Kp);
    const int k = (int)(t - (long long)i * Kp);
    Ap[t] = k < K ? A[(long long)i * lda + k] : pad;
  }
}

// D = id (+) C (or id) for K == 0.
template <typename T>
__global__ void fill_kernel(T* D, long long ldd, int M, int N, T value) {
  const long long total = (long long)M * N;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(t / N);
    const int j = (int)(t - (long long)i * N);
    D[(long long)i * ldd + j] = value;
  }
}

// Change test + copy, the work of comp_update / comp_update2
// (kernel/converge.cuh:6-84): mode 1 |prev-cur| > 1e-4, mode 2 maps cur values
// in (-1,1) to -FLT_MAX first (in cur and prev) then tests inequality, mode 0
// tests bitwise inequality; prev := cur.  One flag word, set by a warp vote.
template <typename T>
__global__ void compare_update_kernel(T* __restrict__ prev, T* __restrict__ cur, long long n, int mode,
                                      int* __restrict__ flag) {
  int ch = 0;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
    T c = cur[t];
    const T pv = prev[t];
    if constexpr (std::is_same<T, float>::value) {
      if (mode == 2 && c > T(-1) && c < T(1)) {
        c = T(-3.402823466e+38f);
        cur[t] = c;
      }
      if (mode == 1) ch |= fabsf((float)pv - (float)c) > 0.0001f;
      else ch |= __float_as_uint((float)pv) != __float_as_uint((float)c);
    } else {
      ch |= pv != c;
    }
    prev[t] = c;
  }
  if (__any_sync(0xffffffffu, ch) && (threadIdx.x & 31) == 0) atomicOr(flag, 1);
}

// D = (C != 0) as 0/1 of type T.
template <typename T>
__global__ void bool_copy_kernel(const T* __restrict__ C, long long ldc, T* __restrict__ D, long long ldd, int M,
                                 int N) {
  const long long total = (long long)M * N;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(t / N);
    const int j = (int)(t - (long long)i * N);
    D[(long long)i * ldd + j] = C[(long long)i * ldc + j] != T(0) ? T(1) : T(0);
  }
}

}  // namespace simd2

namespace simd2 {

// ---------------------------------------------------------------------------
// Operand preparation for the tensor-core paths.  Outputs are K-major with a
// row pitch of Kp elements (Kp a multiple of 8 for BF16, 16 for bytes, so the
// TMA row stride is a multiple of 16 bytes); k in [K, Kp) is zero.
// ---------------------------------------------------------------------------

// x = hi + lo with hi = bf16(x), lo = bf16(x - hi) (both round-to-nearest).
__device__ __forceinline__ void split_bf16(float x, __nv_bfloat16& hi, __nv_bfloat16& lo) {
  hi = __float2bfloat16_rn(x);
  lo = __float2bfloat16_rn(__fsub_rn(x, __bfloat162float(hi)));
}

__device__ __forceinline__ uint32_t pack_bf16x2(__nv_bfloat16 a, __nv_bfloat16 b) {
  return (uint32_t)__bfloat16_as_ushort(a) | ((uint32_t)__bfloat16_as_ushort(b) << 16);
}

// A [M][K] (pitch lda) -> A_hi, A_lo [M][Kp], zeros for k >= K.  Kp is a
// multiple of 8 and hi / lo are 16-byte aligned: a thread converts 8
// consecutive elements of a row (two 16-byte loads when A's rows allow) and
// writes 16 bytes to each output.
__global__ void split_rows_bf16_kernel(const float* __restrict__ A, long long lda, int M, int K,
                                       __nv_bfloat16* __restrict__ hi, __nv_bfloat16* __restrict__ lo, int Kp) {
  const int groups = Kp >> 3;
  const long long total = (long long)M * groups;
  const bool vec = (lda % 4 == 0) && (reinterpret_cast<uintptr_t>(A) % 16 == 0);
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(t / groups);
    const int k0 = (int)(t - (long long)i * groups) * 8;
    const float* row = A + (long long)i * lda;
    float x[8];
    if (vec && k0 + 8 <= K) {
      const float4 u = __ldg(reinterpret_cast<const float4*>(row + k0));
      const float4 w = __ldg(reinterpret_cast<const float4*>(row + k0 + 4));
      x[0] = u.x, x[1] = u.y, x[2] = u.z, x[3] = u.w, x[4] = w.x, x[5] = w.y, x[6] = w.z, x[7] = w.w;
    } else {
#pragma unroll
      for (int e = 0; e < 8; e++) x[e] = k0 + e < K ? row[k0 + e] : 0.f;
    }
    uint32_t hw[4], lw[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      __nv_bfloat16 h0, l0, h1, l1;
      split_bf16(x[2 * q], h0, l0);
      split_bf16(x[2 * q + 1], h1, l1);
      hw[q] = pack_bf16x2(h0, h1);
      lw[q] = pack_bf16x2(l0, l1);
    }
    reinterpret_cast<uint4*>(hi)[t] = make_uint4(hw[0], hw[1], hw[2], hw[3]);
    reinterpret_cast<uint4*>(lo)[t] = make_uint4(lw[0], lw[1], lw[2], lw[3]);
  }
}

// True as the FP4 (E2M1) value 1.0 in each nibble of 8 bytes of 0 / 1 (two words
// of four): byte j of the result holds elements 2j (low nibble) and 2j + 1.
__device__ __forceinline__ uint32_t nibbles_fp4(uint32_t w0, uint32_t w1) {
  // byte pairs (b0, b1) -> b0 | b1 << 4 at the even bytes
  const uint32_t p0 = (w0 | w0 >> 4) & 0x00ff00ffu, p1 = (w1 | w1 >> 4) & 0x00ff00ffu;
  return __byte_perm(p0, p1, 0x6420) << 1;
}

template <typename T>
__device__ __forceinline__ bool is_true(T x) {
  if constexpr (std::is_same<T, __half>::value) return (__half_as_ushort(x) & 0x7fffu) != 0;  // -0 is false
  else return x != T(0);
}

// 16 elements from p, of which `left` exist, as 0 / 1 bytes (16 / sizeof(T)
// elements a load where p is aligned and all exist).
template <typename T>
__device__ __forceinline__ void load_bool16(const T* p, int left, uint32_t (&w)[4]) {
  constexpr int PER = 16 / (int)sizeof(T);
  if (left >= 16 && (reinterpret_cast<uintptr_t>(p) & 15) == 0) {
#pragma unroll
    for (int q = 0; q < 16 / PER; q++) {
      const uint4 u = __ldg(reinterpret_cast<const uint4*>(p) + q);
      const uint32_t in[4] = {u.x, u.y, u.z, u.w};
      if constexpr (sizeof(T) == 1) {
#pragma unroll
        for (int e = 0; e < 4; e++) w[e] = bytes_nonzero_01(in[e]);
      } else if constexpr (sizeof(T) == 4) {
        w[q] = (in[0] != 0u) | (in[1] != 0u) << 8 | (in[2] != 0u) << 16 | (uint32_t)(in[3] != 0u) << 24;
      } else {
#pragma unroll
        for (int e = 0; e < 2; e++)
          w[2 * q + e] = ((in[2 * e] & 0x7fffu) != 0u) | ((in[2 * e] & 0x7fff0000u) != 0u) << 8 |
                         ((in[2 * e + 1] & 0x7fffu) != 0u) << 16 |
                         (uint32_t)((in[2 * e + 1] & 0x7fff0000u) != 0u) << 24;
      }
    }
  } else {
#pragma unroll
    for (int q = 0; q < 4; q++) {
      uint32_t v = 0;
#pragma unroll
      for (int e = 0; e < 4; e++)
        v |= (uint32_t)(4 * q + e < left && is_true(p[4 * q + e])) << (8 * e);
      w[q] = v;
    }
  }
}

// or_and's A: A [M][K] of T -> FP4 [M][Kp / 2 bytes], zeros for k >= K.  Kp is a
// multiple of 32: a thread packs 16 elements of a row into 8 bytes.
template <typename T>
__global__ void __launch_bounds__(256) bool_rows_fp4_kernel(const T* __restrict__ A, long long lda, int M, int K,
                                                            uint8_t* __restrict__ out, int Kp) {
  const int groups = Kp >> 4;
  const long long total = (long long)M * groups;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(t / groups);
    const int k0 = (int)(t - (long long)i * groups) * 16;
    uint32_t w[4];
    load_bool16(A + (long long)i * lda + k0, K - k0, w);
    reinterpret_cast<uint2*>(out)[t] = make_uint2(nibbles_fp4(w[0], w[1]), nibbles_fp4(w[2], w[3]));
  }
}

// or_and's B: B [K][N] of T (pitch ldb) -> FP4 [N][Kp / 2 bytes], zeros for k >= K,
// and, where a4 is set, B's rows as an A operand too ([K][Np / 2 bytes], zeros past
// N: the closure's X is both, read once).  chg_row / chg_col (may be null: all): a
// 256-row group of a4, and the columns of a BN-column group of b4, are written only
// where their byte is set (they hold what they held otherwise).
//
// One tile of 256 k x 128 columns per block, bounded by DRAM: as bytes 0 / 1 in
// shared memory, 16 bytes a store; then a thread takes 32 k of 4 columns, a word of
// 4 bytes per k: two words shifted together hold the nibbles of two k, and four of
// those, transposed as 4 x 4 bytes, 8 k of each column.  A warp covers 8 k groups x 4
// words, so it writes whole 128-byte lines; 4 words of padding per 32 rows keep
// its loads free of bank conflicts.  16384^2 bytes as both operands 115 us (DRAM
// alone: 82).  (A thread that gathered single bytes for one
// column took 169, and 75 more for a separate pass over the rows.)
template <typename T>
__global__ void __launch_bounds__(256) transpose_fp4_kernel(const T* __restrict__ B, long long ldb, int K, int N,
                                                            uint8_t* __restrict__ b4, int Kp,
                                                            uint8_t* __restrict__ a4, int Np,
                                                            const uint8_t* __restrict__ chg_row,
                                                            const uint8_t* __restrict__ chg_col, int BN,
                                                            const int* gate) {
  if (gate && *gate == 0) return;
  __shared__ __align__(16) uint32_t tile[256 * 32 + 8 * 4];
  const int t = threadIdx.x;
  const int k0 = blockIdx.y * 256, j0 = blockIdx.x * 128;
  const bool rows = a4 && (!chg_row || chg_row[blockIdx.y]);
  const bool cols = !chg_col || chg_col[j0 / BN] || chg_col[min(j0 + 127, N - 1) / BN];
  if (!rows && !cols) return;
#pragma unroll(sizeof(T) == 1 ? 8 : 2)
  for (int h = 0; h < 8; h++) {
    const int r = (t >> 3) + 32 * h, c0 = (t & 7) * 16;
    const int k = k0 + r, j = j0 + c0;
    uint32_t w[4] = {0u, 0u, 0u, 0u};
    if (k < K && j < N) load_bool16(B + (long long)k * ldb + j, N - j, w);
    *reinterpret_cast<uint4*>(&tile[r * 32 + (r >> 5) * 4 + (c0 >> 2)]) = make_uint4(w[0], w[1], w[2], w[3]);
    if (rows && k < K && j < Np)
      *reinterpret_cast<uint2*>(a4 + ((long long)k * Np + j) / 2) =
          make_uint2(nibbles_fp4(w[0], w[1]), nibbles_fp4(w[2], w[3]));
  }
  if (!cols) return;
  __syncthreads();
  const int kg = (t & 31) >> 2, cw = (t >> 5) * 4 + (t & 3);
  const int ko = k0 + 32 * kg, jo = j0 + 4 * cw;
  if (ko >= Kp || jo >= N) return;
  const uint32_t* src = &tile[32 * kg * 32 + kg * 4 + cw];
  uint32_t o[4][4];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    uint32_t p[4];
#pragma unroll
    for (int e = 0; e < 4; e++) p[e] = src[(8 * q + 2 * e) * 32] << 1 | src[(8 * q + 2 * e + 1) * 32] << 5;
    const uint32_t a = __byte_perm(p[0], p[1], 0x5140), b = __byte_perm(p[2], p[3], 0x5140);
    const uint32_t c = __byte_perm(p[0], p[1], 0x7362), d = __byte_perm(p[2], p[3], 0x7362);
    o[0][q] = __byte_perm(a, b, 0x5410);
    o[1][q] = __byte_perm(a, b, 0x7632);
    o[2][q] = __byte_perm(c, d, 0x5410);
    o[3][q] = __byte_perm(c, d, 0x7632);
  }
#pragma unroll
  for (int c = 0; c < 4; c++)
    if (jo + c < N)
      *reinterpret_cast<uint4*>(b4 + ((long long)(jo + c) * Kp + ko) / 2) =
          make_uint4(o[c][0], o[c][1], o[c][2], o[c][3]);
}

// Operand preparation of the sums, one launch: blocks [0, a_blocks) take rows of
// A, a warp each, the next b_blocks rows of B, the last ones 16 columns of B each.  FP32 operands are split into BF16 hi / lo copies of the same layout
// (A [M][Kp], B [K][Np], zeros past K and N); float16 ones are copied only where
// TMA cannot read them as they are (a_hi / b_hi set).  minus_square (na / nb set):
// the squared row norms of A and column norms of B, summed in FP64.
struct SumPrepArgs {
  const void* A;
  long long lda;
  const void* B;
  long long ldb;
  int M, N, K, Kp, Np;
  uint16_t *a_hi, *a_lo, *b_hi, *b_lo;
  float *na, *nb;
  int a_blocks, b_blocks;
};

// 8 consecutive elements as floats, zeros past `left`.
template <typename T>
__device__ __forceinline__ void load8(const T* p, int left, float (&x)[8]) {
  if (left >= 8 && (reinterpret_cast<uintptr_t>(p) & 15) == 0) {
    if constexpr (sizeof(T) == 4) {
      const float4 u = __ldg(reinterpret_cast<const float4*>(p)), w = __ldg(reinterpret_cast<const float4*>(p) + 1);
      x[0] = u.x, x[1] = u.y, x[2] = u.z, x[3] = u.w, x[4] = w.x, x[5] = w.y, x[6] = w.z, x[7] = w.w;
    } else {
      const uint4 u = __ldg(reinterpret_cast<const uint4*>(p));
      const uint32_t in[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
      for (int q = 0; q < 4; q++) {
        x[2 * q] = __half2float(__ushort_as_half((unsigned short)(in[q] & 0xffffu)));
        x[2 * q + 1] = __half2float(__ushort_as_half((unsigned short)(in[q] >> 16)));
      }
    }
  } else {
#pragma unroll
    for (int e = 0; e < 8; e++) x[e] = e < left ? (float)p[e] : 0.f;
  }
}

// The copies of 8 elements: hi / lo of BF16, or (lo null) the halves.
template <typename T>
__device__ __forceinline__ void store8(const float (&x)[8], uint16_t* hi, uint16_t* lo) {
  uint32_t hw[4], lw[4];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    if constexpr (sizeof(T) == 4) {
      __nv_bfloat16 h0, l0, h1, l1;
      split_bf16(x[2 * q], h0, l0);
      split_bf16(x[2 * q + 1], h1, l1);
      hw[q] = pack_bf16x2(h0, h1);
      lw[q] = pack_bf16x2(l0, l1);
    } else {
      hw[q] = (uint32_t)__half_as_ushort(__float2half_rn(x[2 * q])) |
              (uint32_t)__half_as_ushort(__float2half_rn(x[2 * q + 1])) << 16;
    }
  }
  *reinterpret_cast<uint4*>(hi) = make_uint4(hw[0], hw[1], hw[2], hw[3]);
  if constexpr (sizeof(T) == 4) *reinterpret_cast<uint4*>(lo) = make_uint4(lw[0], lw[1], lw[2], lw[3]);
}

template <typename T>
__global__ void __launch_bounds__(256) sum_prep_kernel(SumPrepArgs g) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const T* A = static_cast<const T*>(g.A);
  const T* B = static_cast<const T*>(g.B);
  if ((int)blockIdx.x < g.a_blocks) {
    for (int i = blockIdx.x * 8 + warp; i < g.M; i += g.a_blocks * 8) {
      double sum = 0.0;
      for (int k = lane * 8; k < g.Kp; k += 256) {
        float x[8];
        load8(A + (long long)i * g.lda + k, g.K - k, x);
        if (g.a_hi) {
          const long long o = (long long)i * g.Kp + k;
          store8<T>(x, g.a_hi + o, g.a_lo + o);
        }
        if (g.na) {
#pragma unroll
          for (int e = 0; e < 8; e++) sum += (double)x[e] * (double)x[e];
        }
      }
      if (g.na) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (lane == 0) g.na[i] = (float)sum;
      }
    }
  } else if ((int)blockIdx.x < g.a_blocks + g.b_blocks) {
    const int groups = g.Np >> 3;
    const long long total = (long long)g.K * groups;
    for (long long t = (blockIdx.x - g.a_blocks) * 256LL + threadIdx.x; t < total; t += g.b_blocks * 256LL) {
      const int k = (int)(t / groups), j = (int)(t - (long long)k * groups) * 8;
      float x[8];
      load8(B + (long long)k * g.ldb + j, g.N - j, x);
      store8<T>(x, g.b_hi + t * 8, g.b_lo + t * 8);
    }
  } else {
    // thread: one of 16 columns, one of 16 runs of k; the partial sums meet in order
    __shared__ double part[16][16];
    const int c = threadIdx.x & 15, q = threadIdx.x >> 4;
    const int j = (blockIdx.x - g.a_blocks - g.b_blocks) * 16 + c;
    const int per = (g.K + 15) / 16, k1 = min(g.K, (q + 1) * per);
    double sum = 0.0;
    if (j < g.N) {
#pragma unroll 16
      for (int k = q * per; k < k1; k++) {
        const double v = (double)(float)B[(long long)k * g.ldb + j];
        sum += v * v;
      }
    }
    part[q][c] = sum;
    __syncthreads();
    if (q == 0 && j < g.N) {
#pragma unroll
      for (int r = 1; r < 16; r++) sum += part[r][c];
      g.nb[j] = (float)sum;
    }
  }
}

// Squared row norms of A [M][K], accumulated in FP64, rounded to float.
__global__ void row_norms_kernel(const float* __restrict__ A, long long lda, int M, int K, float* __restrict__ out) {
  const int warps = blockDim.x / 32;
  for (int i = blockIdx.x * warps + threadIdx.x / 32; i < M; i += gridDim.x * warps) {
    double s = 0.0;
    for (int k = threadIdx.x % 32; k < K; k += 32) {
      const double v = A[(long long)i * lda + k];
      s += v * v;
    }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (threadIdx.x % 32 == 0) out[i] = (float)s;
  }
}

}  // namespace simd2
