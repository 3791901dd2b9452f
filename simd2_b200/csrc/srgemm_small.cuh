// srgemm_small.cuh -- small min/max products in one launch.
//
// One 32 x 32 tile of D = id (+) A(x)B [(+) C] per CTA of 256 threads, read from A
// and B as they lie: no operand preparation, no tensor maps, several CTAs on an
// SM.  A thread holds 2 x 2 outputs and folds two k at a time (Mac<OP>::mac2, the
// same operations as srgemm_sk.cuh on FP32, so the same bits).  What bounds such a
// call is the launch and the latency of the first loads: 100^3 takes 4.3 us here
// and 13.0 as prep + persistent kernel, 384^3 9.6 and 15.0; from about 450^3 on the
// larger register tiles and the 16-bit codes win (see small_product in capi.cu).
#pragma once
#include "srgemm_sk.cuh"

namespace simd2 {

constexpr int kSmallTile = 32;
constexpr int kSmallBK = 32;

// 4 consecutive elements of a row from p, of which `left` exist, else NaN (a NaN
// in both operands gives a NaN product, which min / max drop).
template <typename T>
__device__ __forceinline__ void small_load4(const T* p, int left, bool aligned, float (&x)[4]) {
  if (aligned && left >= 4) {
    load4(p, x);
  } else {
#pragma unroll
    for (int e = 0; e < 4; e++) x[e] = e < left ? (float)p[e] : __int_as_float(0x7fc00000);
  }
}

template <int OP, typename T>
__global__ void __launch_bounds__(256) srgemm_small_kernel(const T* __restrict__ A, long long lda,
                                                           const T* __restrict__ B, long long ldb, int M, int N,
                                                           int K, EpilogueArgs ep) {
  if (ep.gate && *ep.gate == 0) return;
  // A rows of k (pitch 36 floats: rows on 16-byte boundaries), B as k pairs
  __shared__ __align__(16) float As[2][kSmallTile][kSmallBK + 4];
  __shared__ __align__(16) float2 Bs[2][kSmallBK / 2][kSmallTile + 1];
  const int t = threadIdx.x;
  const int m0 = blockIdx.y * kSmallTile, n0 = blockIdx.x * kSmallTile;
  // loads: 4 elements of one row of A and of one row of B a thread
  const int lr = t >> 3, lc = (t & 7) * 4;
  const bool va = (lda % 4 == 0) && (reinterpret_cast<uintptr_t>(A) % (4 * sizeof(T)) == 0);
  const bool vb = (ldb % 4 == 0) && (reinterpret_cast<uintptr_t>(B) % (4 * sizeof(T)) == 0);
  float a[4], b[4];
  auto fetch = [&](int k0) {
    small_load4(A + (long long)(m0 + lr) * lda + k0 + lc, m0 + lr < M ? K - k0 - lc : 0, va, a);
    small_load4(B + (long long)(k0 + lr) * ldb + n0 + lc, k0 + lr < K ? N - n0 - lc : 0, vb, b);
  };
  auto park = [&](int s) {
    *reinterpret_cast<float4*>(&As[s][lr][lc]) = make_float4(a[0], a[1], a[2], a[3]);
#pragma unroll
    for (int e = 0; e < 4; e++) reinterpret_cast<float*>(&Bs[s][lr >> 1][lc + e])[lr & 1] = b[e];
  };
  const int tx = t & 15, ty = t >> 4;  // outputs (ty, ty + 16) x (tx, tx + 16)
  float acc[2][2];
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int j = 0; j < 2; j++) acc[i][j] = Mac<OP>::identity();
  fetch(0);
  park(0);
  __syncthreads();
  for (int k0 = 0, s = 0; k0 < K; k0 += kSmallBK, s ^= 1) {
    const bool more = k0 + kSmallBK < K;
    if (more) fetch(k0 + kSmallBK);
#pragma unroll
    for (int q = 0; q < kSmallBK / 4; q++) {
      float4 x[2];
#pragma unroll
      for (int i = 0; i < 2; i++) x[i] = *reinterpret_cast<const float4*>(&As[s][ty + 16 * i][4 * q]);
#pragma unroll
      for (int h = 0; h < 2; h++) {
#pragma unroll
        for (int j = 0; j < 2; j++) {
          const float2 y = Bs[s][2 * q + h][tx + 16 * j];
#pragma unroll
          for (int i = 0; i < 2; i++)
            acc[i][j] = Mac<OP>::mac2(acc[i][j], h ? make_float2(x[i].z, x[i].w) : make_float2(x[i].x, x[i].y), y);
        }
      }
    }
    if (more) {
      park(s ^ 1);
      __syncthreads();
    }
  }
  int changed = 0;
  const bool track = ep.changed != nullptr;
#pragma unroll
  for (int i = 0; i < 2; i++) {
#pragma unroll
    for (int j = 0; j < 2; j++) {
      const int row = m0 + ty + 16 * i, col = n0 + tx + 16 * j;
      if (row < M && col < N) {
        const float c = ep.do_epilogue ? ep.C[(long long)row * ep.ldc + col] : 0.f;
        ep.D[(long long)row * ep.ldd + col] =
            epilogue_value<OP>(ep.do_epilogue, ep.conv_mode, track, acc[i][j], c, changed);
      }
    }
  }
  if (track) {
    if (__any_sync(0xffffffffu, changed) && (t & 31) == 0) atomicOr(ep.changed, 1);
  }
}

}  // namespace simd2
