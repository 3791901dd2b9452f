// closure_coop.cuh -- a small closure as one cooperative launch.
//
// X <- X (+) X(x)X until unchanged (apps/apsp/cuASR/apsp_cuASR.cu:37-54) for one
// matrix whose step is short against a launch: every CTA of a cooperative grid
// stays for all steps and meets the others at a grid barrier after each.  X lives
// in its 16-bit codes only (srgemm_sk.cuh), in both operand layouts, ping-pong;
// the FP32 matrix is read once at the start and written once at the end.  A step
// is srgemm_sk_kernel's: 64 x 64 tiles whose k-tiles are split evenly over the
// CTAs, the last contributor of a tile folding the others' partial tiles, all of
// it on packed codes.  An entry or a result without a code ends the kernel with X
// untouched and the caller takes the launch-per-step path.
//
// n = 512 (5 steps): launch per step 213 us, of which the steps' arithmetic is
// 18; the rest was two launches a step, steps enqueued past the fixed point and a
// host round trip per chunk.  Now 94 us: about 10 a step (4.6 of arithmetic, the
// first loads, the fold between CTAs and the barrier), the launch, the two passes
// over X and the host's round trip.
#pragma once
#include "closure_batched.cuh"

namespace simd2 {

// Control words, cleared before the launch.
struct CoopCtl {
  unsigned bar;      // arrivals at the grid barrier
  int last_changed;  // 1 + the last step that changed something
  int over_neg;      // 0, or 2^30 - t for the first step t whose result has no code (t = -1: an entry)
                     // compared with the reader's step: a faster CTA may have raised it for the next one
  int failed;        // set by a CTA in which a bounded wait ran out
};

struct CoopArgs {
  float* X;
  long long ldx;
  int n, Kh, Np;      // k padded to 64, columns padded to 128
  uint16_t* Xc[2];    // [tiles * 64][Kh]
  uint32_t* Pc[2];    // [Kh / 2][Np]
  int tiles;          // 64 x 64 tiles a side
  int whole;          // tiles every CTA computes alone a step; the rest is split by units
  int max_iter, conv;
  int* counters;      // arrivals per split tile, over all steps
  uint4* part;        // two slots of 64 x 64 codes per CTA
  CoopCtl* ctl;
  volatile int* out;  // host memory: steps; 1 converged, 2 not converged, 3 / 4 a result / an entry without a code
                      // (X untouched); 1 when a CTA failed
};

// All CTAs of the grid; `target` arrivals in total.  A CTA in which a wait ran out
// has folded or written wrong codes: it says so before it arrives, and every CTA
// leaves the barrier with *failed set.
__device__ __forceinline__ void coop_barrier(CoopCtl* ctl, unsigned target, volatile int* failed) {
  fence_proxy_async_global();
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    if (*failed) {
      atomicExch(&ctl->failed, 1);
      __threadfence();
    }
    atomicAdd(&ctl->bar, 1u);
    const uint64_t t0 = globaltimer_ns();
    while ((unsigned)ld_acquire(reinterpret_cast<const int*>(&ctl->bar)) < target) {
      if (globaltimer_ns() - t0 > kWaitLimitNs) {
        report_timeout(51);
        *failed = 1;
        break;
      }
    }
    if (*(volatile int*)&ctl->failed) *failed = 1;
  }
  __syncthreads();
  fence_proxy_async_global();
}

template <int OP>
__global__ void __launch_bounds__(kSimtThreads, 1)
    closure_coop_kernel(const __grid_constant__ CUtensorMap a0, const __grid_constant__ CUtensorMap a1,
                        const __grid_constant__ CUtensorMap b0, const __grid_constant__ CUtensorMap b1, CoopArgs g) {
  using Cfg = SkCfg<64>;
  using Code = Code16<OP>;
  constexpr int S = Cfg::kStages;
  constexpr int kPitch = 36;  // words of a row of the fold buffer (32 column pairs)
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint32_t* red = reinterpret_cast<uint32_t*>(smem + S * Cfg::kStage);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + S * Cfg::kStage + Cfg::kRedBytes);
  uint64_t* empty = full + S;
  __shared__ int s_failed, s_last;
  volatile int* failed = &s_failed;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tx = lane & 15;
  const int ty = (warp & 3) * 2 + (lane >> 4);
  const int kg = warp >> 2;
  const int n = g.n, Kh = g.Kh, Np = g.Np;
  const int G = gridDim.x, cta = blockIdx.x;
  const int kt = Kh / kSkBK16;
  const int first_split = g.whole * G;
  const long long units = (long long)(g.tiles * g.tiles - first_split) * kt;
  const long long u0 = units * cta / G, u1 = units * (cta + 1) / G;
  const int nwhole = g.whole * kt;
  const int nloads = nwhole + (int)(u1 - u0);
  if (threadIdx.x == 0) {
    for (int s = 0; s < S; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], kSimtWarps);
    }
    s_failed = 0;
    fence_mbar_init();
    prefetch_tensormap(&a0);
    prefetch_tensormap(&a1);
    prefetch_tensormap(&b0);
    prefetch_tensormap(&b1);
  }

  // codes of X in both layouts, padding of both buffers: 2 rows x 4 columns a thread
  {
    const bool vec = (g.ldx % 4 == 0) && (reinterpret_cast<uintptr_t>(g.X) % 16 == 0);
    const int quads = Np >> 2;
    const long long total = (long long)(Kh >> 1) * quads;
    bool bad = false;
    for (long long t = cta * (long long)kSimtThreads + threadIdx.x; t < total; t += (long long)G * kSimtThreads) {
      const int p = (int)(t / quads), c0 = (int)(t - (long long)p * quads) * 4;
      uint32_t c[2][4];
#pragma unroll
      for (int r = 0; r < 2; r++) {
        const int row = 2 * p + r;
        const float* src = g.X + (long long)row * g.ldx + c0;
        float v[4];
        if (vec && row < n && c0 + 4 <= n) {
          load4(src, v);
        } else {
#pragma unroll
          for (int e = 0; e < 4; e++) v[e] = row < n && c0 + e < n ? src[e] : 0.f;
        }
#pragma unroll
        for (int e = 0; e < 4; e++) c[r][e] = row < n && c0 + e < n ? Code::encode(v[e], bad) : Code::kPad;
        if (c0 < Kh) {
          const uint2 w = make_uint2(c[r][0] | c[r][1] << 16, c[r][2] | c[r][3] << 16);
          *reinterpret_cast<uint2*>(g.Xc[0] + (long long)row * Kh + c0) = w;
          if (c0 + 4 > n || row >= n) *reinterpret_cast<uint2*>(g.Xc[1] + (long long)row * Kh + c0) = w;
        }
      }
      const uint4 w = make_uint4(c[0][0] | c[1][0] << 16, c[0][1] | c[1][1] << 16, c[0][2] | c[1][2] << 16,
                                 c[0][3] | c[1][3] << 16);
      *reinterpret_cast<uint4*>(g.Pc[0] + (long long)p * Np + c0) = w;
      if (c0 + 4 > n || 2 * p + 1 >= n) *reinterpret_cast<uint4*>(g.Pc[1] + (long long)p * Np + c0) = w;
    }
    if (__any_sync(0xffffffffu, bad) && lane == 0) atomicMax(&g.ctl->over_neg, (1 << 30) + 1);
  }
  coop_barrier(g.ctl, (unsigned)G, failed);

  int outcome = 0, it = 0;
  if (*(volatile int*)&g.ctl->over_neg > 1 << 30) outcome = 4;  // an entry; 2^30 is step 0's
  uint32_t base = 0;  // loads of the steps before
  while (!outcome && !*failed) {
    const int cur = it & 1;
    const uint16_t* X = cur ? g.Xc[1] : g.Xc[0];
    uint16_t* Xn = cur ? g.Xc[0] : g.Xc[1];
    uint32_t* Pn = cur ? g.Pc[0] : g.Pc[1];
    const CUtensorMap* tmA = cur ? &a1 : &a0;
    const CUtensorMap* tmB = cur ? &b1 : &b0;
    auto locate = [&](int j, int& tile, int& kk) {
      if (j < nwhole) {
        tile = (j / kt) * G + cta;
        kk = j % kt;
      } else {
        const long long u = u0 + (j - nwhole);
        tile = first_split + (int)(u / kt);
        kk = (int)(u % kt);
      }
    };
    auto issue = [&](int j) {
      const uint32_t q = base + j;
      const int s = q % S;
      if (!sk_wait(&empty[s], ((q / S) & 1) ^ 1, failed, 52)) return;
      int tile, kk;
      locate(j, tile, kk);
      uint8_t* sa = smem + s * Cfg::kStage;
      mbar_arrive_expect_tx(&full[s], Cfg::kStage);
      tma_load_2d(sa, tmA, &full[s], kk * kSkBK16, (tile % g.tiles) * 64);
      tma_load_2d(sa + Cfg::kTileBytes, tmB, &full[s], (tile / g.tiles) * 64, kk * (kSkBK16 / 2));
    };
    if (threadIdx.x == 0)
      for (int j = 0; j < min(S, nloads); j++) issue(j);
    int changed = 0;
    uint32_t over = 0;
    for (int j = 0; j < nloads;) {
      int tile, kk;
      locate(j, tile, kk);
      const int m0 = (tile % g.tiles) * 64, n0 = (tile / g.tiles) * 64;
      const int len = min(kt - kk, nloads - j);
      uint32_t acc[8][4];
#pragma unroll
      for (int i = 0; i < 8; i++)
#pragma unroll
        for (int c = 0; c < 4; c++) acc[i][c] = Code::kIdent;
      for (int e = j + len; j < e; j++) {
        const uint32_t q = base + j;
        const int s = q % S;
        if (lane == 0 && (j & (kSimtWarps - 1)) == warp && j >= Cfg::kLag && j - Cfg::kLag + S < nloads)
          issue(j - Cfg::kLag + S);
        sk_wait(&full[s], (q / S) & 1, failed, 53);
        const uint8_t* As = smem + s * Cfg::kStage;
        sk_ktile16<OP, 64, true>(acc, As, As + Cfg::kTileBytes, ty, tx, 0, kg, 8);
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[s]);
      }
      // fold the four k groups: column pairs of codes through shared memory
      __syncthreads();
#pragma unroll
      for (int i = 0; i < 8; i++)
        *reinterpret_cast<uint2*>(red + (kg * 64 + ty + 8 * i) * kPitch + 2 * tx) =
            make_uint2(Code::pair(acc[i][0], acc[i][1]), Code::pair(acc[i][2], acc[i][3]));
      __syncthreads();
      const uint32_t* src = red + (threadIdx.x >> 3) * kPitch + (threadIdx.x & 7) * 4;
      uint4 v = *reinterpret_cast<const uint4*>(src);
      auto join = [&](const uint4& y) {
        v.x = Code::join(v.x, y.x), v.y = Code::join(v.y, y.y), v.z = Code::join(v.z, y.z), v.w = Code::join(v.w, y.w);
      };
#pragma unroll
      for (int q = 1; q < 4; q++) join(*reinterpret_cast<const uint4*>(src + q * 64 * kPitch));
      if (len < kt) {  // part of a tile
        const long long t0 = (long long)(tile - first_split) * kt;
        const int c_lo = (int)(((t0 + 1) * G - 1) / units), c_hi = (int)(((t0 + kt) * G - 1) / units);
        auto slot_of = [&](int c) -> uint4* {
          return g.part + (size_t)(2 * c + (units * c / G > t0 ? 0 : 1)) * kSimtThreads;
        };
        __stcg(slot_of(cta) + threadIdx.x, v);
        __threadfence();
        __syncthreads();
        // every step adds one arrival of each contributor
        if (threadIdx.x == 0)
          s_last = atomicAdd(&g.counters[tile - first_split], 1) == (it + 1) * (c_hi - c_lo + 1) - 1;
        __syncthreads();
        if (!s_last) continue;
        __threadfence();
        for (int c = c_lo; c <= c_hi; c++)
          if (c != cta) join(__ldcg(slot_of(c) + threadIdx.x));
      }
      // 8 columns of one row: X_{t+1} in both layouts, change test against X_t
      const int row = m0 + (threadIdx.x >> 3), col = n0 + (threadIdx.x & 7) * 8;
      constexpr uint32_t kPad2 = Code::kPad * 0x00010001u;
      const bool in = row < n && col < n;
      const uint4 old = in ? __ldcg(reinterpret_cast<const uint4*>(X + (long long)row * Kh + col))
                           : make_uint4(kPad2, kPad2, kPad2, kPad2);
      const uint32_t ov[4] = {old.x, old.y, old.z, old.w}, mv[4] = {v.x, v.y, v.z, v.w};
      uint32_t w[4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int c = col + 2 * q;
        const uint32_t keep = !in ? 0u : c + 1 < n ? 0xffffffffu : c < n ? 0xffffu : 0u;
        uint32_t b = 0;
        w[q] = Code::finish(mv[q], ov[q], b);
        over |= b & keep;
        w[q] = (w[q] & keep) | (kPad2 & ~keep);
        if (g.conv == SIMD2_CONV_TOL && (OP == SIMD2_MAX_MIN || OP == SIMD2_MIN_MAX)) {
          changed |= conv_changed(g.conv, Code::entry(ov[q] & 0xffffu), Code::entry(w[q] & 0xffffu)) ||
                     conv_changed(g.conv, Code::entry(ov[q] >> 16), Code::entry(w[q] >> 16));
        } else {
          changed |= w[q] != ov[q];
        }
      }
      if (in) *reinterpret_cast<uint4*>(Xn + (long long)row * Kh + col) = make_uint4(w[0], w[1], w[2], w[3]);
      uint32_t d[4];  // the next row's, 8 lanes on
#pragma unroll
      for (int q = 0; q < 4; q++) d[q] = __shfl_down_sync(0xffffffffu, w[q], 8);
      if (in && !(row & 1)) {
        uint4* dst = reinterpret_cast<uint4*>(Pn + (long long)(row >> 1) * Np + col);
        dst[0] = make_uint4(__byte_perm(w[0], d[0], 0x5410), __byte_perm(w[0], d[0], 0x7632),
                            __byte_perm(w[1], d[1], 0x5410), __byte_perm(w[1], d[1], 0x7632));
        dst[1] = make_uint4(__byte_perm(w[2], d[2], 0x5410), __byte_perm(w[2], d[2], 0x7632),
                            __byte_perm(w[3], d[3], 0x5410), __byte_perm(w[3], d[3], 0x7632));
      }
    }
    base += nloads;
    if (__any_sync(0xffffffffu, changed) && lane == 0) atomicMax(&g.ctl->last_changed, it + 1);
    if (__any_sync(0xffffffffu, over != 0) && lane == 0) atomicMax(&g.ctl->over_neg, (1 << 30) - it);
    it++;
    coop_barrier(g.ctl, (unsigned)(it + 1) * (unsigned)G, failed);
    // a CTA already in the next step may have raised either word further, never
    // past what this step decides (a step is only begun after a changed one)
    const int ov = *(volatile int*)&g.ctl->over_neg;
    if (ov && ov >= (1 << 30) - (it - 1)) outcome = 3;
    else if (*(volatile int*)&g.ctl->last_changed < it) outcome = 1;
    else if (it >= g.max_iter) outcome = 2;
  }
  if (*failed) {
    // this CTA's share of X is not written, whatever the others decided
    if (threadIdx.x == 0) {
      g.out[2] = 1;
      for (int s = 0; s < S; s++)
        for (int p = 0; p < 2; p++) mbar_wait(&full[s], p, 1000000ull);
    }
    return;
  }
  if (outcome < 3) {  // X from its codes
    const uint16_t* R = it & 1 ? g.Xc[1] : g.Xc[0];
    const bool vec = (g.ldx % 4 == 0) && (reinterpret_cast<uintptr_t>(g.X) % 16 == 0);
    const int quads = (n + 3) >> 2;
    const long long total = (long long)n * quads;
    for (long long t = cta * (long long)kSimtThreads + threadIdx.x; t < total; t += (long long)G * kSimtThreads) {
      const int i = (int)(t / quads), c0 = (int)(t - (long long)i * quads) * 4;
      const uint2 w = __ldcg(reinterpret_cast<const uint2*>(R + (long long)i * Kh + c0));
      const float v[4] = {Code::entry(w.x & 0xffffu), Code::entry(w.x >> 16), Code::entry(w.y & 0xffffu),
                          Code::entry(w.y >> 16)};
      float* dst = g.X + (long long)i * g.ldx + c0;
      if (vec && c0 + 4 <= n) {
        *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
      } else {
#pragma unroll
        for (int e = 0; e < 4; e++)
          if (c0 + e < n) dst[e] = v[e];
      }
    }
  }
  if (cta == 0 && threadIdx.x == 0) {
    g.out[0] = it;
    g.out[1] = outcome;
  }
}

}  // namespace simd2
