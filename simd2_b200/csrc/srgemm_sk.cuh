// srgemm_sk.cuh -- the CUDA-core srgemm of the six min/max semirings: a
// persistent kernel that spreads the (tile, k-tile) units of a product evenly
// over the SMs, on FP32 operands or on 16-bit codes of them.
//
// 16-bit codes.  min_plus and max_plus on non-negative integers up to 16383
// (and the semiring's add identity), and max_min / min_max on values that are
// exactly FP16, are computed on two 16-bit codes per 32-bit word with the
// packed integer min/max instructions, two k per lane per instruction.  The
// sums of two codes stay below 2^16 and decode to the same float the FP32
// operation gives, and a selection semiring only ever returns an entry, so the
// result has the FP32 path's bits.  The prep kernel writes the codes and notes,
// per block, whether an entry has none; the main kernel reads those notes and
// takes the FP32 operands instead if any is set, so the call stays
// asynchronous.  A packed FP32 add and a three-operand FP32 min take two
// dispatch cycles each for 2 pairs per lane; __viaddmin_u16x2 takes two
// for the same 2 pairs, and two 32-bit adds with a three-operand u16x2 min four
// for 4 pairs (the two forms are mixed, see Code16<>::mac): a register-tile
// loop fed from shared memory measured 124 pairs per clock and SM against 59
// for the FP32 kernel.  Selection: two s16x2 min and a three-operand max for 4
// pairs, 80 against 56 for min/max.f16x2.  Bound by the dispatch of these
// instructions.  Measured, whole calls: min_plus 4096^3 with C 4017 -> 2072 us
// (117 pairs per clock and SM in the kernel), max_min 1000 x 1203 x 1501 with C
// 247 -> 117 us (80 tiles on 148 SMs before, an even split now).
#pragma once
#include "prep.cuh"
#include "srgemm_simt.cuh"

namespace simd2 {

// ---------------------------------------------------------------------------
// 16-bit codes of one operand entry
// ---------------------------------------------------------------------------
template <int OP>
struct Code16 {
  static constexpr bool kHas = false;
};

__device__ __forceinline__ bool int_code(float x, uint32_t& v) {
  const int i = __float2int_rz(x);  // NaN -> 0, infinities saturate
  v = (uint32_t)i;
  return v <= 16383u && __float_as_uint((float)i) == __float_as_uint(x);  // -0.0 and fractions fail
}

// min_plus: v -> v, +inf -> 0x7fff.  A sum is finite below 0x7fff; anything
// that holds a +inf is at least 0x7fff (at most 0xfffe).
template <>
struct Code16<SIMD2_MIN_PLUS> {
  static constexpr bool kHas = true;
  static constexpr uint32_t kPad = 0x7fffu;
  static constexpr uint32_t kIdent = 0xffffffffu;
  __device__ static float entry(uint32_t c) { return c >= 0x7fffu ? __int_as_float(0x7f800000) : (float)c; }
  __device__ static uint32_t encode(float x, bool& bad) {
    if (__float_as_uint(x) == 0x7f800000u) return 0x7fffu;
    uint32_t v;
    bad |= !int_code(x, v);
    return v & 0x3fffu;
  }
  __device__ static float decode(uint32_t acc) {
    const uint32_t m = min(acc & 0xffffu, acc >> 16);
    return m >= 0x7fffu ? __int_as_float(0x7f800000) : (float)m;
  }
  // Two neighbouring columns' accumulators, each over its two halves, as one word.
  __device__ static uint32_t pair(uint32_t a0, uint32_t a1) {
    return join(__byte_perm(a0, a1, 0x5410), __byte_perm(a0, a1, 0x7632));
  }
  __device__ static uint32_t join(uint32_t x, uint32_t y) { return __vminu2(x, y); }
  // Such a word combined with the codes `old`; over gets a bit where a result is
  // finite and has no code.
  __device__ static uint32_t finish(uint32_t m, uint32_t old, uint32_t& over) {
    const uint32_t r = __vminu2(__vminu2(m, 0x7fff7fffu), old);
    over |= r & 0x40004000u & ~((r + 0x00010001u) >> 1);  // bit 14 set, but not 0x7fff
    return r;
  }
  // Folds the pairs (x, y) and (x2, y2) into acc.  Odd columns use the fused
  // add-min, even ones two adds (no carry leaves a half) and a three-operand
  // min: half of each ran at 124 pairs per clock, either alone at 113.
  __device__ static uint32_t mac(uint32_t acc, uint32_t x, uint32_t y, uint32_t x2, uint32_t y2, bool odd) {
    if (odd) return __viaddmin_u16x2(x2, y2, __viaddmin_u16x2(x, y, acc));
    return __vimin3_u16x2(acc, x + y, x2 + y2);
  }
};

// max_plus: v -> v + 0x4000, -inf -> 0.  A finite sum is at least 0x8000;
// anything that holds a -inf is below.
template <>
struct Code16<SIMD2_MAX_PLUS> {
  static constexpr bool kHas = true;
  static constexpr uint32_t kPad = 0u;
  static constexpr uint32_t kIdent = 0u;
  __device__ static float entry(uint32_t c) { return c < 0x4000u ? __int_as_float(0xff800000) : (float)(c - 0x4000u); }
  __device__ static uint32_t encode(float x, bool& bad) {
    if (__float_as_uint(x) == 0xff800000u) return 0u;
    uint32_t v;
    bad |= !int_code(x, v);
    return (v & 0x3fffu) | 0x4000u;
  }
  __device__ static float decode(uint32_t acc) {
    const uint32_t m = max(acc & 0xffffu, acc >> 16);
    return m < 0x8000u ? __int_as_float(0xff800000) : (float)(m - 0x8000u);
  }
  __device__ static uint32_t pair(uint32_t a0, uint32_t a1) {
    return join(__byte_perm(a0, a1, 0x5410), __byte_perm(a0, a1, 0x7632));
  }
  __device__ static uint32_t join(uint32_t x, uint32_t y) { return __vmaxu2(x, y); }
  __device__ static uint32_t finish(uint32_t m, uint32_t old, uint32_t& over) {
    const uint32_t finite = ((m >> 15) & 0x00010001u) * 0xffffu;  // halves that hold a finite sum
    over |= m & finite & 0x40004000u;                             // past 16383
    return __vmaxu2(((m & 0x3fff3fffu) | 0x40004000u) & finite, old);
  }
  __device__ static uint32_t mac(uint32_t acc, uint32_t x, uint32_t y, uint32_t x2, uint32_t y2, bool odd) {
    if (odd) return __viaddmax_u16x2(x2, y2, __viaddmax_u16x2(x, y, acc));
    return __vimax3_u16x2(acc, x + y, x2 + y2);
  }
};

// Selection semirings: the FP16 bits as an order-preserving signed 16-bit
// integer (negative values with their magnitude bits flipped).
struct SelectCode16 {
  static constexpr bool kHas = true;
  __device__ static uint32_t encode(float x, bool& bad) {
    const __half h = __float2half_rn(x);
    // a NaN whose bits survive the trip (the half 0x7fff) has no code either
    bad |= __float_as_uint(__half2float(h)) != __float_as_uint(x) || x != x;
    return code(__half_as_ushort(h));
  }
  __device__ static uint32_t code(uint32_t u) { return u ^ ((u & 0x8000u) ? 0x7fffu : 0u); }
  __device__ static float entry(uint32_t c) { return value((int)c); }
  __device__ static float value(int s) { return __half2float(__ushort_as_half((unsigned short)code((uint32_t)s & 0xffffu))); }
};
template <>
struct Code16<SIMD2_MAX_MIN> : SelectCode16 {
  static constexpr uint32_t kPad = 0x83ffu;  // -inf
  static constexpr uint32_t kIdent = 0x83ff83ffu;
  __device__ static float decode(uint32_t acc) { return value(max((int)(int16_t)(acc & 0xffffu), (int)acc >> 16)); }
  __device__ static uint32_t pair(uint32_t a0, uint32_t a1) {
    return join(__byte_perm(a0, a1, 0x5410), __byte_perm(a0, a1, 0x7632));
  }
  __device__ static uint32_t join(uint32_t x, uint32_t y) { return __vmaxs2(x, y); }
  __device__ static uint32_t finish(uint32_t m, uint32_t old, uint32_t&) { return join(m, old); }
  __device__ static uint32_t mac(uint32_t acc, uint32_t x, uint32_t y, uint32_t x2, uint32_t y2, bool) {
    return __vimax3_s16x2(acc, __vmins2(x, y), __vmins2(x2, y2));
  }
};
template <>
struct Code16<SIMD2_MIN_MAX> : SelectCode16 {
  static constexpr uint32_t kPad = 0x7c00u;  // +inf
  static constexpr uint32_t kIdent = 0x7c007c00u;
  __device__ static float decode(uint32_t acc) { return value(min((int)(int16_t)(acc & 0xffffu), (int)acc >> 16)); }
  __device__ static uint32_t pair(uint32_t a0, uint32_t a1) {
    return join(__byte_perm(a0, a1, 0x5410), __byte_perm(a0, a1, 0x7632));
  }
  __device__ static uint32_t join(uint32_t x, uint32_t y) { return __vmins2(x, y); }
  __device__ static uint32_t finish(uint32_t m, uint32_t old, uint32_t&) { return join(m, old); }
  __device__ static uint32_t mac(uint32_t acc, uint32_t x, uint32_t y, uint32_t x2, uint32_t y2, bool) {
    return __vimin3_s16x2(acc, __vmaxs2(x, y), __vmaxs2(x2, y2));
  }
};

__host__ __device__ constexpr bool has_code16(int op) {
  return op == SIMD2_MIN_PLUS || op == SIMD2_MAX_PLUS || op == SIMD2_MAX_MIN || op == SIMD2_MIN_MAX;
}

// ---------------------------------------------------------------------------
// operand preparation: one launch
// ---------------------------------------------------------------------------
constexpr int kSkBK16 = 64;         // k of a 16-bit k-tile (128-byte rows)
constexpr int kSkMaxPrepBlocks = 1184;  // 8 blocks of 256 threads on each SM
constexpr int kSkMaxCounters = 512;

template <typename T>
struct SkPrepArgs {
  const T* A;
  long long lda;
  const T* B;
  long long ldb;
  int M, N, K;
  int Kh, Kp, Np;    // K padded to 64 / 32, N padded to 128
  uint16_t* A16;     // [M][Kh] codes (null: no 16-bit copies)
  uint32_t* B16;     // [Kh/2][Np] words (code of B[2p][j], code of B[2p+1][j])
  float* B32;        // [Kp/2][2 Np] k-pair interleaved FP32
  float* A32;        // [M][Kp] packed FP32 (null: TMA reads A itself)
  float pad;         // FP32 padding of k >= K
  unsigned* notes;   // per block: 1 when an entry has no code
  int* counters;     // arrivals per split tile, cleared here
  int ncounters;
  const int* gate;
};

// 4 elements, aligned to 4 * sizeof(T).
__device__ __forceinline__ void load4(const float* p, float (&x)[4]) {
  const float4 u = __ldg(reinterpret_cast<const float4*>(p));
  x[0] = u.x, x[1] = u.y, x[2] = u.z, x[3] = u.w;
}
__device__ __forceinline__ void load4(const __half* p, float (&x)[4]) {
  const uint2 u = __ldg(reinterpret_cast<const uint2*>(p));
  x[0] = __half2float(__ushort_as_half((unsigned short)(u.x & 0xffffu)));
  x[1] = __half2float(__ushort_as_half((unsigned short)(u.x >> 16)));
  x[2] = __half2float(__ushort_as_half((unsigned short)(u.y & 0xffffu)));
  x[3] = __half2float(__ushort_as_half((unsigned short)(u.y >> 16)));
}

// Rows of A to codes (8 per thread), 4 columns x 2 k of B to both B layouts,
// rows of A to the packed FP32 copy (4 per thread) where TMA cannot read A.
template <int OP, typename T>
__global__ void __launch_bounds__(256) sk_prep_kernel(SkPrepArgs<T> g) {
  if (g.gate && *g.gate == 0) return;
  bool bad = false;
  const long long tid = blockIdx.x * 256LL + threadIdx.x, step = gridDim.x * 256LL;
  for (long long t = tid; t < g.ncounters; t += step) g.counters[t] = 0;
  // 4 elements of B at a time where its rows allow (16 bytes, or 8 of halves)
  const bool vb = (g.ldb % 4 == 0) && (reinterpret_cast<uintptr_t>(g.B) % (4 * sizeof(T)) == 0);
  constexpr bool k16 = has_code16(OP);
  if constexpr (k16) {
    if (g.A16) {
      const int groups = g.Kh >> 3;
      const long long total = (long long)g.M * groups;
      // a thread that met an entry without a code leaves its other codes out
      for (long long t = tid; t < total && !bad; t += step) {
        const int i = (int)(t / groups);
        const int k0 = (int)(t - (long long)i * groups) * 8;
        const int left = g.K - k0;
        float x[8];
        load8(g.A + (long long)i * g.lda + k0, left, x);
        uint32_t c[8];
        if (left >= 8) {
#pragma unroll
          for (int e = 0; e < 8; e++) c[e] = Code16<OP>::encode(x[e], bad);
        } else {
#pragma unroll
          for (int e = 0; e < 8; e++) c[e] = e < left ? Code16<OP>::encode(x[e], bad) : Code16<OP>::kPad;
        }
        reinterpret_cast<uint4*>(g.A16)[t] =
            make_uint4(c[0] | c[1] << 16, c[2] | c[3] << 16, c[4] | c[5] << 16, c[6] | c[7] << 16);
      }
    }
  }
  {
    const int quads = g.Np >> 2;
    const int prows = (k16 && g.B16 ? g.Kh : g.Kp) >> 1;
    const long long total = (long long)prows * quads;
    for (long long t = tid; t < total; t += step) {
      const int p = (int)(t / quads);
      const int j = (int)(t - (long long)p * quads) * 4;
      float x[2][4];
      bool in[2][4];
#pragma unroll
      for (int r = 0; r < 2; r++) {
        const int k = 2 * p + r;
        const T* row = g.B + (long long)k * g.ldb;
        if (vb && k < g.K && j + 4 <= g.N) {
          load4(row + j, x[r]);
#pragma unroll
          for (int e = 0; e < 4; e++) in[r][e] = true;
        } else {
#pragma unroll
          for (int e = 0; e < 4; e++) {
            in[r][e] = k < g.K && j + e < g.N;
            x[r][e] = in[r][e] ? (float)row[j + e] : g.pad;
          }
        }
      }
      if (p < (g.Kp >> 1)) {
        float4* o = reinterpret_cast<float4*>(g.B32) + 2 * t;
        o[0] = make_float4(x[0][0], x[1][0], x[0][1], x[1][1]);
        o[1] = make_float4(x[0][2], x[1][2], x[0][3], x[1][3]);
      }
      if constexpr (k16) {
        if (g.B16 && !bad) {
          uint32_t w[4];
#pragma unroll
          for (int e = 0; e < 4; e++) {
            const uint32_t lo = in[0][e] ? Code16<OP>::encode(x[0][e], bad) : Code16<OP>::kPad;
            const uint32_t hi = in[1][e] ? Code16<OP>::encode(x[1][e], bad) : Code16<OP>::kPad;
            w[e] = lo | hi << 16;
          }
          reinterpret_cast<uint4*>(g.B16)[t] = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
    }
  }
  if (g.A32) {
    const int quads = g.Kp >> 2;
    const long long total = (long long)g.M * quads;
    for (long long t = tid; t < total; t += step) {
      const int i = (int)(t / quads);
      const int k = (int)(t - (long long)i * quads) * 4;
      const T* row = g.A + (long long)i * g.lda + k;
      float x[4];
#pragma unroll
      for (int e = 0; e < 4; e++) x[e] = k + e < g.K ? (float)row[e] : g.pad;
      reinterpret_cast<float4*>(g.A32)[t] = make_float4(x[0], x[1], x[2], x[3]);
    }
  }
  if (g.notes) {
    const int any = __syncthreads_or(bad);
    if (threadIdx.x == 0) g.notes[blockIdx.x] = any ? 1u : 0u;
  }
}

// ---------------------------------------------------------------------------
// main kernel
// ---------------------------------------------------------------------------
// Output tiles of TILE x TILE (128 or 64).  A thread always holds an 8 x 4
// register tile; with TILE = 64 four groups of 4 warps each take a quarter of
// every k-tile and fold their partial tiles through shared memory, so a small
// product yields four times as many tiles at the same inner loop.
template <int TILE>
struct SkCfg {
  static constexpr int kRows = TILE / 8;  // stride of a thread's 8 rows
  static constexpr int kGroups = (128 / TILE) * (128 / TILE);
  static constexpr int kTileBytes = TILE * 128;  // A or B tile of one stage
  static constexpr int kStage = 2 * kTileBytes;
  static constexpr int kStages = TILE == 128 ? 6 : 8;
  static constexpr int kLag = TILE == 128 ? 2 : 4;  // units between a stage's use and its refill
  static constexpr int kPitch = TILE + 4;
  static constexpr int kRedBytes = kGroups > 1 ? kGroups * TILE * kPitch * 4 : 0;
  static constexpr size_t kSmem = (size_t)kStages * kStage + kRedBytes + 2 * kStages * 8 + 1024;
};

struct SkArgs {
  int M, N, K;
  int tiles_m, tiles_n;
  int whole;              // tiles every CTA computes alone; the rest is split evenly by units
  const unsigned* notes;  // prep blocks' notes (null: no 16-bit copies)
  int nnotes;
  int* counters;          // arrivals per split tile
  float* part;            // partial tiles: two slots of TILE x TILE floats per CTA (null: no tile is split)
  int pair;               // the FP32 kernel follows: this one takes codes only
};

// One k-tile of a warp's register tile on 16-bit codes: chunk q of an A row
// (8 k, 16 bytes) lies at chunk q ^ (row & 7); B pair row pr holds TILE words.
// A warp group takes chunks kg, kg + kGroups, ... below nq (FULL: all 8).
// ROWS < 8 leaves out the rows kRows * i, i >= ROWS.
template <int OP, int TILE, bool FULL, int ROWS = 8>
__device__ __forceinline__ void sk_ktile16(uint32_t (&acc)[8][4], const uint8_t* As, const uint8_t* Bs, int ty, int tx,
                                           int cbase, int kg, int nq) {
  constexpr int KG = SkCfg<TILE>::kGroups;
  const int swz = ty & 7;
  const uint8_t* bp = Bs + (cbase + 4 * tx) * 4;
#pragma unroll(FULL ? 2 : 1)
  for (int q = kg; q < (FULL ? 8 : nq); q += KG) {
    uint4 a[ROWS];
#pragma unroll
    for (int i = 0; i < ROWS; i++)
      a[i] = *reinterpret_cast<const uint4*>(As + (ty + SkCfg<TILE>::kRows * i) * 128 + ((q ^ swz) << 4));
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const uint4 u = *reinterpret_cast<const uint4*>(bp + (4 * q + 2 * h) * (TILE * 4));
      const uint4 v = *reinterpret_cast<const uint4*>(bp + (4 * q + 2 * h + 1) * (TILE * 4));
      const uint32_t b0[4] = {u.x, u.y, u.z, u.w}, b1[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int i = 0; i < ROWS; i++) {
        const uint32_t x = h ? a[i].z : a[i].x, x2 = h ? a[i].w : a[i].y;
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = Code16<OP>::mac(acc[i][j], x, b0[j], x2, b1[j], j & 1);
      }
    }
  }
}

// The same on FP32 operands: chunk q = 4 k of an A row; B' pair row p holds
// 2 TILE floats (see srgemm_simt.cuh).  Columns 32c + 2tx + e of the warp's 64.
template <int OP, int TILE, bool FULL, int ROWS = 8>
__device__ __forceinline__ void sk_ktile32(float (&acc)[8][4], const uint8_t* As, const uint8_t* Bs, int ty, int tx,
                                           int cbase, int kg, int nq) {
  constexpr int KG = SkCfg<TILE>::kGroups;
  const int swz = ty & 7;
#pragma unroll(FULL ? 2 : 1)
  for (int q = kg; q < (FULL ? 8 : nq); q += KG) {
    float4 a[ROWS];
#pragma unroll
    for (int i = 0; i < ROWS; i++)
      a[i] = *reinterpret_cast<const float4*>(As + (ty + SkCfg<TILE>::kRows * i) * 128 + ((q ^ swz) << 4));
#pragma unroll
    for (int h = 0; h < 2; h++) {
      float4 b[2];
#pragma unroll
      for (int c = 0; c < 2; c++)
        b[c] = *reinterpret_cast<const float4*>(Bs + ((2 * q + h) * (2 * TILE) + (cbase + 32 * c + 2 * tx) * 2) * 4);
#pragma unroll
      for (int i = 0; i < ROWS; i++) {
        const float2 ap = h == 0 ? make_float2(a[i].x, a[i].y) : make_float2(a[i].z, a[i].w);
#pragma unroll
        for (int c = 0; c < 2; c++) {
          acc[i][2 * c] = Mac<OP>::mac2(acc[i][2 * c], ap, make_float2(b[c].x, b[c].y));
          acc[i][2 * c + 1] = Mac<OP>::mac2(acc[i][2 * c + 1], ap, make_float2(b[c].z, b[c].w));
        }
      }
    }
  }
}

// A wait that records its failure: once one ran out, later ones return at once,
// so the kernel ends in bounded time.
__device__ __noinline__ bool sk_wait_slow(uint64_t* bar, uint32_t parity, volatile int* failed, int site) {
  if (*failed) return false;
  if (mbar_wait(bar, parity)) return true;
  report_timeout(site);
  *failed = 1;
  return false;
}
__device__ __forceinline__ bool sk_wait(uint64_t* bar, uint32_t parity, volatile int* failed, int site) {
  return mbar_try_wait(bar, parity) || sk_wait_slow(bar, parity, failed, site);
}

// (+) C, the store and the change test of a finished tile.  v[r][2c], v[r][2c+1]
// are neighbouring columns; all C pairs are loaded before any is used, so their
// latencies overlap.  blocks: bit 4 g + q set when an element of the 128-tile's
// 32 x 32 block (row group g, column group q) changed.
template <int OP, int TILE, bool I16, int R>
__device__ __forceinline__ void sk_epilogue(const float (&v)[R][4], int M, int N, const EpilogueArgs& ep, int m0,
                                            int n0, int ty, int tx, int cbase, int& changed, uint32_t& blocks) {
  using Cfg = SkCfg<TILE>;
  const bool track = ep.changed != nullptr;
  const int do_epi = ep.do_epilogue, conv_mode = ep.conv_mode;
  auto at = [&](int r, int c, int& row, int& col) {
    if constexpr (Cfg::kGroups == 1) {
      row = m0 + ty + Cfg::kRows * r;
      col = n0 + cbase + (I16 ? 4 * tx + 2 * c : 32 * c + 2 * tx);
    } else {
      row = m0 + (threadIdx.x >> 3);
      col = n0 + (threadIdx.x & 7) * 8 + 4 * r + 2 * c;
    }
  };
  float2 cpre[R][2];
#pragma unroll
  for (int r = 0; r < R; r++)
#pragma unroll
    for (int c = 0; c < 2; c++) {
      int row, col;
      at(r, c, row, col);
      cpre[r][c] = make_float2(0.f, 0.f);
      if (do_epi && row < M) {
        const float* cp = ep.C + (long long)row * ep.ldc + col;
        if (ep.vec2 && col + 1 < N) {
          cpre[r][c] = *reinterpret_cast<const float2*>(cp);
        } else {
          if (col < N) cpre[r][c].x = cp[0];
          if (col + 1 < N) cpre[r][c].y = cp[1];
        }
      }
    }
#pragma unroll
  for (int r = 0; r < R; r++)
#pragma unroll
    for (int c = 0; c < 2; c++) {
      int row, col;
      at(r, c, row, col);
      if (row < M && col < N) {
        float* dp = ep.D + (long long)row * ep.ldd + col;
        float2 o;
        int ch = 0;
        o.x = epilogue_value<OP>(do_epi, conv_mode, track, v[r][2 * c], cpre[r][c].x, ch);
        if (col + 1 < N) {
          o.y = epilogue_value<OP>(do_epi, conv_mode, track, v[r][2 * c + 1], cpre[r][c].y, ch);
          if (ep.vec2) {
            *reinterpret_cast<float2*>(dp) = o;
          } else {
            dp[0] = o.x;
            dp[1] = o.y;
          }
        } else {
          dp[0] = o.x;
        }
        if (ch) {
          changed = 1;
          if constexpr (Cfg::kGroups == 1)
            blocks |= 1u << (((r >> 1) << 2) | ((cbase >> 5) + (I16 ? tx >> 3 : c)));
        }
      }
    }
}

// Walks this CTA's units: `whole` tiles of its own (tile w * G + cta), then an
// equal share of the units of the remaining tiles, which may begin and end
// inside a tile.  A CTA that computed part of a tile leaves its partial tile in
// its slot and counts itself in; the last of the tile's contributors folds the
// others' partials (min / max: any order gives the same bits) and runs the
// epilogue, so no CTA waits for another.
template <int OP, int TILE, bool I16>
__device__ __forceinline__ void sk_run(const CUtensorMap* tmA, const CUtensorMap* tmB, const SkArgs& g,
                                       const EpilogueArgs& ep, uint8_t* smem, uint64_t* full, uint64_t* empty,
                                       float* red, volatile int* failed, int* s_last) {
  using Cfg = SkCfg<TILE>;
  constexpr int S = Cfg::kStages;
  constexpr int BK = I16 ? kSkBK16 : kBK;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tx = lane & 15;
  const int ty = (warp & (Cfg::kRows / 2 - 1)) * 2 + (lane >> 4);
  const int cbase = Cfg::kGroups == 1 ? (warp >> 3) * 64 : 0;
  const int kg = Cfg::kGroups == 1 ? 0 : warp >> 2;
  const int G = gridDim.x, cta = blockIdx.x;
  const int kt = (g.K + BK - 1) / BK;
  const int tiles = g.tiles_m * g.tiles_n;
  // without partial-tile slots every tile is whole: tiles cta, cta + G, ...
  const int first_split = g.part ? g.whole * G : tiles;
  const long long units = (long long)(tiles - first_split) * kt;
  const long long u0 = units * cta / G, u1 = units * (cta + 1) / G;
  const int nwhole = (g.part ? g.whole : (tiles - cta + G - 1) / G) * kt;
  const int nloads = nwhole + (int)(u1 - u0);

  // Grouped raster: 8 consecutive tile rows share each B column panel in L2.
  auto origin = [&](int t, int& m0, int& n0) {
    const int per_group = 8 * g.tiles_n;
    const int gr = t / per_group;
    const int gsize = min(g.tiles_m - gr * 8, 8);
    const int local = t - gr * per_group;
    m0 = (gr * 8 + local % gsize) * TILE;
    n0 = (local / gsize) * TILE;
  };
  // unit j of this CTA's stream: tile and k-tile
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
  // Load j of the stream, issued by one lane.  The warps take turns (warp j % 16
  // refills at unit j): with one warp issuing every load, the few hundred
  // cycles of an issue held back its share of each k-tile; and a stage is
  // refilled kLag units after its use, when no warp is still on it, so the
  // issuing lane never waits (min_plus 4096^3: 2250 us with one warp and the
  // unit before, 2231 by turns, 2149 by turns and two units later).
  auto issue = [&](int j) {
    const int s = j % S;
    if (!sk_wait(&empty[s], ((j / S) & 1) ^ 1, failed, 31)) return;
    int tile, kk, m0, n0;
    locate(j, tile, kk);
    origin(tile, m0, n0);
    uint8_t* sa = smem + s * Cfg::kStage;
    mbar_arrive_expect_tx(&full[s], Cfg::kStage);
    tma_load_2d(sa, tmA, &full[s], kk * BK, m0);
    tma_load_2d(sa + Cfg::kTileBytes, tmB, &full[s], I16 ? n0 : 2 * n0, kk * (BK / 2));
  };
  if (threadIdx.x == 0) {
    prefetch_tensormap(tmA);
    prefetch_tensormap(tmB);
    for (int j = 0; j < min(S, nloads); j++) issue(j);
  }

  int changed = 0;
  int cs = 0;  // ring position of the next unit
  uint32_t cph = 0;
  for (int j = 0; j < nloads;) {
    int tile, kk, m0, n0;
    locate(j, tile, kk);
    origin(tile, m0, n0);
    const int len = min(kt - kk, nloads - j);
    using AccT = typename std::conditional<I16, uint32_t, float>::type;
    AccT acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
      for (int c = 0; c < 4; c++) {
        if constexpr (I16) acc[i][c] = Code16<OP>::kIdent;
        else acc[i][c] = Mac<OP>::identity();
      }
    auto unit = [&](auto full_tile, int nq) {
      constexpr bool FULL = decltype(full_tile)::value;
      // refill the stage of unit j - kLag, which every warp has left by now
      if (lane == 0 && (j & (kSimtWarps - 1)) == warp && j >= Cfg::kLag && j - Cfg::kLag + S < nloads)
        issue(j - Cfg::kLag + S);
      sk_wait(&full[cs], cph, failed, 32);
      const uint8_t* As = smem + cs * Cfg::kStage;
      if constexpr (I16) sk_ktile16<OP, TILE, FULL>(acc, As, As + Cfg::kTileBytes, ty, tx, cbase, kg, nq);
      else sk_ktile32<OP, TILE, FULL>(acc, As, As + Cfg::kTileBytes, ty, tx, cbase, kg, nq);
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[cs]);
      if (++cs == S) {
        cs = 0;
        cph ^= 1;
      }
      j++;
    };
    // whole k-tiles, then the product's last one if it is a partial one (its
    // chunks past K are left out; a branch in the loop for it cost 3.5 %)
    const int e = kk + len, efull = min(e, g.K / BK);
    for (; kk < efull; kk++) unit(std::true_type{}, 8);
    if (kk < e) unit(std::false_type{}, (g.K - kk * BK + BK / 8 - 1) / (BK / 8));
    // the tile as floats
    constexpr int R = Cfg::kGroups == 1 ? 8 : 2;  // float4s held by a thread from here on
    float v[R][4];
    if constexpr (Cfg::kGroups == 1) {
#pragma unroll
      for (int i = 0; i < 8; i++)
#pragma unroll
        for (int c = 0; c < 4; c++) {
          if constexpr (I16) v[i][c] = Code16<OP>::decode(acc[i][c]);
          else v[i][c] = acc[i][c];
        }
    } else {
      __syncthreads();  // the previous tile's partials have been read
#pragma unroll
      for (int i = 0; i < 8; i++) {
        float* row = red + (kg * TILE + ty + Cfg::kRows * i) * Cfg::kPitch;
        if constexpr (I16) {
          *reinterpret_cast<float4*>(row + 4 * tx) =
              make_float4(Code16<OP>::decode(acc[i][0]), Code16<OP>::decode(acc[i][1]),
                          Code16<OP>::decode(acc[i][2]), Code16<OP>::decode(acc[i][3]));
        } else {
          *reinterpret_cast<float2*>(row + 2 * tx) = make_float2(acc[i][0], acc[i][1]);
          *reinterpret_cast<float2*>(row + 32 + 2 * tx) = make_float2(acc[i][2], acc[i][3]);
        }
      }
      __syncthreads();
      // thread: row tid / 8, columns 8 (tid % 8) .. + 7
      const float* src = red + (threadIdx.x >> 3) * Cfg::kPitch + (threadIdx.x & 7) * 8;
#pragma unroll
      for (int r = 0; r < 2; r++) {
        float4 x = *reinterpret_cast<const float4*>(src + 4 * r);
#pragma unroll
        for (int k2 = 1; k2 < Cfg::kGroups; k2++) {
          const float4 y = *reinterpret_cast<const float4*>(src + k2 * TILE * Cfg::kPitch + 4 * r);
          x.x = Mac<OP>::add(x.x, y.x), x.y = Mac<OP>::add(x.y, y.y);
          x.z = Mac<OP>::add(x.z, y.z), x.w = Mac<OP>::add(x.w, y.w);
        }
        v[r][0] = x.x, v[r][1] = x.y, v[r][2] = x.z, v[r][3] = x.w;
      }
    }
    if (len < kt) {  // part of a tile
      const long long t0 = (long long)(tile - first_split) * kt;
      const int c_lo = (int)(((t0 + 1) * G - 1) / units), c_hi = (int)(((t0 + kt) * G - 1) / units);
      auto slot_of = [&](int c) -> float* {
        return g.part + (size_t)(2 * c + (units * c / G > t0 ? 0 : 1)) * (TILE * TILE);
      };
      float* mine = slot_of(cta);
#pragma unroll
      for (int r = 0; r < R; r++)
        __stcg(reinterpret_cast<float4*>(mine) + r * kSimtThreads + threadIdx.x,
               make_float4(v[r][0], v[r][1], v[r][2], v[r][3]));
      __threadfence();
      __syncthreads();
      if (threadIdx.x == 0) *s_last = atomicAdd(&g.counters[tile - first_split], 1) == c_hi - c_lo;
      __syncthreads();
      if (!*s_last) continue;
      __threadfence();
      for (int c = c_lo; c <= c_hi; c++) {
        if (c == cta) continue;
        const float4* src = reinterpret_cast<const float4*>(slot_of(c));
#pragma unroll
        for (int r = 0; r < R; r++) {
          const float4 y = __ldcg(src + r * kSimtThreads + threadIdx.x);
          v[r][0] = Mac<OP>::add(v[r][0], y.x), v[r][1] = Mac<OP>::add(v[r][1], y.y);
          v[r][2] = Mac<OP>::add(v[r][2], y.z), v[r][3] = Mac<OP>::add(v[r][3], y.w);
        }
      }
    }
    uint32_t blocks = 0;
    sk_epilogue<OP, TILE, I16>(v, g.M, g.N, ep, m0, n0, ty, tx, cbase, changed, blocks);
  }
  if (*failed) {
    // copies still in flight must land before this CTA's shared memory is released
    if (threadIdx.x == 0)
      for (int s = 0; s < S; s++)
        for (int p = 0; p < 2; p++) mbar_wait(&full[s], p, 1000000ull);
  }
  if (ep.changed) {
    if (__any_sync(0xffffffffu, changed) && lane == 0) atomicOr(ep.changed, 1);
  }
}

// FP32: on FP32 operands only; else the notes decide on the device.  One kernel with
// both inner loops runs the FP32 one 6 % slower than a kernel of its own (min_plus
// 4096^3 on fractions 4254 us, 3987 apart), and a second launch costs 2 us: large
// products get both (g.pair), of which one returns at once, and a plan without codes
// the FP32 kernel alone.
template <int OP, int TILE, bool FP32>
__global__ void __launch_bounds__(kSimtThreads, 1)
    srgemm_sk_kernel(const __grid_constant__ CUtensorMap a16, const __grid_constant__ CUtensorMap b16,
                     const __grid_constant__ CUtensorMap a32, const __grid_constant__ CUtensorMap b32, SkArgs g,
                     EpilogueArgs ep) {
  using Cfg = SkCfg<TILE>;
  if (ep.gate && *ep.gate == 0) return;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  float* red = reinterpret_cast<float*>(smem + Cfg::kStages * Cfg::kStage);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + Cfg::kStages * Cfg::kStage + Cfg::kRedBytes);
  uint64_t* empty = full + Cfg::kStages;
  __shared__ int s_failed, s_last;
  if (threadIdx.x == 0) {
    for (int s = 0; s < Cfg::kStages; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], kSimtWarps);
    }
    s_failed = 0;
    fence_mbar_init();
  }
  if constexpr (Code16<OP>::kHas) {
    int bad = g.notes == nullptr;
    if (g.notes)
      for (int i = threadIdx.x; i < g.nnotes; i += kSimtThreads) bad |= (int)g.notes[i];
    const bool coded = !__syncthreads_or(bad);
    if constexpr (FP32) {
      if (coded) return;
    } else {
      if (coded) {
        sk_run<OP, TILE, true>(&a16, &b16, g, ep, smem, full, empty, red, &s_failed, &s_last);
        return;
      }
      if (g.pair) return;
    }
  } else {
    __syncthreads();
  }
  sk_run<OP, TILE, false>(&a32, &b32, g, ep, smem, full, empty, red, &s_failed, &s_last);
}

// ---------------------------------------------------------------------------
// block skipping
// ---------------------------------------------------------------------------
struct SkSkipArgs {
  int M, N, K;
  int tiles_m, tiles_n;
  const unsigned* notes;
  int nnotes;
  int* queue;           // next tile (cleared by the prep kernel)
  const uint8_t* occA;  // occupancy maps (null: every k-tile is taken)
  const uint8_t* occB;
};

// The 128 x 128 tiles of a product whose k list differs from tile to tile: a
// tile's list holds the k-tiles with a 32-wide k block whose A block (128 rows)
// and B block (128 columns) both hold an entry other than the annihilator, and
// with ep.dA / ep.dB (a closure's delta step) one of which changed in the step
// before (see EpilogueArgs).  CTAs take tiles from a counter, since the lists'
// lengths are not known to the host.  ep.chgA / ep.chgB: as in srgemm_simt_kernel.
template <int OP, bool I16>
__device__ __forceinline__ void sk_skip_run(const CUtensorMap* tmA, const CUtensorMap* tmB, const SkSkipArgs& g,
                                            const EpilogueArgs& ep, uint8_t* smem, uint64_t* full, uint64_t* empty,
                                            uint16_t* list, int* warp_cnt, volatile int* failed, int* s_tile) {
  using Cfg = SkCfg<128>;
  constexpr int S = Cfg::kStages;
  constexpr int BK = I16 ? kSkBK16 : kBK;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tx = lane & 15;
  const int ty = (warp & 7) * 2 + (lane >> 4);
  const int cbase = (warp >> 3) * 64;
  const int kt = (g.K + BK - 1) / BK;
  const int kb = (g.K + 31) / 32;  // 32-wide k blocks, the maps' grid
  const int tiles = g.tiles_m * g.tiles_n;
  uint32_t base = 0;  // loads issued for earlier tiles
  int changed = 0;
  if (threadIdx.x == 0) {
    prefetch_tensormap(tmA);
    prefetch_tensormap(tmB);
  }
  while (true) {
    if (threadIdx.x == 0) *s_tile = atomicAdd(g.queue, 1);
    __syncthreads();
    const int t = *s_tile;
    if (t >= tiles) break;
    const int per_group = 8 * g.tiles_n;
    const int gr = t / per_group;
    const int gsize = min(g.tiles_m - gr * 8, 8);
    const int local = t - gr * per_group;
    const int tm = gr * 8 + local % gsize, tn = local / gsize;
    const int m0 = tm * 128, n0 = tn * 128;
    int n = 0;
    for (int b0 = 0; b0 < kt; b0 += kSimtThreads) {
      const int k = b0 + threadIdx.x;
      bool need = k < kt && !g.occA;
      if (k < kt && g.occA) {
#pragma unroll
        for (int h = 0; h < BK / 32; h++) {
          const int q = k * (BK / 32) + h;
          if (q < kb) {
            const long long ia = (long long)tm * kb + q, ib = (long long)q * g.tiles_n + tn;
            need |= g.occA[ia] && g.occB[ib] && (!ep.dA || ep.dA[ia] || ep.dB[ib]);
          }
        }
      }
      const unsigned ballot = __ballot_sync(0xffffffffu, need);
      if (lane == 0) warp_cnt[warp] = __popc(ballot);
      __syncthreads();
      int off = 0, total = 0;
      for (int w = 0; w < kSimtWarps; w++) {
        const int c = warp_cnt[w];
        off += w < warp ? c : 0;
        total += c;
      }
      if (need) list[n + off + __popc(ballot & ((1u << lane) - 1u))] = (uint16_t)k;
      n += total;
      __syncthreads();
    }
    auto issue = [&](int i) {
      const uint32_t j = base + i;
      const int s = j % S;
      if (!sk_wait(&empty[s], ((j / S) & 1) ^ 1, failed, 33)) return;
      const int k = list[i];
      uint8_t* sa = smem + s * Cfg::kStage;
      mbar_arrive_expect_tx(&full[s], Cfg::kStage);
      tma_load_2d(sa, tmA, &full[s], k * BK, m0);
      tma_load_2d(sa + Cfg::kTileBytes, tmB, &full[s], I16 ? n0 : 2 * n0, k * (BK / 2));
    };
    if (threadIdx.x == 0)
      for (int i = 0; i < min(S, n); i++) issue(i);
    using AccT = typename std::conditional<I16, uint32_t, float>::type;
    AccT acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
      for (int c = 0; c < 4; c++) {
        if constexpr (I16) acc[i][c] = Code16<OP>::kIdent;
        else acc[i][c] = Mac<OP>::identity();
      }
    for (int i = 0; i < n; i++) {
      const uint32_t j = base + i;
      const int s = j % S;
      if (lane == 0 && (i & (kSimtWarps - 1)) == warp && i >= Cfg::kLag && i - Cfg::kLag + S < n)
        issue(i - Cfg::kLag + S);
      sk_wait(&full[s], (j / S) & 1, failed, 34);
      const uint8_t* As = smem + s * Cfg::kStage;
      // k past K holds the padding codes / NaN, which leave every result as it is
      if constexpr (I16) sk_ktile16<OP, 128, true>(acc, As, As + Cfg::kTileBytes, ty, tx, cbase, 0, 8);
      else sk_ktile32<OP, 128, true>(acc, As, As + Cfg::kTileBytes, ty, tx, cbase, 0, 8);
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[s]);
    }
    base += n;
    float v[8][4];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
      for (int c = 0; c < 4; c++) {
        if constexpr (I16) v[i][c] = Code16<OP>::decode(acc[i][c]);
        else v[i][c] = acc[i][c];
      }
    uint32_t blocks = 0;
    sk_epilogue<OP, 128, I16>(v, g.M, g.N, ep, m0, n0, ty, tx, cbase, changed, blocks);
    if (ep.chgA) {
      // every writer stores 1, so no atomics; a set bit implies an element
      // inside the matrix, so both indices are in range
      const uint32_t m = __reduce_or_sync(0xffffffffu, blocks);
      if (lane == 0 && m) {
#pragma unroll
        for (int q = 0; q < 4; q++) {
          if (m & (0x1111u << q)) ep.chgA[(long long)tm * kb + 4 * tn + q] = 1;
          if (m & (0xfu << (4 * q))) ep.chgB[(long long)(4 * tm + q) * g.tiles_n + tn] = 1;
        }
      }
    }
  }
  if (*failed) {
    if (threadIdx.x == 0)
      for (int s = 0; s < S; s++)
        for (int p = 0; p < 2; p++) mbar_wait(&full[s], p, 1000000ull);
  }
  if (ep.changed) {
    if (__any_sync(0xffffffffu, changed) && lane == 0) atomicOr(ep.changed, 1);
  }
}

template <int OP>
__global__ void __launch_bounds__(kSimtThreads, 1)
    srgemm_sk_skip_kernel(const __grid_constant__ CUtensorMap a16, const __grid_constant__ CUtensorMap b16,
                          const __grid_constant__ CUtensorMap a32, const __grid_constant__ CUtensorMap b32,
                          SkSkipArgs g, EpilogueArgs ep) {
  using Cfg = SkCfg<128>;
  if (ep.gate && *ep.gate == 0) return;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + Cfg::kStages * Cfg::kStage + Cfg::kRedBytes);
  uint64_t* empty = full + Cfg::kStages;
  __shared__ uint16_t list[kMaxSkipKtiles];
  __shared__ int warp_cnt[kSimtWarps];
  __shared__ int s_failed, s_tile;
  if (threadIdx.x == 0) {
    for (int s = 0; s < Cfg::kStages; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], kSimtWarps);
    }
    s_failed = 0;
    fence_mbar_init();
  }
  int bad = g.notes == nullptr;
  if (g.notes)
    for (int i = threadIdx.x; i < g.nnotes; i += kSimtThreads) bad |= (int)g.notes[i];
  if (!__syncthreads_or(bad))
    sk_skip_run<OP, true>(&a16, &b16, g, ep, smem, full, empty, list, warp_cnt, &s_failed, &s_tile);
  else
    sk_skip_run<OP, false>(&a32, &b32, g, ep, smem, full, empty, list, warp_cnt, &s_failed, &s_tile);
}

}  // namespace simd2
