// tc_gemm.cuh -- tensor-core (tcgen05 / TMEM) srgemm paths for sm_100a.
//
// Used for the semirings that are dense contractions:
//   * or_and       : kind::mxf4, true as the FP4 value 1.0 with every block scale
//                    1.0, FP32 accumulate; D = (sum > 0) | C.  Exact: the products
//                    are 0 or 1, a sum of them is exact up to 2^24 and never
//                    shrinks, so it is positive just when a product was 1.  Twice
//                    the rate of kind::i8 on half the operand bytes; what bounds it
//                    is the shared memory's bandwidth (operand reads and TMA writes
//                    of a 256 x 224 pair tile: 165 of 128 bytes a clock at full
//                    rate).  16384^3 step, kernel: kind::i8 2240 us, now 1400;
//                    3000 x 2500 x 2000 int32 call 117 us, now 51.
//   * plus_mul     : kind::f16 with BF16 hi/lo operands, FP32 accumulate:
//                    a*b ~= a_hi*b_hi + a_hi*b_lo + a_lo*b_hi  (three MMAs per k step).
//   * float16 operands (KIND 2): one kind::f16 MMA per k step on the halves
//                    themselves, whose products FP32 holds exactly.
//   * minus_square : the same BF16 hi/lo product gives a.b; the epilogue forms
//                    |a|^2 + |b|^2 - 2 a.b with FP64-accumulated norms and
//                    recomputes sum_k (a-b)^2 exactly in FP32 inside the
//                    cancellation band (small distance relative to the norms).
//
// Persistent: one CTA per SM walks the 128 x 256 tiles of D (grouped raster)
// with 10 warps:
//   warp 0 lane 0  -- TMA producer (2D tiled loads, no multicast, 128-byte
//                     swizzled rows) over every k-tile of every tile, one ring
//                     of stages,
//   warp 1 lane 0  -- MMA issuer (tcgen05.mma, cta_group::1, M=128, N=256 or
//                     224) into one of two TMEM accumulators, so the next
//                     tile's MMAs run while the previous tile is written out,
//   warps 2..9     -- epilogue: tcgen05.ld of the accumulator (warp w reads
//                     TMEM lanes 32(w%4)..+31 = tile rows, the lower or the upper
//                     half of the tile's columns), fused (+) C, stores.
// A is K-major in shared memory, [M][K] as given.  B: or_and's FP4 copy and
// k-NN's references are K-major ([N][K]); the sums read B [K][N] as it is, N-major
// (BT), so that no transposed copy is made (plus_mul 8192^3: the transposing
// BF16 split of B took 163 us, the plain one takes 85).
#pragma once
#include "common.cuh"
#include "prep.cuh"

namespace simd2 {

constexpr int kTcBM = 128;
constexpr int kTcBN = 256;
// Columns of a tile.  or_and takes 224: two accumulators of 224 columns leave
// the 512 TMEM columns room for the block scales.
template <int KIND>
__host__ __device__ constexpr int tc_bn() { return KIND == 1 ? 224 : kTcBN; }
constexpr int kTcScaleCol = 448;  // first TMEM column of the block scales
constexpr int kTcScaleCols = 32;  // 4 columns of A's and 8 of B's, all the same byte
constexpr int kTcEpiWarps = 8;
constexpr int kTcThreads = (2 + kTcEpiWarps) * 32;  // TMA warp, MMA warp, 8 epilogue warps
template <int KIND>
struct TcCfg;
// BF16 hi/lo: BK = 64 elements, two A tiles and two B tiles per stage.  128-byte
// rows halve the rows TMA has to fetch for A against 64-byte ones (BK = 32, twice
// the stages): 4096^3 320 us for 308, 1000 x 800 x 3000 50 for 42.
template <>
struct TcCfg<0> {
  static constexpr int kBK = 64;
  static constexpr int kRowBytes = 128;
  static constexpr int kNumA = 2;
  static constexpr int kNumB = 2;
  static constexpr int kStages = 2;
  static constexpr int kKStep = 16;  // K per tcgen05.mma kind::f16
  // c_format F32 (1), a/b format BF16 (1), K-major A and B, N=256, M=128
  static constexpr uint32_t kIdesc =
      (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kTcBN >> 3) << 17) | ((uint32_t)(kTcBM >> 4) << 24);
};
// FP4 0/1, two per byte: BK = 256 elements, one A and one B tile per stage.
template <>
struct TcCfg<1> {
  static constexpr int kBK = 256;
  static constexpr int kRowBytes = 128;
  static constexpr int kNumA = 1;
  static constexpr int kNumB = 1;
  static constexpr int kStages = 4;
  static constexpr int kKStep = 64;  // K per tcgen05.mma kind::mxf4
  // a/b format E2M1 (1), scale format UE8M0 (bit 23), scale ids 0, K-major, N=224, M=128 (bits 27-28: M / 128)
  static constexpr uint32_t kIdesc = (1u << 7) | (1u << 10) | ((uint32_t)(224 >> 3) << 17) | (1u << 23) |
                                     ((uint32_t)(kTcBM >> 7) << 27);
};

// Float16: BK = 64 elements, one A and one B tile per stage.
template <>
struct TcCfg<2> {
  static constexpr int kBK = 64;
  static constexpr int kRowBytes = 128;
  static constexpr int kNumA = 1;
  static constexpr int kNumB = 1;
  static constexpr int kStages = 4;
  static constexpr int kKStep = 16;
  // c_format F32 (1), a/b format F16 (0)
  static constexpr uint32_t kIdesc =
      (1u << 4) | ((uint32_t)(kTcBN >> 3) << 17) | ((uint32_t)(kTcBM >> 4) << 24);
};

// Instruction descriptor with N = n, B N-major when bt.
template <int KIND>
__host__ __device__ constexpr uint32_t tc_idesc(int n, bool bt) {
  return (TcCfg<KIND>::kIdesc & ~(0x3Fu << 17)) | ((uint32_t)(n >> 3) << 17) | (bt ? 1u << 16 : 0u);
}

template <int KIND>
__host__ __device__ constexpr int tc_a_tile() { return kTcBM * TcCfg<KIND>::kRowBytes; }
template <int KIND>
__host__ __device__ constexpr int tc_b_tile() { return tc_bn<KIND>() * TcCfg<KIND>::kRowBytes; }

// k-tile step in tensor-map elements: BF16 values, or bytes of two FP4 values.
template <int KIND>
__host__ __device__ constexpr int tc_box_x() { return KIND == 1 ? TcCfg<1>::kRowBytes : TcCfg<KIND>::kBK; }
// N-major B: one box holds kBK rows of 64 columns.
template <int KIND>
__host__ __device__ constexpr int tc_b_group() { return TcCfg<KIND>::kBK * 128; }
template <int KIND>
__host__ __device__ constexpr int tc_stage_bytes() {
  return TcCfg<KIND>::kNumA * tc_a_tile<KIND>() + TcCfg<KIND>::kNumB * tc_b_tile<KIND>();
}
template <int KIND>
constexpr size_t tc_smem_bytes() {
  return (size_t)TcCfg<KIND>::kStages * tc_stage_bytes<KIND>() + (size_t)kTcEpiWarps * 32 * 33 * 4 + 1024 + 256;
}

// Shared-memory matrix descriptor for a K-major operand tile written by TMA
// with a 128- or 64-byte swizzle: rows of row_bytes, 8-row core-matrix groups
// 8 * row_bytes apart (stride byte offset), leading byte offset unused (1),
// version 1, layout type 2 = SWIZZLE_128B or 4 = SWIZZLE_64B.  Advancing K
// inside a row moves the start address by the byte offset.
__device__ __forceinline__ uint64_t umma_desc_swizzled(uint32_t smem_addr, int row_bytes) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr >> 4) & 0x3FFFu);
  d |= (uint64_t)1u << 16;                             // leading byte offset (unused for swizzled K-major)
  d |= (uint64_t)((8u * row_bytes) >> 4) << 32;        // stride byte offset
  d |= (uint64_t)1u << 46;                             // descriptor version (sm_100)
  d |= (uint64_t)(row_bytes == 128 ? 2u : 4u) << 61;   // SWIZZLE_128B / SWIZZLE_64B
  return d;
}

// The descriptor of an N-major operand tile: groups of 64 columns (128 bytes,
// 128-byte swizzle) `group_bytes` apart (leading byte offset), 8-k groups 1024
// bytes apart (stride byte offset).  Advancing K by 16 moves the start by 2048.
__device__ __forceinline__ uint64_t umma_desc_nmajor(uint32_t smem_addr, int group_bytes) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr >> 4) & 0x3FFFu);
  d |= (uint64_t)((uint32_t)group_bytes >> 4) << 16;
  d |= (uint64_t)(1024u >> 4) << 32;
  d |= (uint64_t)1u << 46;
  d |= (uint64_t)2u << 61;
  return d;
}

// The descriptor for 128-byte swizzled rows (8-row groups 1024 bytes apart).
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t smem_addr) {
  return umma_desc_swizzled(smem_addr, 128);
}

__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }

// `scales`: TMEM address of the block scales (KIND 1; both operands read the same columns).
template <int KIND>
__device__ __forceinline__ void tc_mma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t accumulate,
                                       uint32_t idesc, uint32_t scales = 0) {
  if constexpr (KIND != 1) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0), "r"(0), "r"(0), "r"(0));
  } else {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::mxf4.block_scale.scale_vec::2X [%0], %1, %2, %3, [%5], [%5], p;\n\t}\n" ::"r"(
            tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(scales));
  }
}

// Sets this warp's 32 TMEM lanes of the scale columns to 1.0 (UE8M0 127): with
// every scale the same, their layout does not matter.
__device__ __forceinline__ void tc_fill_scales(uint32_t taddr) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1};" ::"r"(taddr),
      "r"(0x7f7f7f7fu)
      : "memory");
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// Arrive on `bar` once every tcgen05 operation issued so far by this thread completes.
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

// 32 lanes x 32 consecutive 32-bit columns: thread t of the warp gets lane t.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// 32 lanes x 64 consecutive 32-bit columns in one round trip.
__device__ __forceinline__ void tmem_ld64(uint32_t taddr, uint32_t (&r)[64]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x64.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,"
      "%32,%33,%34,%35,%36,%37,%38,%39,%40,%41,%42,%43,%44,%45,%46,%47,"
      "%48,%49,%50,%51,%52,%53,%54,%55,%56,%57,%58,%59,%60,%61,%62,%63}, [%64];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31]),
        "=r"(r[32]), "=r"(r[33]), "=r"(r[34]), "=r"(r[35]), "=r"(r[36]), "=r"(r[37]), "=r"(r[38]), "=r"(r[39]),
        "=r"(r[40]), "=r"(r[41]), "=r"(r[42]), "=r"(r[43]), "=r"(r[44]), "=r"(r[45]), "=r"(r[46]), "=r"(r[47]),
        "=r"(r[48]), "=r"(r[49]), "=r"(r[50]), "=r"(r[51]), "=r"(r[52]), "=r"(r[53]), "=r"(r[54]), "=r"(r[55]),
        "=r"(r[56]), "=r"(r[57]), "=r"(r[58]), "=r"(r[59]), "=r"(r[60]), "=r"(r[61]), "=r"(r[62]), "=r"(r[63])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

enum TcOrType { kOrU8 = 0, kOrI32 = 1, kOrF32 = 2 };

// Epilogue arguments of the tensor-core paths.
struct TcEpilogue {
  int op;               // SIMD2_PLUS_MUL, SIMD2_MINUS_SQUARE or SIMD2_OR_AND
  int do_epilogue;
  const void* C;        // float (sums) or out_type (or_and)
  long long ldc;
  void* D;
  long long ldd;
  int out_type;         // or_and: type of C and D (kOrU8, kOrI32, kOrF32)
  // minus_square: row norms of A (M), column norms of B (N), and the operands
  // as given (FP32, KIND 2: float16) for the exact recompute inside the
  // cancellation band.
  const float* norm_a;
  const float* norm_b;
  const void* A32;
  long long lda32;
  const void* B32;
  long long ldb32;
  int K;
  float band;           // recompute when dist < band * (|a|^2 + |b|^2)
  int b_rows;           // 1: B32 holds B transposed ([N][K], e.g. k-NN reference points)
  int* changed;         // or_and closure: set to 1 when any D differs from C
  const int* gate;      // nullable: the launch does nothing when it is 0 (a closure past its fixed point)
  // Delta steps of the or_and closure (tc_gemm2_kernel only): chg_row[i] /
  // chg_col[j] receive a 1 when an element of 256-row tile row i / 256-column
  // tile column j changed; with need_row / need_col (the previous step's maps)
  // a tile whose tile row and tile column both stayed unchanged is skipped --
  // every product it would form was formed in that step and is already in C.
  uint8_t* chg_row;
  uint8_t* chg_col;
  const uint8_t* need_row;
  const uint8_t* need_col;
};

// sum_k (a[k] - B[k][col])^2 in FP32, k in order; B is [K][N] (pitch ldb) or, when
// b_rows, stored transposed as [N][K].  One thread waits for its loads alone, so 16
// of each operand are in flight (zeros past K leave the sum as it is).  k-NN with one
// query in twenty on top of a reference, 4 at a time / 16: 16384 x 16000 x 256, k = 32,
// 700 / 648 us, 16384 x 1000 x 64, k = 16, 103 / 96.
template <typename T>
__device__ __forceinline__ float exact_minus_square(const T* a, const T* B, long long ldb, int col, int K,
                                                    int b_rows) {
  constexpr int U = 16;
  const T* b = b_rows ? B + (long long)col * ldb : B + col;
  const long long step = b_rows ? 1 : ldb;
  float s = 0.f;
#pragma unroll 1
  for (int k = 0; k < K; k += U) {
    float x[U], y[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      x[u] = k + u < K ? (float)a[k + u] : 0.f;
      y[u] = k + u < K ? (float)b[(k + u) * step] : 0.f;
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      const float d = __fsub_rn(x[u], y[u]);
      s = __fmaf_rn(d, d, s);
    }
  }
  return s;
}

// or_and: the (sum > 0) flags of one warp's 32 rows x ncols columns, taken out of
// TMEM as bits (lane l: row l, word c: columns 32c..) and parked in the warp's
// shared buffer, row pitch kOrPitch words.  The accumulator is free after this.
constexpr int kOrPitch = 9;
__device__ __forceinline__ void tc_or_bits(uint32_t trow, uint32_t* buf, int lane, int ncols) {
  __syncwarp();  // the previous tile's bits have been read
#pragma unroll 1
  for (int c0 = 0; c0 < ncols; c0 += 32) {
    uint32_t r[32];
    tmem_ld32(trow + c0, r);
    uint32_t w = 0;
#pragma unroll
    for (int j = 0; j < 32; j++) w |= (uint32_t)(r[j] != 0u) << j;
    buf[lane * kOrPitch + (c0 >> 5)] = w;
  }
  __syncwarp();
}

// Writes the parked flags | C.  A row's columns go to the warp's lanes in order,
// four to a lane where D's (and C's) rows allow a word of bytes or an int4 --
// each instruction then covers 128 columns of one row -- else one to a lane;
// C is loaded for 8 rows before any of it is used: the loads' latency bounds a
// product of short k (3000 x 2500 x 2000 int32 call with C, 4 rows / 8: 55.9 / 52.4 us;
// a 1000-vertex closure 231 / 213).  (With a lane per row, every
// store of unaligned rows touched 32 rows: the 3000^3 kernel on bytes 184 us, now 39.)
template <typename T>
__device__ __forceinline__ void tc_or_store(const TcEpilogue& ep, int M, int N, int n0, int row0, const uint32_t* buf,
                                            int lane, int& changed, int ncols) {
  T* D = static_cast<T*>(ep.D);
  const T* C = static_cast<const T*>(ep.C);
  const bool epi = ep.do_epilogue != 0;
  const int rows = min(32, M - row0);
  constexpr int kVec = sizeof(T) == 1 ? 4 : 16;  // bytes of 4 elements
  constexpr int R = 8;  // rows of C in flight
  const bool vec = (n0 + ncols <= N) && ((ep.ldd * (long long)sizeof(T)) % kVec == 0) &&
                   ((reinterpret_cast<uintptr_t>(D) + (size_t)n0 * sizeof(T)) % kVec == 0) &&
                   (!epi || (((ep.ldc * (long long)sizeof(T)) % kVec == 0) &&
                             ((reinterpret_cast<uintptr_t>(C) + (size_t)n0 * sizeof(T)) % kVec == 0)));
  if (vec) {
    using V = typename std::conditional<sizeof(T) == 1, uint32_t, int4>::type;
#pragma unroll 1
    for (int c = lane * 4; c < ncols; c += 128) {
#pragma unroll 1
      for (int r0 = 0; r0 < rows; r0 += R) {
        V old[R];
#pragma unroll
        for (int q = 0; q < R; q++)
          if (epi && r0 + q < rows) old[q] = *reinterpret_cast<const V*>(C + (row0 + r0 + q) * ep.ldc + n0 + c);
#pragma unroll
        for (int q = 0; q < R; q++) {
          if (r0 + q >= rows) break;
          const uint32_t nib = (buf[(r0 + q) * kOrPitch + (c >> 5)] >> (c & 31)) & 15u;
          V* dst = reinterpret_cast<V*>(D + (row0 + r0 + q) * ep.ldd + n0 + c);
          if constexpr (sizeof(T) == 1) {
            uint32_t v = (nib * 0x00204081u) & 0x01010101u;  // bit i to byte i
            if (epi) {
              const uint32_t o = bytes_nonzero_01(old[q]);
              v |= o;
              if (v != o) changed = 1;
            }
            *dst = v;
          } else {
            // a float 1.0 and 0.0 by their bits; -0.0 is false
            constexpr bool kF32 = std::is_same<T, float>::value;
            constexpr int one = kF32 ? 0x3f800000 : 1, mask = kF32 ? 0x7fffffff : -1;
            uint32_t f = nib;
            if (epi)
              f |= (uint32_t)((old[q].x & mask) != 0) | (uint32_t)((old[q].y & mask) != 0) << 1 |
                   (uint32_t)((old[q].z & mask) != 0) << 2 | (uint32_t)((old[q].w & mask) != 0) << 3;
            *dst = make_int4(f & 1 ? one : 0, f & 2 ? one : 0, f & 4 ? one : 0, f & 8 ? one : 0);
          }
        }
      }
    }
  } else {
#pragma unroll 1
    for (int c = lane; c < ncols && n0 + c < N; c += 32) {
#pragma unroll 1
      for (int r0 = 0; r0 < rows; r0 += R) {
        T old[R];
#pragma unroll
        for (int q = 0; q < R; q++)
          if (epi && r0 + q < rows) old[q] = C[(row0 + r0 + q) * ep.ldc + n0 + c];
#pragma unroll
        for (int q = 0; q < R; q++) {
          if (r0 + q >= rows) break;
          uint32_t v = (buf[(r0 + q) * kOrPitch + (c >> 5)] >> (c & 31)) & 1u;
          if (epi) {
            const uint32_t o = is_true(old[q]);
            v |= o;
            if (v != o) changed = 1;
          }
          D[(row0 + r0 + q) * ep.ldd + n0 + c] = static_cast<T>(v);
        }
      }
    }
  }
}

// Epilogue of the 32 rows x ncols columns (a multiple of 32) of one warp: lane l
// holds row row0 + l of the accumulator in TMEM at trow (lane quadrant and column
// base included), columns n0...  release() hands the accumulator back.  Sets changed when an or_and output differs from C.
template <int KIND, typename F>
__device__ __forceinline__ void tc_tile_epilogue(const TcEpilogue& ep, int M, int N, int n0, int row0, uint32_t trow,
                                                 uint32_t* epi_tile, int lane, int& changed, F release, int ncols) {
  ncols = min(ncols, max(0, (N - n0 + 31) & ~31));
  if constexpr (KIND == 1) {
    tc_or_bits(trow, epi_tile, lane, ncols);
    release();
    if (ep.out_type == kOrU8) tc_or_store<uint8_t>(ep, M, N, n0, row0, epi_tile, lane, changed, ncols);
    else if (ep.out_type == kOrI32) tc_or_store<int32_t>(ep, M, N, n0, row0, epi_tile, lane, changed, ncols);
    else tc_or_store<float>(ep, M, N, n0, row0, epi_tile, lane, changed, ncols);
  } else {
    // Sums: a 32 x 32 chunk is transposed through shared memory (the stage
    // ring is idle now) and written row by row: lane l handles column l, so
    // every store instruction covers 32 consecutive floats of one row.  The
    // chunk's C values (one column per lane, 32 independent loads) and the
    // warp's 32 row norms are fetched before the TMEM read, so their latency
    // overlaps it instead of being paid row by row.
    uint32_t* tile = epi_tile;
    const bool msq = ep.op == SIMD2_MINUS_SQUARE;
    const float na_lane = (msq && row0 + lane < M) ? ep.norm_a[row0 + lane] : 0.f;
    const int rows_here = min(32, M - row0);
#pragma unroll 1
    for (int c0 = 0; c0 < ncols; c0 += 32) {
      const int col = n0 + c0 + lane;
      const bool col_ok = col < N;
      float cv[32];
      if (ep.do_epilogue) {
        const float* Cc = static_cast<const float*>(ep.C) + col;
#pragma unroll
        for (int rr = 0; rr < 32; rr++)
          cv[rr] = (col_ok && rr < rows_here) ? Cc[(long long)(row0 + rr) * ep.ldc] : 0.f;
      }
      const float nb = (msq && col_ok) ? ep.norm_b[col] : 0.f;
      uint32_t r[32];
      tmem_ld32(trow + c0, r);  // all lanes take part (sync.aligned)
#pragma unroll
      for (int j = 0; j < 32; j++) tile[lane * 33 + j] = r[j];
      __syncwarp();
      if (msq) {
        // distances in place; rows inside the cancellation band are
        // recomputed exactly in a separate, rarely taken loop (one copy of
        // the recompute code)
        uint32_t band = 0;
#pragma unroll
        for (int rr = 0; rr < 32; rr++) {
          const float nsum = __shfl_sync(0xffffffffu, na_lane, rr) + nb;
          const float v = __fmaf_rn(-2.0f, __uint_as_float(tile[rr * 33 + lane]), nsum);
          tile[rr * 33 + lane] = __float_as_uint(v);
          band |= (v < ep.band * nsum && rr < rows_here && col_ok ? 1u : 0u) << rr;
        }
        while (band) {
          const int rr = __ffs(band) - 1;
          band &= band - 1;
          using T = typename std::conditional<KIND == 2, __half, float>::type;
          tile[rr * 33 + lane] = __float_as_uint(
              exact_minus_square(static_cast<const T*>(ep.A32) + (long long)(row0 + rr) * ep.lda32,
                                 static_cast<const T*>(ep.B32), ep.ldb32, col, ep.K, ep.b_rows));
        }
      }
      if (col_ok) {
        float* Dc = static_cast<float*>(ep.D) + col;
#pragma unroll
        for (int rr = 0; rr < 32; rr++) {
          if (rr < rows_here) {
            float v = __uint_as_float(tile[rr * 33 + lane]);
            if (ep.do_epilogue) v = __fadd_rn(v, cv[rr]);
            Dc[(long long)(row0 + rr) * ep.ldd] = v;
          }
        }
      }
      __syncwarp();
    }
    release();
  }
}
// The columns of a tile's epilogue that fall to `half` (0, 1): whole 32s.
__device__ __forceinline__ void tc_epi_columns(int ncols, int half, int& first, int& count) {
  const int h = (ncols / 2 + 31) & ~31;
  first = half ? h : 0;
  count = half ? ncols - h : h;
}

// Ring of the single-SM kernel: a stage holds A and bn columns of B, and as many
// stages as fit are used, at most kTcMaxStages: a narrow tile's k-tiles pass
// faster, so more of them have to be on their way.
constexpr int kTcMaxStages = 8;
template <int KIND, bool BT>
__host__ __device__ constexpr int tc_stage_of(int bn) {
  return BT ? TcCfg<KIND>::kNumA * tc_a_tile<KIND>() + TcCfg<KIND>::kNumB * (bn >> 6) * tc_b_group<KIND>()
            : tc_stage_bytes<KIND>();
}
template <int KIND, bool BT>
__host__ __device__ constexpr int tc_stages_of(int bn) {
  const int fit = TcCfg<KIND>::kStages * tc_stage_bytes<KIND>() / tc_stage_of<KIND, BT>(bn);
  return fit < kTcMaxStages ? fit : kTcMaxStages;
}

// SPLIT: the CTAs of a cluster share one tile, each a range of its k-tiles.  A warp
// parks its 32 rows x ncols columns of the accumulator in its CTA's shared memory
// (the ring, idle by then) ...
__device__ __forceinline__ int tc_part_pitch(int bn) { return bn + 4; }
__device__ __forceinline__ void tc_park(uint32_t trow, float* row, int ncols) {
#pragma unroll 1
  for (int c0 = 0; c0 < ncols; c0 += 32) {
    uint32_t r[32];
    tmem_ld32(trow + c0, r);
#pragma unroll
    for (int j = 0; j < 32; j += 4) *reinterpret_cast<uint4*>(row + c0 + j) = make_uint4(r[j], r[j + 1], r[j + 2], r[j + 3]);
  }
}

// ... and every CTA adds up the parts of 128 / S of the rows, in the order of the
// ranks, and writes them out.  A thread has the parts of 8 / S quads of columns on
// their way at once: one at a time, the fold of a tile took 10 to 25 us of latency.
template <int KIND, int S>
__device__ __forceinline__ void tc_fold(const TcEpilogue& ep, int M, int N, int m0, int n0, const float* part, int bn,
                                        int rank, int thread) {
  constexpr int U = 8 / S, T = kTcEpiWarps * 32;
  constexpr int per = kTcBM / S;
  const int first = rank * per, quads = bn >> 2;
  const int end = min(per, M - m0 - first) * quads;
  const bool msq = ep.op == SIMD2_MINUS_SQUARE;
  const float* C = ep.do_epilogue ? static_cast<const float*>(ep.C) : nullptr;
  float* D = static_cast<float*>(ep.D);
  const bool vec = (reinterpret_cast<uintptr_t>(D) & 15) == 0 && (ep.ldd & 3) == 0 &&
                   (!C || ((reinterpret_cast<uintptr_t>(C) & 15) == 0 && (ep.ldc & 3) == 0));
  for (int e0 = thread; e0 < end; e0 += U * T) {
    float4 p[U][S];
    float4 c[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int e = e0 + u * T;
      if (e >= end) break;
      const int r = e / quads, j = (e - r * quads) * 4, left = N - n0 - j;
      const uint32_t at = smem_u32(part + (first + r) * tc_part_pitch(bn) + j);
#pragma unroll
      for (int q = 0; q < S; q++) {
        uint32_t remote;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(at), "r"(q));
        asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                     : "=f"(p[u][q].x), "=f"(p[u][q].y), "=f"(p[u][q].z), "=f"(p[u][q].w)
                     : "r"(remote)
                     : "memory");
      }
      if (C) {
        const float* cr = C + (long long)(m0 + first + r) * ep.ldc + n0 + j;
        if (vec && left >= 4) c[u] = *reinterpret_cast<const float4*>(cr);
        else c[u] = make_float4(left > 0 ? cr[0] : 0.f, left > 1 ? cr[1] : 0.f, left > 2 ? cr[2] : 0.f, left > 3 ? cr[3] : 0.f);
      }
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int e = e0 + u * T;
      if (e >= end) break;
      const int r = e / quads, j = (e - r * quads) * 4, left = N - n0 - j;
      const long long row = m0 + first + r;
      float v[4] = {p[u][0].x, p[u][0].y, p[u][0].z, p[u][0].w};
#pragma unroll
      for (int q = 1; q < S; q++) {
        v[0] = __fadd_rn(v[0], p[u][q].x);
        v[1] = __fadd_rn(v[1], p[u][q].y);
        v[2] = __fadd_rn(v[2], p[u][q].z);
        v[3] = __fadd_rn(v[3], p[u][q].w);
      }
      if (msq) {
        const float na = ep.norm_a[row];
        uint32_t band = 0;
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const float nsum = na + (i < left ? ep.norm_b[n0 + j + i] : 0.f);
          v[i] = __fmaf_rn(-2.0f, v[i], nsum);
          band |= (i < left && v[i] < ep.band * nsum ? 1u : 0u) << i;
        }
        while (band) {  // rare: inside the cancellation band
          const int i = __ffs(band) - 1;
          band &= band - 1;
          using A = typename std::conditional<KIND == 2, __half, float>::type;
          const float d =
              exact_minus_square(static_cast<const A*>(ep.A32) + row * ep.lda32, static_cast<const A*>(ep.B32),
                                 ep.ldb32, n0 + j + i, ep.K, ep.b_rows);
          if (i == 0) v[0] = d;
          else if (i == 1) v[1] = d;
          else if (i == 2) v[2] = d;
          else v[3] = d;
        }
      }
      if (C) {
        v[0] = __fadd_rn(v[0], c[u].x);
        v[1] = __fadd_rn(v[1], c[u].y);
        v[2] = __fadd_rn(v[2], c[u].z);
        v[3] = __fadd_rn(v[3], c[u].w);
      }
      float* dr = D + row * ep.ldd + n0 + j;
      if (vec && left >= 4) *reinterpret_cast<float4*>(dr) = make_float4(v[0], v[1], v[2], v[3]);
      else {
#pragma unroll
        for (int i = 0; i < 4; i++)
          if (i < left) dr[i] = v[i];
      }
    }
  }
}

__device__ __forceinline__ void tc_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// bn: columns of a tile (a multiple of 64, at most 256; 224 for or_and).
// SPLIT (the sums): a cluster of 2, 4 or 8 CTAs per tile, one tile each.  A product of
// few tiles leaves most SMs idle and walks its k alone (64 x 64 x 20000: 1 SM, 205 us;
// now 8, 59 us, of which the operands' split takes about 28).  No scratch memory, and the
// parts are added in one order.
template <int KIND, bool BT, bool SPLIT = false>
__global__ void __launch_bounds__(kTcThreads, 1)
    tc_gemm_kernel(const __grid_constant__ CUtensorMap tmA0, const __grid_constant__ CUtensorMap tmA1,
                   const __grid_constant__ CUtensorMap tmB0, const __grid_constant__ CUtensorMap tmB1, int M, int N,
                   int K, TcEpilogue ep, int tiles_m, int tiles_n, int bn) {
  if (ep.gate && *ep.gate == 0) return;
  using Cfg = TcCfg<KIND>;
  const int S = tc_stages_of<KIND, BT>(bn);
  const int stage_bytes = tc_stage_of<KIND, BT>(bn);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint32_t* epi_smem = reinterpret_cast<uint32_t*>(smem + Cfg::kStages * tc_stage_bytes<KIND>());  // 32 x 33 words per epilogue warp
  uint64_t* full = reinterpret_cast<uint64_t*>(epi_smem + kTcEpiWarps * 32 * 33);
  uint64_t* empty = full + kTcMaxStages;
  uint64_t* acc_full = empty + kTcMaxStages;
  uint64_t* acc_empty = acc_full + 2;
  uint64_t* fin = acc_empty + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(fin + 1);

  const int tiles = tiles_m * tiles_n;
  const uint32_t idesc = tc_idesc<KIND>(bn, BT);
  const int all_ktiles = (K + Cfg::kBK - 1) / Cfg::kBK;
  int splits = 1, rank = 0;
  if constexpr (SPLIT) {
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(splits));
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  }
  const int kt0 = (int)((long long)all_ktiles * rank / splits);
  const int ktiles = (int)((long long)all_ktiles * (rank + 1) / splits);  // of this CTA: [kt0, ktiles)
  const int first_tile = SPLIT ? blockIdx.x / splits : blockIdx.x, tile_step = SPLIT ? tiles : gridDim.x;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  // Grouped raster over (tile_m, tile_n): 8 tile rows per group.
  auto tile_origin = [&](int t, int& m0, int& n0) {
    const int group = 8;
    const int per_group = group * tiles_n;
    const int g = t / per_group;
    const int first_m = g * group;
    const int gsize = min(tiles_m - first_m, group);
    const int local = t - g * per_group;
    m0 = (first_m + local % gsize) * kTcBM;
    n0 = (local / gsize) * bn;
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; a++) {
      mbar_init(&acc_full[a], 1);
      mbar_init(&acc_empty[a], kTcEpiWarps);
    }
    mbar_init(fin, 1);
    fence_mbar_init();
  }
  if (warp == 0) {
    // 512 TMEM columns: two FP32 accumulators (and or_and's scales).
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  if constexpr (KIND == 1) {
    if (warp >= 2) tc_fill_scales(tmem + kTcScaleCol + ((uint32_t)((warp & 3) * 32) << 16));
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
  }

  if (warp == 0) {
    if (lane == 0) {
      // ---------------- TMA producer: every k-tile of every tile of this CTA ----------------
      prefetch_tensormap(&tmA0);
      prefetch_tensormap(&tmB0);
      int s = 0;  // ring position
      uint32_t ph = 1;
      bool ok = true;
      for (int t = first_tile; t < tiles && ok; t += tile_step) {
        int m0, n0;
        tile_origin(t, m0, n0);
        for (int kt = kt0; kt < ktiles; kt++) {
          if (!mbar_wait(&empty[s], ph)) {
            report_timeout(101);
            ok = false;
            break;
          }
          uint8_t* st = smem + s * stage_bytes;
          mbar_arrive_expect_tx(&full[s], stage_bytes);
          const int kx = kt * tc_box_x<KIND>();
          tma_load_2d(st, &tmA0, &full[s], kx, m0);
          if constexpr (Cfg::kNumA == 2) tma_load_2d(st + tc_a_tile<KIND>(), &tmA1, &full[s], kx, m0);
          uint8_t* sb = st + Cfg::kNumA * tc_a_tile<KIND>();
          if constexpr (BT) {
            for (int g = 0; g < (bn >> 6); g++) {
              tma_load_2d(sb + g * tc_b_group<KIND>(), &tmB0, &full[s], n0 + 64 * g, kx);
              if constexpr (Cfg::kNumB == 2)
                tma_load_2d(sb + ((bn >> 6) + g) * tc_b_group<KIND>(), &tmB1, &full[s], n0 + 64 * g, kx);
            }
          } else {
            tma_load_2d(sb, &tmB0, &full[s], kx, n0);
            if constexpr (Cfg::kNumB == 2) tma_load_2d(sb + tc_b_tile<KIND>(), &tmB1, &full[s], kx, n0);
          }
          if (++s == S) {
            s = 0;
            ph ^= 1;
          }
        }
      }
    }
    __syncwarp();  // lanes 1..31 wait here, off the issue slots, while lane 0 runs the loop
  } else if (warp == 1) {
    if (lane == 0) {
      // ---------------- MMA issuer: tile lt accumulates into TMEM half lt & 1 ----------------
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      int lt = 0;
      for (int t = first_tile; t < tiles && ok; t += tile_step, lt++) {
        const int acc = lt & 1;
        if (!mbar_wait(&acc_empty[acc], ((lt >> 1) & 1) ^ 1)) {
          report_timeout(104);
          break;
        }
        tc_fence_after();
        const uint32_t d = tmem + acc * tc_bn<KIND>();
        for (int kt = kt0; kt < ktiles; kt++) {
          if (!mbar_wait(&full[s], ph)) {
            report_timeout(102);
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t st = smem_u32(smem + s * stage_bytes);
          const uint32_t a0 = st, a1 = st + tc_a_tile<KIND>();
          const uint32_t b0 = st + Cfg::kNumA * tc_a_tile<KIND>();
          const uint32_t b1 = b0 + (BT ? (bn >> 6) * tc_b_group<KIND>() : tc_b_tile<KIND>());
          constexpr int RB = Cfg::kRowBytes;
#pragma unroll
          for (int ks = 0; ks < Cfg::kBK / Cfg::kKStep; ks++) {
            const uint32_t koff = ks * 32;  // bytes along the swizzled row
            const uint32_t acc0 = (kt > kt0 || ks > 0) ? 1u : 0u;
            auto bdesc = [&](uint32_t b) {
              return BT ? umma_desc_nmajor(b + ks * 2048, tc_b_group<KIND>()) : umma_desc_swizzled(b + koff, RB);
            };
            if constexpr (KIND == 0) {
              // hi*hi, hi*lo, lo*hi
              tc_mma<0>(d, umma_desc_swizzled(a0 + koff, RB), bdesc(b0), acc0, idesc);
              tc_mma<0>(d, umma_desc_swizzled(a0 + koff, RB), bdesc(b1), 1u, idesc);
              tc_mma<0>(d, umma_desc_swizzled(a1 + koff, RB), bdesc(b0), 1u, idesc);
            } else {
              tc_mma<KIND>(d, umma_desc_swizzled(a0 + koff, RB), bdesc(b0), acc0, idesc, tmem + kTcScaleCol);
            }
          }
          tc_commit(&empty[s]);  // stage s is free once these MMAs have read it
          if (++s == S) {
            s = 0;
            ph ^= 1;
          }
        }
        if (ok) tc_commit(&acc_full[acc]);  // accumulator complete
      }
      tc_commit(fin);  // every MMA issued above has completed when fin flips
    }
    __syncwarp();
  } else {
    // ---------------- epilogue warps 2..9: warp w reads TMEM lanes 32 (w % 4) .. ----------------
    int cfirst, ccount;
    tc_epi_columns(bn, (warp - 2) >> 2, cfirst, ccount);
    const int quad = warp & 3;
    uint32_t* epi_tile = epi_smem + (warp - 2) * (32 * 33);
    bool ok = true;
    int lt = 0;
    for (int t = first_tile; t < tiles; t += tile_step, lt++) {
      const int acc = lt & 1;
      if (ok && !mbar_wait(&acc_full[acc], (lt >> 1) & 1)) {
        report_timeout(103);
        ok = false;
      }
      ok = __all_sync(0xffffffffu, ok);  // tcgen05.ld below is warp-collective
      if (!ok) break;
      tc_fence_after();
      int m0, n0;
      tile_origin(t, m0, n0);
      const uint32_t trow = tmem + acc * tc_bn<KIND>() + cfirst + ((uint32_t)(quad * 32) << 16);
      if constexpr (SPLIT) {
        tc_park(trow, reinterpret_cast<float*>(smem) + (quad * 32 + lane) * tc_part_pitch(bn) + cfirst, ccount);
        break;
      }
      const int row0 = m0 + quad * 32;
      int changed = 0;
      // the accumulator half is read out: the MMA warp may reuse it
      auto release = [&] {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&acc_empty[acc]);
      };
      tc_tile_epilogue<KIND>(ep, M, N, n0 + cfirst, row0, trow, epi_tile, lane, changed, release, ccount);
      if (ep.changed && KIND == 1) {
        if (__any_sync(0xffffffffu, changed) && lane == 0) atomicOr(ep.changed, 1);
      }
    }
  }

  if constexpr (SPLIT) {
    static_assert(kTcBM * (kTcBN + 4) * 4 <= Cfg::kStages * tc_stage_bytes<KIND>(), "parts fit the ring");
    int m0, n0;
    tile_origin(first_tile, m0, n0);
    tc_cluster_sync();  // every part is in place
    if (warp >= 2) {
      const float* part = reinterpret_cast<const float*>(smem);
      const int thread = threadIdx.x - 64;
      if (splits == 2) tc_fold<KIND, 2>(ep, M, N, m0, n0, part, bn, rank, thread);
      else if (splits == 4) tc_fold<KIND, 4>(ep, M, N, m0, n0, part, bn, rank, thread);
      else tc_fold<KIND, 8>(ep, M, N, m0, n0, part, bn, rank, thread);
    }
    tc_cluster_sync();  // peers stay until every CTA has read their parts
  }

  // every MMA has completed before TMEM is released
  if (warp == 0) {
    if (!mbar_wait(fin, 0)) report_timeout(105);
    tc_fence_after();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}

}  // namespace simd2
