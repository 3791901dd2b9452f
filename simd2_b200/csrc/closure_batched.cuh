// closure_batched.cuh -- many independent closures in one persistent launch.
//
// Each graph g (n_g vertices) is closed by repeated squaring X <- X (+) X(x)X
// until unchanged, as in the reference's closure apps
// (apps/apsp/cuASR/apsp_cuASR.cu:37-54, convergence kernel/converge.cuh:6-69).
//
// Work is handed out by 128 x 128 tiles.  A graph of more than one tile is
// shared: CTAs claim the open step's tiles by a ticket, and the CTA that
// finishes the step's last tile decides (change flag, step limit) and opens the
// next step's tiles.  Graphs of one tile are taken from a counter and closed by
// one CTA each.  A CTA only waits while every open tile is held by a running
// CTA, so the waits end; they are bounded all the same.  With one CTA per graph,
// the largest graph's chain of steps set the time of a batch whose other graphs
// left SMs idle long before: 512 graphs of up to 1024 vertices, min_plus,
// 54-59 ms, now 10.3 ms (on codes); 4096 such graphs, 148 ms, now 87 ms.  The
// arithmetic is 7 of the 10.3 ms; the rest is about 9 us a tile for the
// epilogue, the fences and the claim, against 18 us of arithmetic for a tile of
// a 256-vertex graph and 73 us of a 1024-vertex one.
//
// Operands are the 16-bit codes of srgemm_sk.cuh where the semiring has them
// and every entry of the graph has one, else FP32 (k-pair interleaved B, see
// srgemm_simt.cuh).  A sum that outgrows the codes sends its graph back to the
// start on FP32: the caller's matrix is only written at the end.  Tiles are
// staged by TMA through per-graph tensor maps kept in device memory into the
// ring of srgemm_sk_kernel; the epilogue of a step writes both layouts of
// X_{t+1}, and a generic-to-async proxy fence and a release order those writes
// before the next step's TMA reads on any SM.
#pragma once
#include "srgemm_sk.cuh"

namespace simd2 {

struct BatchGraph {
  int n;        // vertices
  int Mp;       // rows padded to a multiple of 128
  int Kp, Kh;   // k extent padded to a multiple of 32 (FP32) / 64 (codes)
  int Np;       // columns padded to a multiple of 128 (B role)
  float* X[2];     // [Mp][Kp], ping-pong
  float* P[2];     // [Kp/2][2*Np] interleaved, ping-pong
  // Codes, ping-pong, in the memory of X and P (null: the semiring has none): a
  // graph is on codes or, after kPrep32 has written X and P anew, on FP32.
  uint16_t* Xc[2];  // [Mp][Kh]
  uint32_t* Pc[2];  // [Kh/2][Np] words (code of X[2p][j], code of X[2p+1][j])
  float* user;  // caller's matrix (result is copied back here)
  long long ldu;
  int iters;    // out: steps run (including the final unchanged one)
  int changed;  // out: 1 if the last step still changed something
  int coded;    // out: 1 when the result lies in Xc
};

__device__ __forceinline__ void fence_proxy_async_global() {
  asm volatile("fence.proxy.async.global;" ::: "memory");
}

// Tensor maps of one graph, in device memory, encoded once per plan: A role
// ([Mp][Kp] floats / [Mp][Kh] codes, 128-row boxes of 128 bytes, swizzled) and
// B role (16 x 256 floats / 32 x 128 words).
struct BatchMaps {
  CUtensorMap a[2];
  CUtensorMap b[2];
  CUtensorMap ac[2];
  CUtensorMap bc[2];
};

// What an open step of a graph does.
enum BatchKind { kStep16 = 1, kPrep32 = 2, kStep32 = 3 };

// Cleared before every run.
struct BatchState {
  int bad;       // an entry has no code (set by the prep kernel)
  int done;      // tiles of the open step finished
  int flags[2];  // the open step changed something; a result of it has no code
};
struct BatchCtl {
  unsigned next;             // slots claimed (8-byte aligned pair with `open`)
  unsigned open;             // slots opened
  unsigned lost;             // set when steps no longer fit the slots: 2^31 - the first slot never written
  int alone_next;            // graphs taken to be closed alone
  int closed;                // shared graphs closed (counts up to nbig)
  int failed;                // a bounded wait ran out somewhere
};

struct BatchArgs {
  BatchGraph* graphs;
  const BatchMaps* maps;
  // nbig graphs shared by tiles, then nalone that one CTA closes alone, then the
  // empty ones, which have no tile and are done once the prep kernel has run
  const int* order;
  int nbig, nalone, count;
  BatchState* state;
  BatchCtl* ctl;
  // One slot per tile of every opened step, in the order of opening: the first
  // nfirst are the shared graphs' first steps (written with the plan), the rest
  // start at 0 and are written as steps open.
  unsigned long long* slots;
  unsigned nfirst, cap;
  int max_iter, conv_mode;
  int use_codes;      // the plan has coded buffers
};

__device__ __forceinline__ int ld_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned long long ld_acquire64(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release64(unsigned long long* p, unsigned long long v) {
  asm volatile("st.release.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// A slot: 1 | kind (2 bits, 0: the graph has not begun) | step (10) | tile (20) | graph (20).
__host__ __device__ inline unsigned long long batch_slot(int kind, int step, int tile, int graph) {
  return 1ull << 52 | (unsigned long long)kind << 50 | (unsigned long long)step << 40 |
         (unsigned long long)tile << 20 | (unsigned long long)graph;
}
constexpr int kBatchSlotMax = 1 << 20;   // graphs and tiles per graph that a slot can name
constexpr int kBatchSlotSteps = 40;      // steps of a graph that are opened for sharing

// A claimed piece of work: one tile of a graph's open step.
struct BatchTask {
  int graph;  // -1: nothing left
  int n, tile;
  int kind, step;
  int pre;    // loads already issued for it
  int alone;  // this CTA runs every tile and step of the graph
  int shared; // the graph is one of the nbig
};

__device__ __forceinline__ int batch_tiles_1d(int n) { return (n + 127) / 128; }

// Claims the next slot if one looks open; one thread.  Others may claim in
// between: a slot that is not open yet is kept and waited for (its step is about
// to open; a compare-and-swap that cannot overshoot let one of 148 crowding CTAs
// through per round trip).
__device__ __forceinline__ bool batch_claim(const BatchArgs& a, unsigned& t) {
  const unsigned long long w = *(volatile unsigned long long*)&a.ctl->next;
  if ((unsigned)w >= (unsigned)(w >> 32)) return false;
  t = atomicAdd(&a.ctl->next, 1u);
  return true;
}

// What a graph begins with: without codes it was prepared in FP32 before the launch.
__device__ __forceinline__ int batch_first_kind(const BatchArgs& a, int graph) {
  return !a.use_codes ? kStep32 : __ldcg(&a.state[graph].bad) ? kPrep32 : kStep16;
}

// The task of claimed slot t, if it is written; one thread.
__device__ __forceinline__ bool batch_task_of(const BatchArgs& a, unsigned t, BatchTask& k) {
  if (t >= a.cap) return false;
  const unsigned long long v = ld_acquire64(&a.slots[t]);
  if (v == 0) return false;
  k.graph = (int)(v & (kBatchSlotMax - 1));
  k.tile = (int)(v >> 20 & (kBatchSlotMax - 1));
  k.step = (int)(v >> 40 & 1023);
  k.kind = (int)(v >> 50 & 3);
  if (k.kind == 0) k.kind = batch_first_kind(a, k.graph);
  k.n = __ldg(&a.graphs[k.graph].n);
  k.pre = 0;
  k.alone = 0;
  k.shared = 1;
  return true;
}

// A slot claimed whose task is not known yet.
constexpr unsigned kNoSlot = 0xffffffffu;

// The next task, waiting for one while others are still at work; one thread.
// `slot`: a slot already claimed, or kNoSlot.
__device__ __forceinline__ void batch_pop(const BatchArgs& a, unsigned& slot, BatchTask& t) {
  uint64_t t0 = 0;
  t.alone = 0;
  while (true) {
    if (*(volatile int*)&a.ctl->failed) break;
    if (slot == kNoSlot && !batch_claim(a, slot)) slot = kNoSlot;
    if (slot != kNoSlot) {
      if (batch_task_of(a, slot, t)) {
        slot = kNoSlot;
        return;
      }
      const unsigned lost = *(volatile unsigned*)&a.ctl->lost;
      if (slot >= a.cap || (lost && slot >= 0x80000000u - lost)) slot = kNoSlot;  // will never be written
    }
    if (slot == kNoSlot && *(volatile int*)&a.ctl->alone_next < a.nalone) {
      const int q = atomicAdd(&a.ctl->alone_next, 1);
      if (q < a.nalone) {
        t.graph = a.order[a.nbig + q];
        t.n = a.graphs[t.graph].n;
        t.tile = 0;
        t.kind = batch_first_kind(a, t.graph);
        t.step = 0;
        t.pre = 0;
        t.alone = 1;
        t.shared = 0;
        return;
      }
    }
    if (ld_acquire(&a.ctl->closed) == a.nbig) break;
    const uint64_t now = globaltimer_ns();
    if (t0 == 0) t0 = now;
    else if (now - t0 > kWaitLimitNs) {
      // without a slot it may leave to the others; a claimed one has to come
      if (slot != kNoSlot) {
        report_timeout(41);
        atomicExch(&a.ctl->failed, 1);
      }
      break;
    }
    __nanosleep(64);
  }
  t.graph = -1;
}

// Opens the next step's tiles for claiming: the first slot, or cap when they no
// longer fit (and from then on none do); one thread.
__device__ __forceinline__ unsigned batch_open(const BatchArgs& a, int tiles, int step) {
  if (step >= 1023) return a.cap;
  const unsigned first = atomicAdd(&a.ctl->open, (unsigned)tiles);
  if (first + (unsigned)tiles <= a.cap) return first;
  atomicMax(&a.ctl->lost, 0x80000000u - first);
  return a.cap;
}

// CTA-wide context of the batched kernel.
struct BatchCta {
  uint8_t* smem;
  uint64_t *full, *empty;
  volatile int* failed;
  uint32_t base;  // loads issued for earlier tiles (ring position)
};

// Issues load i of tile (m0, n0): one lane.
template <bool I16>
__device__ __forceinline__ void batch_issue(const BatchCta& x, uint32_t j, const BatchMaps* mp, int cur, int i, int m0,
                                            int n0) {
  using Cfg = SkCfg<128>;
  constexpr int S = Cfg::kStages;
  constexpr int BK = I16 ? kSkBK16 : kBK;
  const int s = j % S;
  if (!sk_wait(&x.empty[s], ((j / S) & 1) ^ 1, x.failed, 42)) return;
  uint8_t* sa = x.smem + s * Cfg::kStage;
  mbar_arrive_expect_tx(&x.full[s], Cfg::kStage);
  tma_load_2d(sa, I16 ? &mp->ac[cur] : &mp->a[cur], &x.full[s], i * BK, m0);
  tma_load_2d(sa + Cfg::kTileBytes, I16 ? &mp->bc[cur] : &mp->b[cur], &x.full[s], I16 ? n0 : 2 * n0, i * (BK / 2));
}

// One FP32 k-tile of the first `groups` of a tile's eight 16-row groups.
template <int OP>
__device__ __forceinline__ void batch_rows32(int groups, float (&acc)[8][4], const uint8_t* As, const uint8_t* Bs,
                                             int ty, int tx, int cbase, int nq) {
  switch (groups) {
    case 1: sk_ktile32<OP, 128, false, 1>(acc, As, Bs, ty, tx, cbase, 0, nq); break;
    case 2: sk_ktile32<OP, 128, false, 2>(acc, As, Bs, ty, tx, cbase, 0, nq); break;
    case 3: sk_ktile32<OP, 128, false, 3>(acc, As, Bs, ty, tx, cbase, 0, nq); break;
    case 4: sk_ktile32<OP, 128, false, 4>(acc, As, Bs, ty, tx, cbase, 0, nq); break;
    case 5: sk_ktile32<OP, 128, false, 5>(acc, As, Bs, ty, tx, cbase, 0, nq); break;
    case 6: sk_ktile32<OP, 128, false, 6>(acc, As, Bs, ty, tx, cbase, 0, nq); break;
    case 7: sk_ktile32<OP, 128, false, 7>(acc, As, Bs, ty, tx, cbase, 0, nq); break;
    default: sk_ktile32<OP, 128, false>(acc, As, Bs, ty, tx, cbase, 0, nq); break;
  }
}

// One tile of step `step`: X[nxt] (+)= on both layouts.  `pre` loads are already
// on their way; before_last() runs on every thread before the last k-tile,
// before_epilogue() after it.
template <int OP, bool I16, typename F1, typename F2>
__device__ __forceinline__ void batch_tile(const BatchArgs& a, BatchCta& x, const BatchGraph& G, const BatchMaps* mp,
                                           int n, int step, int tile, int pre, int& changed, bool& over,
                                           F1 before_last, F2 before_epilogue) {
  using Cfg = SkCfg<128>;
  constexpr int S = Cfg::kStages;
  constexpr int BK = I16 ? kSkBK16 : kBK;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tx = lane & 15;
  const int ty = (warp & 7) * 2 + (lane >> 4);
  const int cbase = (warp >> 3) * 64;
  const int cur = step & 1, nxt = cur ^ 1;
  const int tm = batch_tiles_1d(n);
  const int m0 = (tile % tm) * 128, n0 = (tile / tm) * 128;
  const int units = (n + BK - 1) / BK;
  if (threadIdx.x == 0)
    for (int i = pre; i < min(S, units); i++) batch_issue<I16>(x, x.base + i, mp, cur, i, m0, n0);
  using AccT = typename std::conditional<I16, uint32_t, float>::type;
  AccT acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; i++)
#pragma unroll
    for (int c = 0; c < 4; c++) {
      if constexpr (I16) acc[i][c] = Code16<OP>::kIdent;
      else acc[i][c] = Mac<OP>::identity();
    }
  // What lies past the graph is not computed: 16-row groups (on codes by halves of
  // the register tile), and the warps of the upper column half.
  const int groups = min(8, (n - m0 + 15) >> 4);
  const int rows = groups <= 2 ? 2 : groups <= 4 ? 4 : 8;
  const bool idle = n0 + cbase >= n;
  for (int i = 0; i < units; i++) {
    const uint32_t j = x.base + i;
    const int s = j % S;
    if (i == units - 1) before_last();
    if (lane == 0 && (i & (kSimtWarps - 1)) == warp && i >= Cfg::kLag && i - Cfg::kLag + S < units)
      batch_issue<I16>(x, j - Cfg::kLag + S, mp, cur, i - Cfg::kLag + S, m0, n0);
    sk_wait(&x.full[s], (j / S) & 1, x.failed, 43);
    const uint8_t* As = x.smem + s * Cfg::kStage;
    const uint8_t* Bs = As + Cfg::kTileBytes;
    const int nq = (n - i * BK + BK / 8 - 1) / (BK / 8);
    if (!idle) {
      if constexpr (I16) {
        if (rows == 8 && nq >= 8) sk_ktile16<OP, 128, true>(acc, As, Bs, ty, tx, cbase, 0, 8);
        else if (rows == 8) sk_ktile16<OP, 128, false>(acc, As, Bs, ty, tx, cbase, 0, nq);
        else if (rows == 4) sk_ktile16<OP, 128, false, 4>(acc, As, Bs, ty, tx, cbase, 0, min(nq, 8));
        else sk_ktile16<OP, 128, false, 2>(acc, As, Bs, ty, tx, cbase, 0, min(nq, 8));
      } else {
        if (groups == 8 && nq >= 8) sk_ktile32<OP, 128, true>(acc, As, Bs, ty, tx, cbase, 0, 8);
        else batch_rows32<OP>(groups, acc, As, Bs, ty, tx, cbase, min(nq, 8));
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&x.empty[s]);
  }
  x.base += units;
  before_epilogue();
  const int conv = a.conv_mode;
  if constexpr (I16) {
    // In the code domain, two columns a word.  Lanes l and l + 16 hold rows 2p
    // and 2p + 1 of the same 4 columns: each stores its row's 8 bytes of X, the
    // lower one the pair's 16 bytes of P.
    const int col = n0 + cbase + 4 * tx;
    const uint16_t* X = G.Xc[cur];
    uint16_t* Xn = G.Xc[nxt];
    uint32_t* Pn = G.Pc[nxt];
    const int Kh = G.Kh, Np = G.Np;
    const bool colin = col < n;
    // columns past the graph keep the padding
    const uint32_t keep0 = col + 1 < n ? 0xffffffffu : colin ? 0xffffu : 0u;
    const uint32_t keep1 = col + 3 < n ? 0xffffffffu : col + 2 < n ? 0xffffu : 0u;
    constexpr uint32_t kPad2 = Code16<OP>::kPad * 0x00010001u;
    uint2 old[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const int row = m0 + ty + 16 * i;
      old[i] = row < n && colin ? __ldcg(reinterpret_cast<const uint2*>(X + (long long)row * Kh + col))
                                : make_uint2(kPad2, kPad2);
    }
    uint32_t bad = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const int row = m0 + ty + 16 * i;
      uint32_t c0 = kPad2, c1 = kPad2;
      if (row < n && colin) {
        uint32_t b0 = 0, b1 = 0;
        c0 = Code16<OP>::finish(Code16<OP>::pair(acc[i][0], acc[i][1]), old[i].x, b0);
        c1 = Code16<OP>::finish(Code16<OP>::pair(acc[i][2], acc[i][3]), old[i].y, b1);
        bad |= (b0 & keep0) | (b1 & keep1);
        c0 = (c0 & keep0) | (kPad2 & ~keep0);
        c1 = (c1 & keep1) | (kPad2 & ~keep1);
        if (conv == SIMD2_CONV_TOL && (OP == SIMD2_MAX_MIN || OP == SIMD2_MIN_MAX)) {
          // fractions may move by less than the tolerance (integers cannot)
#pragma unroll
          for (int e = 0; e < 4; e++) {
            const uint32_t o = (e < 2 ? old[i].x : old[i].y) >> (16 * (e & 1)) & 0xffffu;
            const uint32_t v = (e < 2 ? c0 : c1) >> (16 * (e & 1)) & 0xffffu;
            if (conv_changed(conv, Code16<OP>::entry(o), Code16<OP>::entry(v))) changed = 1;
          }
        } else {
          changed |= (c0 != old[i].x) | (c1 != old[i].y);
        }
        *reinterpret_cast<uint2*>(Xn + (long long)row * Kh + col) = make_uint2(c0, c1);
      }
      const uint32_t d0 = __shfl_down_sync(0xffffffffu, c0, 16), d1 = __shfl_down_sync(0xffffffffu, c1, 16);
      if (lane < 16 && row < n && colin)
        *reinterpret_cast<uint4*>(Pn + (long long)(row >> 1) * Np + col) =
            make_uint4(__byte_perm(c0, d0, 0x5410), __byte_perm(c0, d0, 0x7632), __byte_perm(c1, d1, 0x5410),
                       __byte_perm(c1, d1, 0x7632));
    }
    over |= bad != 0;
  } else {
    // Columns 32c + 2tx + e: lane l of the pair (l, l + 16) stores the 16 bytes
    // of P for c = 0, lane l + 16 those for c = 1.
    auto result = [&](float v, float old_v) -> float {
      v = Mac<OP>::add(v, old_v);
      if (conv == SIMD2_CONV_APLP && v > -1.0f && v < 1.0f) v = -3.402823466e+38f;
      if (conv_changed(conv, old_v, v)) changed = 1;
      return v;
    };
    const float* X = G.X[cur];
    float* Xn = G.X[nxt];
    float* Pn = G.P[nxt];
    const float nanv = __int_as_float(0x7fc00000);
    const bool upper = lane >= 16;
    float2 old[8][2];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
      for (int c = 0; c < 2; c++) {
        const int row = m0 + ty + 16 * i, col = n0 + cbase + 32 * c + 2 * tx;
        old[i][c] = row < n && col < n ? __ldcg(reinterpret_cast<const float2*>(X + (long long)row * G.Kp + col))
                                       : make_float2(0.f, 0.f);
      }
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const int row = m0 + ty + 16 * i;
      float2 o[2];
#pragma unroll
      for (int c = 0; c < 2; c++) {
        const int col = n0 + cbase + 32 * c + 2 * tx;
        o[c] = make_float2(nanv, nanv);
        if (row < n && col < n) {
          o[c].x = result(acc[i][2 * c], old[i][c].x);
          if (col + 1 < n) o[c].y = result(acc[i][2 * c + 1], old[i][c].y);
          *reinterpret_cast<float2*>(Xn + (long long)row * G.Kp + col) = o[c];
        }
      }
      const float2 give = upper ? o[0] : o[1], keep = upper ? o[1] : o[0];
      const float gx = __shfl_xor_sync(0xffffffffu, give.x, 16), gy = __shfl_xor_sync(0xffffffffu, give.y, 16);
      const int erow = row & ~1, col = n0 + cbase + (upper ? 32 : 0) + 2 * tx;
      if (erow < n && col < n)
        *reinterpret_cast<float4*>(Pn + (long long)(erow >> 1) * (2LL * G.Np) + 2 * col) =
            upper ? make_float4(gx, keep.x, gy, keep.y) : make_float4(keep.x, gx, keep.y, gy);
    }
  }
}

// 2 rows x 4 columns of a caller's matrix (from row 2 p, column c0), `fill` past it.
__device__ __forceinline__ void batch_load2x4(const BatchGraph& G, int p, int c0, bool vec, float fill,
                                              float (&v)[2][4]) {
#pragma unroll
  for (int r = 0; r < 2; r++) {
    const int row = 2 * p + r;
    const float* src = G.user + (long long)row * G.ldu + c0;
    if (vec && row < G.n && c0 + 4 <= G.n) {
      load4(src, v[r]);
    } else {
#pragma unroll
      for (int e = 0; e < 4; e++) v[r][e] = row < G.n && c0 + e < G.n ? src[e] : fill;
    }
  }
}
__device__ __forceinline__ bool batch_vec4(const BatchGraph& G) {
  return (G.ldu % 4 == 0) && (reinterpret_cast<uintptr_t>(G.user) % 16 == 0);
}

// The FP32 preparation of row pairs [p0, p1) and columns [c0, c1) (multiples of 4,
// below Kp), `thread` of `threads`: X[0] and P[0] from the caller's matrix, NaN in
// the k past it, and those of X[1] and P[1] (steps write the rest).  Rows of A and
// columns of B past the graph only reach outputs that are never stored.
__device__ __forceinline__ void batch_prep32(const BatchGraph& G, int p0, int p1, int c0, int c1, int thread,
                                             int threads) {
  const bool vec = batch_vec4(G);
  const int n = G.n, quads = (c1 - c0) >> 2, items = max(0, p1 - p0) * max(0, quads);
  for (int t = thread; t < items; t += threads) {
    const int p = p0 + t / quads, c = c0 + (t % quads) * 4;
    float v[2][4];
    batch_load2x4(G, p, c, vec, __int_as_float(0x7fc00000), v);
#pragma unroll
    for (int r = 0; r < 2; r++) {
      const long long o = (long long)(2 * p + r) * G.Kp + c;
      const float4 w = make_float4(v[r][0], v[r][1], v[r][2], v[r][3]);
      *reinterpret_cast<float4*>(G.X[0] + o) = w;
      if (c + 4 > n) *reinterpret_cast<float4*>(G.X[1] + o) = w;
    }
    const long long o = (long long)p * (2LL * G.Np) + 2 * c;
    const float4 w0 = make_float4(v[0][0], v[1][0], v[0][1], v[1][1]);
    const float4 w1 = make_float4(v[0][2], v[1][2], v[0][3], v[1][3]);
    *reinterpret_cast<float4*>(G.P[0] + o) = w0;
    *reinterpret_cast<float4*>(G.P[0] + o + 4) = w1;
    if (2 * p + 1 >= n) {
      *reinterpret_cast<float4*>(G.P[1] + o) = w0;
      *reinterpret_cast<float4*>(G.P[1] + o + 4) = w1;
    }
  }
}

// One tile of it, for a graph that leaves its codes.
__device__ __forceinline__ void batch_prep_tile(const BatchGraph& G, int tile) {
  const int tm = batch_tiles_1d(G.n), m0 = (tile % tm) * 128, n0 = (tile / tm) * 128;
  batch_prep32(G, m0 >> 1, min(m0 + 128, G.Kp) >> 1, n0, min(n0 + 128, G.Kp), threadIdx.x, kSimtThreads);
}

template <int OP>
__global__ void __launch_bounds__(kSimtThreads, 1) closure_batched_kernel(BatchArgs a) {
  using Cfg = SkCfg<128>;
  extern __shared__ uint8_t smem_raw[];
  __shared__ int s_failed;
  __shared__ BatchTask s_task, s_next;
  // Graphs this CTA has to go on with alone because the slots are used up (a
  // tile claimed ahead runs first, and may end another such graph: two at most)
  __shared__ BatchTask s_own[2];
  __shared__ int s_nown;
  // The step this CTA opened (graph -1: none).  All threads read it after an
  // iteration's last barrier, so it is written only past the next one's first.
  __shared__ BatchTask s_opened;
  __shared__ unsigned s_first;    // its first slot
  __shared__ int s_flags[2];      // BatchState::flags of the graph this CTA runs alone
  BatchCta x;
  x.smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  x.full = reinterpret_cast<uint64_t*>(x.smem + Cfg::kStages * Cfg::kStage + Cfg::kRedBytes);
  x.empty = x.full + Cfg::kStages;
  x.failed = &s_failed;
  x.base = 0;
  unsigned slot = kNoSlot;  // thread 0's claimed slot
  if (threadIdx.x == 0) {
    for (int s = 0; s < Cfg::kStages; s++) {
      mbar_init(&x.full[s], 1);
      mbar_init(&x.empty[s], kSimtWarps);
    }
    fence_mbar_init();
    s_failed = 0;
    s_next.graph = -1;
    s_task.alone = 0;
    s_opened.graph = -1;
    s_nown = 0;
    s_flags[0] = s_flags[1] = 0;
  }
  __syncthreads();
  while (true) {
    if (threadIdx.x == 0) {
      if (s_next.graph >= 0) s_task = s_next;
      else if (s_task.alone) ;  // the next step's first tile, left there by the last tile
      else if (s_nown > 0) s_task = s_own[--s_nown];
      else batch_pop(a, slot, s_task);
      s_next.graph = -1;
    }
    __syncthreads();
    const BatchTask task = s_task;
    if (task.graph < 0) break;
    // every thread has passed the barrier above, so none still publishes the step before
    if (threadIdx.x == 0) s_opened.graph = -1;
    fence_proxy_async_global();  // the acquire that claimed the task, before its TMA reads
    BatchGraph& G = a.graphs[task.graph];
    const BatchMaps* mp = a.maps + task.graph;
    BatchState* st = &a.state[task.graph];
    int changed = 0;
    bool over = false;
    // Thread 0 claims the next tile before the last k-tile and starts its first
    // loads after it, so that they run under the epilogue.  (A list of steps
    // with a counter each, on which the CTAs crowded, held the CTA's barrier up
    // for 6 us a tile with 64 tiles a step and 22 us with 4.)
    auto claim_early = [&]() {
      if (threadIdx.x == 0 && !task.alone && s_nown == 0 && slot == kNoSlot && !batch_claim(a, slot)) slot = kNoSlot;
    };
    auto look_ahead = [&]() {
      if (threadIdx.x != 0) return;
      BatchTask t;
      if (task.alone) {  // its own next tile of the step
        t = task;
        t.pre = 0;
        if (++t.tile == batch_tiles_1d(t.n) * batch_tiles_1d(t.n)) return;
      } else {
        if (slot == kNoSlot || !batch_task_of(a, slot, t)) return;
        slot = kNoSlot;
      }
      if (t.kind != kPrep32) {
        fence_proxy_async_global();
        const int tm = batch_tiles_1d(t.n), m0 = (t.tile % tm) * 128, n0 = (t.tile / tm) * 128;
        const int bk = t.kind == kStep16 ? kSkBK16 : kBK;
        const int want = min(Cfg::kStages, (t.n + bk - 1) / bk);
        for (; t.pre < want; t.pre++) {
          if (t.kind == kStep16) batch_issue<true>(x, x.base + t.pre, a.maps + t.graph, t.step & 1, t.pre, m0, n0);
          else batch_issue<false>(x, x.base + t.pre, a.maps + t.graph, t.step & 1, t.pre, m0, n0);
        }
      }
      s_next = t;
    };
    if (task.kind == kPrep32) {
      batch_prep_tile(G, task.tile);
    } else {
      bool ran = false;
      if constexpr (Code16<OP>::kHas) {
        if (task.kind == kStep16) {
          batch_tile<OP, true>(a, x, G, mp, task.n, task.step, task.tile, task.pre, changed, over, claim_early,
                               look_ahead);
          ran = true;
        }
      }
      if (!ran)
        batch_tile<OP, false>(a, x, G, mp, task.n, task.step, task.tile, task.pre, changed, over, claim_early,
                              look_ahead);
    }
    // The outcome of a graph that this CTA runs alone stays in shared memory, and its
    // writes only have to be ordered for this CTA (the flags in global memory and the
    // wider fence cost a step of a small graph about 3 us).
    int* flags = task.alone ? s_flags : st->flags;
    if (__any_sync(0xffffffffu, changed) && (threadIdx.x & 31) == 0) atomicOr(&flags[0], 1);
    if (__any_sync(0xffffffffu, over) && (threadIdx.x & 31) == 0) atomicOr(&flags[1], 1);
    fence_proxy_async_global();  // this tile's generic writes, before any TMA read of them
    if (!task.alone) __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
      const int tiles = batch_tiles_1d(task.n) * batch_tiles_1d(task.n);
      const bool last = task.alone ? task.tile == tiles - 1 : atomicAdd(&st->done, 1) == tiles - 1;
      if (!last) {
        if (task.alone && s_next.graph < 0) s_task.tile++;  // a preparation tile
      } else {
        // the step's last tile: decide and open what follows
        if (!task.alone) __threadfence();
        const int ch = *(volatile int*)&flags[0], ov = *(volatile int*)&flags[1];
        int kind = task.kind, step = task.step + 1;
        bool closed = false;
        if (kind == kPrep32) {
          kind = kStep32;
          step = 0;
        } else if (ov) {
          kind = kPrep32;
          step = 0;
        } else {
          closed = !ch || step >= a.max_iter;
        }
        flags[0] = flags[1] = 0;
        if (!task.alone) st->done = 0;
        if (closed) {
          G.iters = step;
          G.changed = ch;
          G.coded = kind == kStep16;
          s_task.alone = 0;
          __threadfence();
          if (task.shared) atomicAdd(&a.ctl->closed, 1);
        } else {
          BatchTask t;
          t.graph = task.graph;
          t.n = task.n;
          t.tile = 0;
          t.kind = kind;
          t.step = step;
          t.pre = 0;
          t.alone = 1;
          t.shared = task.shared;
          if (task.alone) {
            s_task = t;
          } else {
            s_first = batch_open(a, tiles, step);
            if (s_first < a.cap) s_opened = t;
            else s_own[s_nown++] = t;
          }
        }
      }
      if (*x.failed) atomicExch(&a.ctl->failed, 1);
    }
    __syncthreads();
    if (s_opened.graph >= 0) {
      const int tiles = batch_tiles_1d(s_opened.n) * batch_tiles_1d(s_opened.n);
      for (int i = threadIdx.x; i < tiles; i += kSimtThreads)
        st_release64(&a.slots[s_first + i], batch_slot(s_opened.kind, s_opened.step, i, s_opened.graph));
    }
    if (*x.failed) break;
  }
  if (s_failed && threadIdx.x == 0)  // copies in flight land before shared memory is released
    for (int s = 0; s < Cfg::kStages; s++)
      for (int p = 0; p < 2; p++) mbar_wait(&x.full[s], p, 1000000ull);
}

// The coded operands of every graph: X and P codes from the caller's matrix,
// the padding of both buffers (steps write the rest of the second), `bad` where
// an entry has no code; and the results' fields as of an unfinished run.
// A thread takes 2 rows x 4 columns.
template <int OP>
__global__ void __launch_bounds__(256) batched_prep_kernel(BatchArgs a) {
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0)
    a.ctl->open = a.nfirst;  // the first steps are open
  for (int g = blockIdx.y; g < a.count; g += gridDim.y) {
    BatchGraph& G = a.graphs[g];
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      G.iters = G.n == 0;  // an empty graph is done in one unchanged step
      G.changed = G.n != 0;
      G.coded = -1;
    }
    if (!a.use_codes) {
      batch_prep32(G, 0, G.Kp >> 1, 0, G.Kp, blockIdx.x * 256 + threadIdx.x, gridDim.x * 256);
      continue;
    }
    if constexpr (Code16<OP>::kHas) {
      const int n = G.n, Kh = G.Kh, Np = G.Np;
      const int quads = Np >> 2;
      const long long total = (long long)(Kh >> 1) * quads;
      const bool vec = batch_vec4(G);
      bool bad = false;
      for (long long t = blockIdx.x * 256LL + threadIdx.x; t < total; t += gridDim.x * 256LL) {
        const int p = (int)(t / quads), c0 = (int)(t - (long long)p * quads) * 4;
        uint32_t c[2][4];
        float v[2][4];
        batch_load2x4(G, p, c0, vec, 0.f, v);
#pragma unroll
        for (int r = 0; r < 2; r++) {
          const int row = 2 * p + r;
#pragma unroll
          for (int e = 0; e < 4; e++)
            c[r][e] = row < n && c0 + e < n ? Code16<OP>::encode(v[r][e], bad) : Code16<OP>::kPad;
          if (c0 < Kh) {
            const uint2 w = make_uint2(c[r][0] | c[r][1] << 16, c[r][2] | c[r][3] << 16);
            *reinterpret_cast<uint2*>(G.Xc[0] + (long long)row * Kh + c0) = w;
            if (c0 + 4 > n || row >= n) *reinterpret_cast<uint2*>(G.Xc[1] + (long long)row * Kh + c0) = w;
          }
        }
        const uint4 w = make_uint4(c[0][0] | c[1][0] << 16, c[0][1] | c[1][1] << 16, c[0][2] | c[1][2] << 16,
                                   c[0][3] | c[1][3] << 16);
        *reinterpret_cast<uint4*>(G.Pc[0] + (long long)p * Np + c0) = w;
        if (c0 + 4 > n || 2 * p + 1 >= n) *reinterpret_cast<uint4*>(G.Pc[1] + (long long)p * Np + c0) = w;
      }
      if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(&a.state[g].bad, 1);
    }
  }
}

// Copies every result X[iters & 1] (or its codes' values) back into the
// caller's matrix; a graph the run did not finish keeps its input.
template <int OP>
__global__ void __launch_bounds__(256) batched_finish_kernel(BatchArgs a) {
  for (int g = blockIdx.y; g < a.count; g += gridDim.y) {
    const BatchGraph& G = a.graphs[g];
    const int n = G.n, b = G.iters & 1;
    if (G.coded < 0) continue;
    const int quads = (n + 3) >> 2;
    const long long total = (long long)n * quads;
    const bool vec = (G.ldu % 4 == 0) && (reinterpret_cast<uintptr_t>(G.user) % 16 == 0);
    for (long long t = blockIdx.x * 256LL + threadIdx.x; t < total; t += gridDim.x * 256LL) {
      const int i = (int)(t / quads), c0 = (int)(t - (long long)i * quads) * 4;
      float v[4];
      if (G.coded) {
        if constexpr (Code16<OP>::kHas) {
          const uint2 w = *reinterpret_cast<const uint2*>(G.Xc[b] + (long long)i * G.Kh + c0);
          v[0] = Code16<OP>::entry(w.x & 0xffffu), v[1] = Code16<OP>::entry(w.x >> 16);
          v[2] = Code16<OP>::entry(w.y & 0xffffu), v[3] = Code16<OP>::entry(w.y >> 16);
        }
      } else {
        const float4 u = *reinterpret_cast<const float4*>(G.X[b] + (long long)i * G.Kp + c0);
        v[0] = u.x, v[1] = u.y, v[2] = u.z, v[3] = u.w;
      }
      float* dst = G.user + (long long)i * G.ldu + c0;
      if (vec && c0 + 4 <= n) {
        *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
      } else {
#pragma unroll
        for (int e = 0; e < 4; e++)
          if (c0 + e < n) dst[e] = v[e];
      }
    }
  }
}

}  // namespace simd2
