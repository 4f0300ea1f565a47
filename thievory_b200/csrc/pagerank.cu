// PageRank, pull (CSC in-edges) and push (CSR out-edges).
//
// Method (fixed by the engine's contract, not the reference's): FP32 ranks,
// damping d, a fixed iteration count, dangling mass spread uniformly:
//     r'(v) = (1-d)/N + d * ( sum_{u->v} r(u)/outdeg(u) + D/N ),
//     D = sum of r(u) over vertices with outdeg(u) = 0,   r0 = 1/N.
// The reference's kernels this replaces are src/pr/pr_kernels.cu:23-160
// (pull: static/demand/filter) with PR32_Update_Values :449-476, and
// :504-681 (push) with PR32_Update_Values_PUSH :846-860; those iterate to a
// 1e-3 tolerance in FP64 without dangling redistribution.
//
// Every iteration streams all edges.  A warp (or a CTA: push on large
// resident graphs) takes one tile, consecutive vertices inside one edge
// block with at most 480 (4,096) edges, reads the tile's adjacency with
// 16-byte vector loads -- full 128-byte lines whether the block is in HBM or
// read zero-copy from pinned host memory -- and gathers (pull) or scatters
// (push) per edge.  Per-vertex sums are FP64; stored ranks and contributions
// are FP32.
// Pull fuses the rank update into the gather: a vertex's sum is complete
// inside its tile, except high-degree vertices cut into parts, whose last
// part (atomic counter) finishes the update.
#include <algorithm>

#include "thv_device.cuh"
#include "thv_internal.h"

namespace thv {

constexpr int kPrThreads = 256;
constexpr int kPrWarps = kPrThreads / 32;
constexpr int kStageEdges = (int)kTileShape[kCtaTiles].edges;

struct PrArgs {
  const PrTile *tiles;
  const uint64_t *blk_base;
  const uint64_t *off;
  const uint32_t *outdeg;  // CSC: explicit; CSR: nullptr (from offsets)
  const float *cur;
  float *nxt;
  float *rank;
  double *sum;
  double *split_acc;
  uint32_t *split_done;
  const uint32_t *split_parts;
  double *dang;
  uint32_t *tile_ctr;
  uint32_t ntiles, nv, it;
  uint32_t wshift;  // packed weighted edges: the id is e >> wshift
  uint32_t last;    // last iteration
  uint32_t draw;    // warp tiles: tiles a warp draws at a time
  uint32_t first;   // warp tiles: warps of a CTA with tiles of a round
  uint32_t fixed;   // warp tiles: tiles handed out by place
  double damping, inv_n;
};

struct PrState {
  uint64_t nv = 0;
  uint32_t iters = 0;
  float *d_c[2] = {nullptr, nullptr};
  float *d_rank = nullptr;
  double *d_sum = nullptr;
  double *d_split_acc = nullptr;
  uint32_t *d_split_done = nullptr;
  double *d_dang = nullptr;
  uint32_t *d_tile_ctr = nullptr;
  uint32_t cap_iters = 0;
  size_t nsplit = 0;
  bool push = false;
  // reference semantics (THV_RUN_PR_REFERENCE): FP64 values
  bool ref = false;
  double *d_val = nullptr, *d_acc = nullptr, *d_delta = nullptr;
  uint8_t *d_act = nullptr;
  unsigned long long *d_cnt = nullptr, *h_cnt = nullptr;  // active vertices, their edges
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
};

__device__ __forceinline__ uint32_t out_degree(const PrArgs &a, uint32_t v) {
  return a.outdeg ? __ldg(a.outdeg + v)
                  : (uint32_t)(__ldg(a.off + v + 1) - __ldg(a.off + v));
}

__device__ __forceinline__ double finish_vertex(const PrArgs &a, uint32_t v,
                                                double sum, double base) {
  const double r = base + a.damping * sum;
  if (a.last) a.rank[v] = (float)r;  // only the last iteration's ranks are read
  const uint32_t od = out_degree(a, v);
  a.nxt[v] = od ? (float)(r / (double)od) : 0.f;
  return od ? 0.0 : r;
}

template <int ESZ>
__device__ __forceinline__ uint32_t staged_id(const uint32_t *s_e, uint32_t i, uint32_t wshift) {
  return ESZ == 4 ? edge_dst(s_e[i], wshift) : s_e[(size_t)i * 2];
}

// Stage edges [t.ebegin, t.eend) of a tile; returns the element shift.
template <int ESZ>
__device__ __forceinline__ uint32_t stage_tile(const PrArgs &a, const PrTile &t,
                                               uint32_t *s_e) {
  const uintptr_t b = (uintptr_t)__ldg(a.blk_base + t.block);
  const uintptr_t s0 = b + (uintptr_t)t.ebegin * ESZ;
  const uintptr_t s1 = b + (uintptr_t)t.eend * ESZ;
  const uintptr_t a0 = s0 & ~(uintptr_t)15;
  const uint32_t nvec = (uint32_t)((s1 - a0 + 15) / 16);
  uint4 *dst = reinterpret_cast<uint4 *>(s_e);
  for (uint32_t i = threadIdx.x; i < nvec; i += blockDim.x) dst[i] = ld_nc_v4(a0 + 16u * i);
  return (uint32_t)((s0 - a0) / ESZ);
}

__device__ __forceinline__ double block_sum(double x, double *s_red) {
  x = warp_sum(x);
  const unsigned w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) s_red[w] = x;
  __syncthreads();
  double t = 0;
  if (threadIdx.x < 32) {
    t = threadIdx.x < (unsigned)kPrWarps ? s_red[threadIdx.x] : 0.0;
    t = warp_sum(t);
  }
  __syncthreads();
  return t;  // valid in thread 0..31
}

// Pull gather, one tile per warp.  In-edge graphs hold plain 4-byte ids
// (CSC), so a tile's edges fill at most kPullSlots slots counted from the
// start of a 128-byte line: each of a warp's loads covers whole lines, in
// HBM and over the host link alike.  Each slot is handled twice: striped for the
// gather (coalesced id loads, kPullPer independent gathers in flight per
// lane) and blocked for the sums (kPullPer consecutive slots per lane), with
// the gathered contributions crossing over in the warp's shared memory.
//
// A lane adds its consecutive slots one after the other in FP64 and closes a
// row's sum at the row's end; rows that cross a lane's span are combined by
// one segmented warp reduction per tile.  Nothing in the loop waits for
// another warp, and the ids of the warp's next tile load during the sums of
// this one, so some warps gather while others add.  What bounds it is the
// gather: one L2 sector per edge through each SM's L1 pipe.
//
// Measured per iteration at 4.2 M vertices and 65 M in-edges (RMAT, all in
// HBM): segmented reduction per 32 edges, one gather per lane in flight
// (about 30 shuffles per 32 edges, L1 pipe 61% busy) 455 us; these sums on
// 4,092-edge tiles of a 256-thread CTA, two block barriers per tile (a third
// of the stalls) 390 us; one tile per warp 287 us (227 G edges/s; 4.3 M edges
// of 262 K vertices: 62 -> 35 us).  With 60% of the edges over the host link,
// 2.1 M vertices: 2,690 -> 2,606 us (49.8 GB/s of the 51.5 zero-copy rate;
// 2,879 us while the loads started at 16-byte words).
constexpr int kPer = 16;              // slots per lane
constexpr int kSlots = 32 * kPer;     // >= kTileShape[kWarpTiles].edges + 31
constexpr int kPullVec = kPer / 4;    // 16-byte words of ids per lane
constexpr int kRows = (int)kTileShape[kWarpTiles].verts;
static_assert(kTileShape[kWarpTiles].edges + 31 < kSlots, "a tile fits the slots from any line offset");
static_assert(kTileShape[kWarpTiles].split_deg <= kTileShape[kWarpTiles].edges, "rows fit tiles");

// Rows of a warp's tile in slot numbers.
struct WarpRows {
  uint16_t off[kRows + 2];  // first slot of each row
  uint16_t row[32];         // row of each lane's first slot
};

// Position of 16-byte word v of per-slot floats in shared memory: striped
// accesses (consecutive words) and blocked ones (every fourth word) both
// touch all banks once per eight lanes.
__device__ __forceinline__ uint32_t slot_word(uint32_t v) { return v ^ ((v >> 3) & 7u); }

// The 128-byte line of a tile's first edge, the 16-byte words from there to
// its last edge, and the slot of its first edge.
struct TileSpan {
  uintptr_t a0;
  uint32_t nvec, p0;
};
template <int ESZ>
__device__ __forceinline__ TileSpan tile_span(const PrArgs &a, const PrTile &t) {
  const uintptr_t s0 = (uintptr_t)__ldg(a.blk_base + t.block) + (uintptr_t)t.ebegin * ESZ;
  const uintptr_t a0 = s0 & ~(uintptr_t)127;
  return {a0, (uint32_t)((s0 + (uintptr_t)(t.eend - t.ebegin) * ESZ - a0 + 15) / 16),
          (uint32_t)(s0 - a0) / ESZ};
}

// This lane's striped words [first, first + 32 * N) of a tile's edges.
template <int ESZ, int N>
__device__ __forceinline__ void tile_words(const TileSpan &s, uint32_t first, uint4 (&q)[N]) {
  const unsigned long long stream = l2_evict_first();
#pragma unroll
  for (int k = 0; k < N; k++) {
    const uint32_t v = first + 32u * k + lane_id();
    q[k] = v >= s.p0 / (16 / ESZ) && v < s.nvec ? ld_stream_v4(s.a0 + 16u * v, stream)
                                                : make_uint4(0, 0, 0, 0);
  }
}

// Row table of an unsplit tile whose first edge sits in slot p0.
__device__ __forceinline__ void tile_rows(const PrArgs &a, const PrTile &t, uint32_t p0, WarpRows &s) {
  const uint32_t nrows = t.vend - t.vbegin;
  for (uint32_t r = lane_id(); r < nrows; r += 32) {
    const uint32_t o0 = p0 + (uint32_t)(__ldg(a.off + t.vbegin + r) - t.ebegin);
    const uint32_t o1 = p0 + (uint32_t)(__ldg(a.off + t.vbegin + r + 1) - t.ebegin);
    s.off[r] = (uint16_t)o0;
    if (r + 1 == nrows) s.off[nrows] = (uint16_t)o1;
    if (o1 > o0) {
      // lanes whose span starts inside this row; the first row with edges
      // also takes the lanes that start in the empty slots before it (p0
      // reaches into the second lane's span)
      for (uint32_t k = o0 == p0 ? 0u : (o0 + kPer - 1) / kPer; k * kPer < o1; k++)
        s.row[k] = (uint16_t)r;
    }
  }
}

// Tiles, a.draw at a time per warp.  The first a.fixed are handed out by place,
// in rounds: the first warps of all CTAs take a round's first tiles, then the
// second warps, and so on (a.first of them).  The rest come from the
// iteration's counter: ask before the work on tile ti, which hides the draw,
// and take the tile after it.
//
// Resident graphs have one such round and draw the rest, which evens out best.
// With host-resident edges all tiles of up to kPlacedRounds rounds go by place,
// and half of more.  The order of reads over the link counts: where all warps
// drew their tiles, and where the warps of a CTA stood side by side, an
// iteration took up to twice its time on some boxes and for some placements of
// the host's pages, the more so the more edges the rows have, since early CTAs
// read one part of the array and late ones another.  In this order the CTAs
// that start together read all over a round's part of it.  All edges on the
// host, us per iteration on one box, three graphs each: tiles drawn, the warps
// of a CTA side by side, this order; a 16 KB tile per CTA (before there were
// warp tiles) on another box; the link alone takes 155, 466, 1,390 and 3,730:
//   uniform  50 K vertices,  2 M edges   258-394      213-289      174        202-248
//   uniform 100 K,           6 M         500-530      498-619      494-495    527-640
//   uniform 300 K,          18 M       1,713-1,749  1,470-1,494  1,460-1,466  1,542-1,587
//   uniform 600 K,          48 M       4,245-4,381  3,879-3,915  3,864-3,866  4,020-4,063
//   RMAT    300 K,          12 M         886-900      890-910      892-900    968-1,007
// Over very many rounds uneven tiles add up: push of RMAT 67 M vertices, half
// on the host, 530 rounds, 44.6 ms with tiles or half of them drawn, 46.1 with
// all by place (45.9 with 16 KB tiles per CTA); RMAT 17 M vertices, 350
// rounds, 40.6 and 40.7.
constexpr uint32_t kPlacedRounds = 256;
struct TileDraw {
  uint32_t left, drawn;
};
__device__ __forceinline__ uint32_t tile_round(const PrArgs &a) { return gridDim.x * a.first * a.draw; }
__device__ __forceinline__ uint32_t first_tile(const PrArgs &a, TileDraw &d) {
  const uint32_t w = threadIdx.x >> 5;
  d.left = a.draw;
  return w < a.first ? (w * gridDim.x + blockIdx.x) * a.draw : a.ntiles;
}
__device__ __forceinline__ uint32_t next_fixed(const PrArgs &a, uint32_t ti) {
  return ti + 1 - a.draw + tile_round(a);  // ti is the last of its draw
}
__device__ __forceinline__ void ask_tile(const PrArgs &a, TileDraw &d, uint32_t ti) {
  d.drawn = 0;
  if (d.left == 1 && lane_id() == 0 && next_fixed(a, ti) >= a.fixed)
    d.drawn = a.fixed + atomicAdd(a.tile_ctr + a.it, a.draw);
}
__device__ __forceinline__ uint32_t take_tile(const PrArgs &a, TileDraw &d, uint32_t ti) {
  if (--d.left) return ti + 1;
  d.left = a.draw;
  const uint32_t next = next_fixed(a, ti);
  return next < a.fixed ? next : __shfl_sync(kFull, d.drawn, 0);
}

struct PullWarp {
  float4 x[kSlots / 4];  // contributions by slot
  double sum[kRows];     // row sums; zero between tiles
  WarpRows rows;
};

// Their contributions; 0 outside the slots [p0, p1).
__device__ __forceinline__ void pull_gather(const PrArgs &a, uint32_t first, uint32_t p0, uint32_t p1,
                                            const uint4 (&q)[kPullVec], float (&x)[kPullVec][4]) {
#pragma unroll
  for (int k = 0; k < kPullVec; k++) {
    const uint32_t id[4] = {q[k].x, q[k].y, q[k].z, q[k].w};
    const uint32_t p = 4u * (first + 32u * k + lane_id());
#pragma unroll
    for (int j = 0; j < 4; j++) x[k][j] = p + j >= p0 && p + j < p1 ? __ldg(a.cur + id[j]) : 0.f;
  }
}

__global__ void __launch_bounds__(kPrThreads, 4) pr_pull_kernel(PrArgs a) {
  __shared__ PullWarp s_warp[kPrWarps];
  __shared__ double s_red[kPrWarps];
  PullWarp &s = s_warp[threadIdx.x >> 5];
  const unsigned lane = lane_id();
  const double base = (1.0 - a.damping) * a.inv_n + a.damping * ldcg(a.dang + a.it) * a.inv_n;
  double dsum = 0.0;
  for (uint32_t r = lane; r < (uint32_t)kRows; r += 32) s.sum[r] = 0.0;
  TileDraw draw;
  uint32_t ti = first_tile(a, draw);
  PrTile t{};
  TileSpan sp{};
  uint4 q[kPullVec];
  if (ti < a.ntiles) {
    t = a.tiles[ti];
    sp = tile_span<4>(a, t);
    tile_words<4>(sp, 0, q);
  }
  while (ti < a.ntiles) {
    ask_tile(a, draw, ti);
    const uint32_t p0 = sp.p0, p1 = p0 + (uint32_t)(t.eend - t.ebegin);
    const uint32_t nrows = t.vend - t.vbegin;
    if (!t.split) tile_rows(a, t, p0, s.rows);
    double acc = 0.0;
    {
      float x[kPullVec][4];
      pull_gather(a, 0, p0, p1, q, x);
      if (t.split) {
#pragma unroll
        for (int k = 0; k < kPullVec; k++)
          acc += ((double)x[k][0] + (double)x[k][1]) + ((double)x[k][2] + (double)x[k][3]);
      } else {
#pragma unroll
        for (int k = 0; k < kPullVec; k++)
          s.x[slot_word(32u * k + lane)] = make_float4(x[k][0], x[k][1], x[k][2], x[k][3]);
      }
    }
    const PrTile c = t;
    const TileSpan cs = sp;
    ti = take_tile(a, draw, ti);
    if (c.split) {
      // the rest of a long row's part
      for (uint32_t first = 32 * kPullVec; first < cs.nvec; first += 32 * kPullVec) {
        float x[kPullVec][4];
        tile_words<4>(cs, first, q);
        pull_gather(a, first, p0, p1, q, x);
#pragma unroll
        for (int k = 0; k < kPullVec; k++)
          acc += ((double)x[k][0] + (double)x[k][1]) + ((double)x[k][2] + (double)x[k][3]);
      }
    }
    if (ti < a.ntiles) {
      t = a.tiles[ti];
      sp = tile_span<4>(a, t);
      tile_words<4>(sp, 0, q);
    }
    if (c.split) {
      acc = warp_sum(acc);
      if (lane == 0) {
        const uint32_t sv = c.split - 1, parts = __ldg(a.split_parts + sv);
        bool last = parts == 1;
        if (!last) {
          atomicAdd(a.split_acc + sv, acc);
          __threadfence();
          last = atomicAdd(a.split_done + sv, 1u) + 1 == parts;
          if (last) {
            __threadfence();
            acc = __longlong_as_double((long long)atomicExch(
                reinterpret_cast<unsigned long long *>(a.split_acc + sv), 0ull));
            a.split_done[sv] = 0;
          }
        }
        if (last) dsum += finish_vertex(a, c.vbegin, acc, base);
      }
      continue;
    }
    __syncwarp();  // contributions and row table are in place
    const uint32_t b0 = kPer * lane;  // this lane's span [b0, b0 + kPer)
    uint32_t key = 0x10000u + lane;       // row whose open part this lane holds; else its own
    if (p1 > p0 && b0 < p1) {
      uint32_t r = s.rows.row[lane], end = s.rows.off[r + 1];
      bool open = s.rows.off[r] < b0;  // the row began in an earlier span
#pragma unroll
      for (int k = 0; k < kPullVec; k++) {
        const float4 f = s.x[slot_word(kPullVec * lane + k)];
        const float x[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const uint32_t p = b0 + 4u * k + j;
          if (p >= end && p < p1) {
            s.sum[r] = acc;  // the whole row, or its last open part
            acc = 0.0;
            open = false;
            do r++;
            while (s.rows.off[r + 1] <= p);
            end = s.rows.off[r + 1];
          }
          acc += (double)x[j];
        }
      }
      if (open || end > b0 + kPer) key = r;
      else s.sum[r] = acc;
    }
    __syncwarp();
    // open parts of one row in neighbouring lanes meet in the first of them,
    // which adds them to the part of the lane that closed the row (if any)
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const double y = __shfl_down_sync(kFull, acc, d);
      const uint32_t ky = __shfl_down_sync(kFull, key, d);
      if (lane + d < 32 && ky == key) acc += y;
    }
    const uint32_t kp = __shfl_up_sync(kFull, key, 1);
    if (key < 0x10000u && (lane == 0 || kp != key)) s.sum[key] += acc;
    __syncwarp();
    for (uint32_t r = lane; r < nrows; r += 32) {
      const double sum = s.sum[r];
      s.sum[r] = 0.0;
      dsum += finish_vertex(a, c.vbegin + r, sum, base);
    }
    __syncwarp();
  }
  dsum = block_sum(dsum, s_red);
  if (threadIdx.x == 0 && dsum != 0.0) atomicAdd(a.dang + a.it + 1, dsum);
}

// Push scatter, one tile per warp (the tiles and slots of the pull): every
// slot's source contribution is laid out by the lane whose span holds the
// slot, then the ids, striped over the lanes, add it to their sums, kPer
// FP64 reductions in flight per lane while the next tile's ids load.  Two
// CTAs per SM fill the reduction units; more only queue behind them (RMAT
// 4.2 M vertices, resident: 1 CTA 574 us per iteration, 2 438, 3 438, 4 485).
// With host-resident edges the link is far from filling them, and four CTAs
// keep more reads in flight (uniform 200 K vertices, 2 M edges on the host: 2
// CTAs 180 us, 4 178; RMAT 200 K 173 and 168).
//
// With host-resident edges this kernel is chosen throughout, for its loads of
// whole lines over the link: half of the edges on the host, per iteration
// against pr_push_cta_kernel, 262 K vertices 359 -> 336 us, 3 M (35 M edges)
// 1,562 -> 1,520 (46.9 -> 48.2 GB/s).
//
// Resident graphs take it while there are at most kPushWarpTiles tiles per
// warp: with more, the reduction units bound both kernels and two CTAs per SM
// bring fewer of them than the CTA kernel's eight.  CTA and warp tiles, us per
// iteration, RMAT and uniform:
//   50 K vertices,  2 M edges (1.8 tiles a warp)  37.2  30.6    31.3  24.4
//   200 K,          2 M       (1.8)               40.4  37.6    34.3  28.4
//   200 K,          2.8 M     (2.5)               45.6  44.2    38.4  33.3
//   400 K,          3.2 M     (2.8)               50.2  49.6    39.3  37.6
//   1 M,            1 M       (3.3)               37.9  49.8    35.6  44.4
//   250 K,          4 M       (3.5)               54.8  51.8    39.7  41.5
//   1 M,            4 M       (3.5)               61.0  62.0    47.9  52.2
//   450 K,          7 M       (6)                 71.4  70.8    52.1  61.7
//   1 M,            16 M      (14)                 125   125     100   118
//   4.2 M,          66 M      (58)                 461   466     398   414
constexpr int kPushCtas = 2, kPushHostCtas = 4;
constexpr uint64_t kPushWarpTiles = 3;
struct PushWarp {
  float4 x[kSlots / 4];  // source contribution of each slot
  float c[kRows];        // and of each row
  WarpRows rows;
};

template <int ESZ>
__global__ void __launch_bounds__(kPrThreads, 4) pr_push_kernel(PrArgs a) {
  constexpr int EPW = 16 / ESZ;      // edges per 16-byte word
  constexpr int NV = kPer / EPW;     // words per lane
  __shared__ PushWarp s_warp[kPrWarps];
  PushWarp &s = s_warp[threadIdx.x >> 5];
  const unsigned lane = lane_id();
  TileDraw draw;
  uint32_t ti = first_tile(a, draw);
  PrTile t{};
  TileSpan sp{};
  uint4 qn[NV];
  if (ti < a.ntiles) {
    t = a.tiles[ti];
    sp = tile_span<ESZ>(a, t);
    tile_words<ESZ>(sp, 0, qn);
  }
  while (ti < a.ntiles) {
    ask_tile(a, draw, ti);
    const PrTile c = t;
    const TileSpan cs = sp;
    const uint32_t p0 = cs.p0, p1 = p0 + (uint32_t)(c.eend - c.ebegin);
    float cv = 0.f;  // split tiles: the row's contribution
    if (c.split) {
      cv = __ldg(a.cur + c.vbegin);
    } else {
      for (uint32_t r = lane; r < c.vend - c.vbegin; r += 32) s.c[r] = __ldg(a.cur + c.vbegin + r);
      tile_rows(a, c, p0, s.rows);
      __syncwarp();
      const uint32_t b0 = kPer * lane;
      if (p1 > p0 && b0 < p1) {
        uint32_t r = s.rows.row[lane], end = s.rows.off[r + 1];
        float f = s.c[r];
#pragma unroll
        for (int k = 0; k < kPer / 4; k++) {
          float x[4];
#pragma unroll
          for (int j = 0; j < 4; j++) {
            const uint32_t p = b0 + 4u * k + j;
            if (p >= end && p < p1) {
              do r++;
              while (s.rows.off[r + 1] <= p);
              end = s.rows.off[r + 1];
              f = s.c[r];
            }
            x[j] = f;
          }
          s.x[slot_word((kPer / 4) * lane + k)] = make_float4(x[0], x[1], x[2], x[3]);
        }
      }
      __syncwarp();
    }
    uint4 q[NV];
#pragma unroll
    for (int k = 0; k < NV; k++) q[k] = qn[k];
    ti = take_tile(a, draw, ti);
    if (ti < a.ntiles) {
      t = a.tiles[ti];
      sp = tile_span<ESZ>(a, t);
      tile_words<ESZ>(sp, 0, qn);
    }
    for (uint32_t first = 0;;) {
#pragma unroll
      for (int k = 0; k < NV; k++) {
        const uint32_t v = first + 32u * k + lane, p = EPW * v;
        const uint32_t e[4] = {q[k].x, q[k].y, q[k].z, q[k].w};
        float f[4] = {cv, cv, cv, cv};
        if (!c.split) {
          // EPW slots of the 16-byte word that holds slot p
          const float *w = reinterpret_cast<const float *>(&s.x[slot_word(p / 4)]) + (p & 3u);
#pragma unroll
          for (int j = 0; j < EPW; j++) f[j] = w[j];
        }
#pragma unroll
        for (int j = 0; j < EPW; j++)
          if (p + j >= p0 && p + j < p1)
            atomicAdd(a.sum + (ESZ == 4 ? edge_dst(e[j], a.wshift) : e[2 * j]), (double)f[j]);
      }
      first += 32 * NV;
      if (first >= cs.nvec) break;  // only split tiles go on
      tile_words<ESZ>(cs, first, q);
    }
    __syncwarp();
  }
}

// Push with a tile per CTA, staged in shared memory: resident graphs of more
// than kPushWarpTiles warp tiles per warp.
template <int ESZ>
__global__ void __launch_bounds__(kPrThreads) pr_push_cta_kernel(PrArgs a) {
  __shared__ __align__(16) uint32_t s_e[kStageEdges * (ESZ / 4) + 16];
  __shared__ uint32_t s_tile;
  const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
  for (;;) {
    if (threadIdx.x == 0) s_tile = atomicAdd(a.tile_ctr + a.it, 1u);
    __syncthreads();
    const uint32_t ti = s_tile;
    if (ti >= a.ntiles) break;
    const PrTile t = a.tiles[ti];
    const uint32_t shift = stage_tile<ESZ>(a, t, s_e);
    __syncthreads();
    if (t.split) {
      const double c = (double)__ldg(a.cur + t.vbegin);
      const uint32_t cnt = (uint32_t)(t.eend - t.ebegin);
      for (uint32_t i = threadIdx.x; i < cnt; i += blockDim.x)
        atomicAdd(a.sum + staged_id<ESZ>(s_e, shift + i, a.wshift), c);
    } else {
      const uint32_t nverts = t.vend - t.vbegin;
      const uint32_t ngroups = (nverts + 31) / 32;
      for (uint32_t g = warp; g < ngroups; g += kPrWarps) {
        const uint32_t u = t.vbegin + g * 32 + lane;
        uint32_t ls = 0, deg = 0;
        float c = 0.f;
        if (u < t.vend) {
          const uint64_t e0 = __ldg(a.off + u), e1 = __ldg(a.off + u + 1);
          ls = (uint32_t)(e0 - t.ebegin);
          deg = (uint32_t)(e1 - e0);
          c = __ldg(a.cur + u);
        }
        const unsigned incl = warp_incl_scan<unsigned>(deg);
        const unsigned excl = incl - deg;
        const unsigned total = __shfl_sync(kFull, incl, 31);
        for (unsigned k = 0; k < total; k += 32) {
          const unsigned tt = k + lane;
          const int o = warp_owner(excl, tt);
          const unsigned ols = __shfl_sync(kFull, ls, o);
          const unsigned oex = __shfl_sync(kFull, excl, o);
          const float oc = __shfl_sync(kFull, c, o);
          if (tt < total)
            atomicAdd(a.sum + staged_id<ESZ>(s_e, shift + ols + (tt - oex), a.wshift), (double)oc);
        }
      }
    }
    __syncthreads();
  }
}

__global__ void pr_push_update(PrArgs a) {
  __shared__ double s_red[kPrWarps];
  const double base = (1.0 - a.damping) * a.inv_n + a.damping * ldcg(a.dang + a.it) * a.inv_n;
  double dsum = 0.0;
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < a.nv; v += gridDim.x * blockDim.x) {
    const double s = a.sum[v];
    a.sum[v] = 0.0;
    dsum += finish_vertex(a, v, s, base);
  }
  dsum = block_sum(dsum, s_red);
  if (threadIdx.x == 0 && dsum != 0.0) atomicAdd(a.dang + a.it + 1, dsum);
}

__global__ void pr_init(PrArgs a, float *c0) {
  __shared__ double s_red[kPrWarps];
  double dsum = 0.0;
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < a.nv; v += gridDim.x * blockDim.x) {
    const uint32_t od = out_degree(a, v);
    c0[v] = od ? (float)(a.inv_n / (double)od) : 0.f;
    if (!od) dsum += a.inv_n;
    if (a.sum) a.sum[v] = 0.0;
  }
  dsum = block_sum(dsum, s_red);
  if (threadIdx.x == 0 && dsum != 0.0) atomicAdd(a.dang, dsum);
}

// Ranks as the doubles the caller gets: vertices below half into lo, the
// rest into hi.  The host used to widen a pageable copy of the ranks one by
// one, which took longer than a resident run's 20 iterations (4.2 M
// vertices: 8.5 ms after 9.1 ms of iterations).  Widened here, the ranks
// cross the link as twice the bytes but straight into the caller's buffer
// (33.5 MB, 0.6 ms; the whole call 17.7 -> 9.7 ms); the two contribution
// arrays, which nothing reads between runs, hold exactly one half each, so no
// memory is added.
__global__ void pr_widen(const float *rank, uint64_t nv, uint64_t half, double *lo, double *hi) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < half;
       i += (uint64_t)gridDim.x * blockDim.x) {
    lo[i] = (double)rank[i];
    if (half + i < nv) hi[i] = (double)rank[half + i];
  }
}

// ------------------------------------------- reference semantics (FP64) --
//
// THV_RUN_PR_REFERENCE reproduces the reference engine's own PageRank so its
// values.bin can be compared with the reference comparer's 1e-3 absolute
// tolerance (comparer/compare.cpp:155).  Its constants are floats
// (src/common.cuh:48-49) mixed into double expressions; the same expressions
// here give the same promoted values.
//   pull: r0 = 1/N (src/graph.cuh:239-240); per round every active vertex
//         sums r(u)/outdeg(u) over its in-edges from the previous round's
//         values, then r = (1-a) + a*sum and it stays active while the change
//         exceeds the tolerance (src/pr/pr_kernels.cu:23-55, :449-476);
//   push: r0 = 1-a, delta0 = (1-a)*a/outdeg in float, residual 0
//         (src/graph.cuh:233-237); per round each active u adds delta(u) to
//         residual(w) over its out-edges (pr_kernels.cu:504-681), then every
//         vertex with residual > tol takes it and becomes active, the rest
//         inactive (pr_kernels.cu:846-860, frontier cleared each round at
//         src/pr/pr.cu:1067-1077).
// Rounds run until no vertex is active.  The gather/scatter kernels reuse
// tiles sized for a CTA and skip tiles without an active
// vertex, so converged regions cost one flag read per vertex.  Pull sums are
// warp-segmented (fixed order) with atomics only across the parts of a split
// vertex; push adds with FP64 atomics like the reference.
constexpr float kRefAlpha = 0.85f, kRefTol = 0.001f;

struct PrRefArgs {
  const PrTile *tiles;
  const uint64_t *blk_base;
  const uint64_t *off;
  const uint32_t *outdeg;  // CSC: explicit; CSR: nullptr
  double *val, *acc, *delta;
  uint8_t *act;
  double *split_acc;
  uint32_t *split_done;
  const uint32_t *split_parts;
  uint32_t *tile_ctr;
  unsigned long long *cnt;  // [0] active vertices, [1] their edges
  uint32_t ntiles, nv, wshift, pad;
};

__device__ __forceinline__ uint32_t ref_out_degree(const PrRefArgs &a, uint32_t v) {
  return a.outdeg ? __ldg(a.outdeg + v)
                  : (uint32_t)(__ldg(a.off + v + 1) - __ldg(a.off + v));
}

// Stage edges [t.ebegin, t.eend) of a tile (same layout as stage_tile).
template <int ESZ>
__device__ __forceinline__ uint32_t ref_stage(const PrRefArgs &a, const PrTile &t, uint32_t *s_e) {
  const uintptr_t b = (uintptr_t)__ldg(a.blk_base + t.block);
  const uintptr_t s0 = b + (uintptr_t)t.ebegin * ESZ;
  const uintptr_t s1 = b + (uintptr_t)t.eend * ESZ;
  const uintptr_t a0 = s0 & ~(uintptr_t)15;
  const uint32_t nvec = (uint32_t)((s1 - a0 + 15) / 16);
  uint4 *dst = reinterpret_cast<uint4 *>(s_e);
  for (uint32_t i = threadIdx.x; i < nvec; i += blockDim.x) dst[i] = ld_nc_v4(a0 + 16u * i);
  return (uint32_t)((s0 - a0) / ESZ);
}

// Next tile with an active vertex; returns false when the tiles are done.
__device__ __forceinline__ bool ref_next_tile(const PrRefArgs &a, PrTile *t, uint32_t *s_tile) {
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) *s_tile = atomicAdd(a.tile_ctr, 1u);
    __syncthreads();
    const uint32_t ti = *s_tile;
    if (ti >= a.ntiles) return false;
    *t = a.tiles[ti];
    int any = 0;
    for (uint32_t v = t->vbegin + threadIdx.x; v < t->vend; v += blockDim.x) any |= a.act[v];
    if (__syncthreads_or(any)) return true;
  }
}

template <int ESZ>
__global__ void __launch_bounds__(kPrThreads) pr_ref_pull_kernel(PrRefArgs a) {
  __shared__ __align__(16) uint32_t s_e[kStageEdges * (ESZ / 4) + 16];
  __shared__ double s_acc[kPrWarps][32];
  __shared__ double s_red[kPrWarps];
  __shared__ uint32_t s_tile;
  const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
  PrTile t;
  while (ref_next_tile(a, &t, &s_tile)) {
    const uint32_t shift = ref_stage<ESZ>(a, t, s_e);
    __syncthreads();
    if (t.split) {
      const uint32_t cnt = (uint32_t)(t.eend - t.ebegin);
      double part = 0.0;
      for (uint32_t i = threadIdx.x; i < cnt; i += blockDim.x) {
        const uint32_t u = staged_id<ESZ>(s_e, shift + i, a.wshift);
        const uint32_t od = __ldg(a.outdeg + u);
        if (od) part += a.val[u] / (double)od;
      }
      part = block_sum(part, s_red);
      if (threadIdx.x == 0) {
        const uint32_t sv = t.split - 1;
        atomicAdd(a.split_acc + sv, part);
        __threadfence();
        const uint32_t done = atomicAdd(a.split_done + sv, 1u);
        if (done + 1 == __ldg(a.split_parts + sv)) {
          __threadfence();
          const unsigned long long bits =
              atomicExch(reinterpret_cast<unsigned long long *>(a.split_acc + sv), 0ull);
          a.split_done[sv] = 0;
          a.acc[t.vbegin] = __longlong_as_double((long long)bits);
        }
      }
    } else {
      const uint32_t nverts = t.vend - t.vbegin;
      const uint32_t ngroups = (nverts + 31) / 32;
      for (uint32_t g = warp; g < ngroups; g += kPrWarps) {
        const uint32_t v = t.vbegin + g * 32 + lane;
        const bool on = v < t.vend && a.act[v];
        uint32_t ls = 0, deg = 0;
        if (on) {
          const uint64_t e0 = __ldg(a.off + v), e1 = __ldg(a.off + v + 1);
          ls = (uint32_t)(e0 - t.ebegin);
          deg = (uint32_t)(e1 - e0);
        }
        const unsigned incl = warp_incl_scan<unsigned>(deg);
        const unsigned excl = incl - deg;
        const unsigned total = __shfl_sync(kFull, incl, 31);
        s_acc[warp][lane] = 0.0;
        __syncwarp();
        for (unsigned k = 0; k < total; k += 32) {
          const unsigned tt = k + lane;
          const int o = warp_owner(excl, tt);
          const unsigned ols = __shfl_sync(kFull, ls, o);
          const unsigned oex = __shfl_sync(kFull, excl, o);
          double x = 0.0;
          int pos = 32;
          if (tt < total) {
            const uint32_t u = staged_id<ESZ>(s_e, shift + ols + (tt - oex), a.wshift);
            const uint32_t od = __ldg(a.outdeg + u);
            x = od ? a.val[u] / (double)od : 0.0;
            pos = o;
          }
#pragma unroll
          for (int d = 1; d < 32; d <<= 1) {
            const double y = __shfl_up_sync(kFull, x, d);
            const int pp = __shfl_up_sync(kFull, pos, d);
            if (lane >= (unsigned)d && pp == pos) x += y;
          }
          const int nxt = __shfl_down_sync(kFull, pos, 1);
          if ((lane == 31 || nxt != pos) && pos < 32) s_acc[warp][pos] += x;
          __syncwarp();
        }
        if (on) a.acc[v] = s_acc[warp][lane];
        __syncwarp();
      }
    }
  }
}

template <int ESZ>
__global__ void __launch_bounds__(kPrThreads) pr_ref_push_kernel(PrRefArgs a) {
  __shared__ __align__(16) uint32_t s_e[kStageEdges * (ESZ / 4) + 16];
  __shared__ uint32_t s_tile;
  const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
  PrTile t;
  while (ref_next_tile(a, &t, &s_tile)) {
    const uint32_t shift = ref_stage<ESZ>(a, t, s_e);
    __syncthreads();
    if (t.split) {
      const double c = a.delta[t.vbegin];
      const uint32_t cnt = (uint32_t)(t.eend - t.ebegin);
      for (uint32_t i = threadIdx.x; i < cnt; i += blockDim.x)
        atomicAdd(a.acc + staged_id<ESZ>(s_e, shift + i, a.wshift), c);
    } else {
      const uint32_t nverts = t.vend - t.vbegin;
      const uint32_t ngroups = (nverts + 31) / 32;
      for (uint32_t g = warp; g < ngroups; g += kPrWarps) {
        const uint32_t u = t.vbegin + g * 32 + lane;
        uint32_t ls = 0, deg = 0;
        double c = 0.0;
        if (u < t.vend && a.act[u]) {
          const uint64_t e0 = __ldg(a.off + u), e1 = __ldg(a.off + u + 1);
          ls = (uint32_t)(e0 - t.ebegin);
          deg = (uint32_t)(e1 - e0);
          c = a.delta[u];
        }
        const unsigned incl = warp_incl_scan<unsigned>(deg);
        const unsigned excl = incl - deg;
        const unsigned total = __shfl_sync(kFull, incl, 31);
        for (unsigned k = 0; k < total; k += 32) {
          const unsigned tt = k + lane;
          const int o = warp_owner(excl, tt);
          const unsigned ols = __shfl_sync(kFull, ls, o);
          const unsigned oex = __shfl_sync(kFull, excl, o);
          const double oc = __shfl_sync(kFull, c, o);
          if (tt < total) atomicAdd(a.acc + staged_id<ESZ>(s_e, shift + ols + (tt - oex), a.wshift), oc);
        }
      }
    }
  }
}

__device__ __forceinline__ void ref_count(const PrRefArgs &a, unsigned long long nact,
                                          unsigned long long nedge) {
  nact = warp_sum(nact);
  nedge = warp_sum(nedge);
  if (lane_id() == 0 && nact) {
    atomicAdd(a.cnt, nact);
    atomicAdd(a.cnt + 1, nedge);
  }
}

// Edges the next round reads for an active vertex: its in-edges (pull over
// CSC) or its out-edges (push over CSR), both given by the offsets.
__device__ __forceinline__ uint32_t ref_edges(const PrRefArgs &a, uint32_t v) {
  return (uint32_t)(__ldg(a.off + v + 1) - __ldg(a.off + v));
}

__global__ void pr_ref_init(PrRefArgs a, int push) {
  unsigned long long nact = 0, nedge = 0;
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < a.nv; v += gridDim.x * blockDim.x) {
    a.act[v] = 1;
    a.acc[v] = 0.0;
    if (push) {
      a.val[v] = (double)(1.0f - kRefAlpha);
      a.delta[v] = (double)((1.0f - kRefAlpha) * kRefAlpha / (float)ref_out_degree(a, v));
    } else {
      a.val[v] = 1.0 / (double)a.nv;
    }
    nact++;
    nedge += ref_edges(a, v);
  }
  ref_count(a, nact, nedge);
}

__global__ void pr_ref_pull_update(PrRefArgs a) {
  unsigned long long nact = 0, nedge = 0;
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < a.nv; v += gridDim.x * blockDim.x) {
    if (!a.act[v]) continue;
    const double t = (1 - kRefAlpha) + kRefAlpha * a.acc[v];
    const double old = a.val[v];
    const double diff = t > old ? t - old : old - t;
    a.val[v] = t;
    const bool on = diff > kRefTol;
    a.act[v] = on;
    if (on) {
      nact++;
      nedge += ref_edges(a, v);
    }
  }
  ref_count(a, nact, nedge);
}

__global__ void pr_ref_push_update(PrRefArgs a) {
  unsigned long long nact = 0, nedge = 0;
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < a.nv; v += gridDim.x * blockDim.x) {
    const double r = a.acc[v];
    const bool on = r > kRefTol;
    if (on) {
      a.val[v] += r;
      a.delta[v] = r * kRefAlpha / (double)ref_out_degree(a, v);
      a.acc[v] = 0.0;
      nact++;
      nedge += ref_edges(a, v);
    }
    a.act[v] = on;
  }
  ref_count(a, nact, nedge);
}

// ------------------------------------------------------------------ host --

void pagerank_free(thv_graph *g) {
  PrState *p = g->ps;
  if (!p) return;
  dev_free(p->d_c[0]);
  dev_free(p->d_c[1]);
  dev_free(p->d_rank);
  dev_free(p->d_sum);
  dev_free(p->d_split_acc);
  dev_free(p->d_split_done);
  dev_free(p->d_dang);
  dev_free(p->d_tile_ctr);
  dev_free(p->d_val);
  dev_free(p->d_acc);
  dev_free(p->d_delta);
  dev_free(p->d_act);
  dev_free(p->d_cnt);
  pinned_free(p->h_cnt);
  if (p->ev0) cudaEventDestroy(p->ev0);
  if (p->ev1) cudaEventDestroy(p->ev1);
  delete p;
  g->ps = nullptr;
}

static thv_status ensure_pr_state(thv_graph *g, bool push, uint32_t iters, bool ref,
                                  const PrTiles &tiles) {
  PrState *&p = g->ps;
  const size_t nsplit = std::max<size_t>(1, tiles.split_parts.size());
  if (p && p->push == push && p->ref == ref && (ref || p->cap_iters >= iters) && p->nsplit == nsplit)
    return THV_OK;
  pagerank_free(g);
  p = new PrState();
  p->nv = g->nv;
  p->push = push;
  p->ref = ref;
  p->nsplit = nsplit;
  if (ref) {
    THV_TRY(dev_alloc((void **)&p->d_val, g->nv * 8 + 64, "pr values"));
    THV_TRY(dev_alloc((void **)&p->d_acc, g->nv * 8 + 64, "pr sums"));
    if (push) THV_TRY(dev_alloc((void **)&p->d_delta, g->nv * 8 + 64, "pr deltas"));
    THV_TRY(dev_alloc((void **)&p->d_act, g->nv + 64, "pr active flags"));
    THV_TRY(dev_alloc((void **)&p->d_cnt, 16, "pr round counters"));
    THV_TRY(pinned_alloc((void **)&p->h_cnt, 16, "pr round counters"));
    THV_TRY(dev_alloc((void **)&p->d_split_acc, nsplit * 8, "pr split sums"));
    THV_TRY(dev_alloc((void **)&p->d_split_done, nsplit * 4, "pr split counters"));
    THV_TRY(dev_alloc((void **)&p->d_tile_ctr, 4, "pr tile counter"));
    THV_CUDA(cudaEventCreate(&p->ev0));
    THV_CUDA(cudaEventCreate(&p->ev1));
    return THV_OK;
  }
  p->cap_iters = std::max<uint32_t>(iters, 32);
  THV_TRY(dev_alloc((void **)&p->d_c[0], g->nv * 4 + 64, "pr contributions"));
  THV_TRY(dev_alloc((void **)&p->d_c[1], g->nv * 4 + 64, "pr contributions"));
  THV_TRY(dev_alloc((void **)&p->d_rank, g->nv * 4 + 64, "pr ranks"));
  if (push) THV_TRY(dev_alloc((void **)&p->d_sum, g->nv * 8 + 64, "pr sums"));
  THV_TRY(dev_alloc((void **)&p->d_split_acc, nsplit * 8, "pr split sums"));
  THV_TRY(dev_alloc((void **)&p->d_split_done, nsplit * 4, "pr split counters"));
  THV_TRY(dev_alloc((void **)&p->d_dang, (p->cap_iters + 1) * 8, "pr dangling"));
  THV_TRY(dev_alloc((void **)&p->d_tile_ctr, p->cap_iters * 4, "pr tile counters"));
  THV_CUDA(cudaEventCreate(&p->ev0));
  THV_CUDA(cudaEventCreate(&p->ev1));
  return THV_OK;
}

template <int ESZ>
static thv_status pr_iterate(thv_graph *g, PrArgs &a, bool push, PrTileKind kind, uint32_t iters,
                             cudaStream_t st, uint32_t &launches) {
  PrState *p = g->ps;
  const bool host = g->plan.host_edge_bytes > 0;
  int bpsm = 0;
  if (push && kind == kWarpTiles)
    bpsm = host ? kPushHostCtas : kPushCtas;
  else if (push)
    THV_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bpsm, pr_push_cta_kernel<ESZ>, kPrThreads, 0));
  else
    THV_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bpsm, pr_pull_kernel, kPrThreads, 0));
  const int grid = std::max(1, bpsm) * g->num_sms;
  const int ugrid = std::max(1, std::min<int>(g->num_sms * 8, (int)((g->nv + kPrThreads - 1) / kPrThreads)));
  // several tiles per draw only while every warp still draws often enough
  // for the last ones to even out
  const uint32_t warps = (uint32_t)grid * kPrWarps;
  a.draw = host ? 1u : std::min(4u, std::max(1u, a.ntiles / (16u * warps)));
  a.first = std::min((uint32_t)kPrWarps, (a.ntiles + (uint32_t)grid - 1) / (uint32_t)grid);
  const uint32_t rounds = (a.ntiles + warps - 1) / warps;
  a.fixed = (host ? rounds <= kPlacedRounds ? rounds : rounds / 2 : 1u) * (uint32_t)grid * a.first * a.draw;
  for (uint32_t it = 0; it < iters; it++) {
    a.it = it;
    a.last = it + 1 == iters;
    a.cur = p->d_c[it & 1];
    a.nxt = p->d_c[(it + 1) & 1];
    if (push) {
      if (kind == kWarpTiles) pr_push_kernel<ESZ><<<grid, kPrThreads, 0, st>>>(a);
      else pr_push_cta_kernel<ESZ><<<grid, kPrThreads, 0, st>>>(a);
      pr_push_update<<<ugrid, kPrThreads, 0, st>>>(a);
      launches += 2;
    } else {
      pr_pull_kernel<<<grid, kPrThreads, 0, st>>>(a);
      launches += 1;
    }
    THV_CUDA(cudaGetLastError());
  }
  return THV_OK;
}

// Reference semantics: one gather/scatter launch and one update launch per
// round; the host reads the round's active count (16 bytes) to stop.
static thv_status run_pagerank_ref(thv_graph *g, thv_algo algo, const thv_run_opts *o,
                                   cudaStream_t st, thv_stats *stats) {
  const bool push = algo == THV_ALGO_PR_PUSH;
  const uint32_t max_rounds = o && o->pr_iters ? o->pr_iters : 100000u;
  THV_TRY(ensure_plan(g));
  THV_TRY(build_tiles(g, kCtaTiles));
  const PrTiles &tiles = g->plan.tiles[kCtaTiles];
  THV_TRY(ensure_pr_state(g, push, 0, true, tiles));
  PrState *p = g->ps;
  PrRefArgs a{};
  a.tiles = tiles.d_tiles;
  a.blk_base = g->plan.d_base;
  a.off = g->d_off;
  a.outdeg = g->fmt == THV_FMT_CSC ? g->d_outdeg : nullptr;
  a.val = p->d_val;
  a.acc = p->d_acc;
  a.delta = p->d_delta;
  a.act = p->d_act;
  a.split_acc = p->d_split_acc;
  a.split_done = p->d_split_done;
  a.split_parts = tiles.d_split_parts;
  a.tile_ctr = p->d_tile_ctr;
  a.cnt = p->d_cnt;
  a.ntiles = (uint32_t)tiles.tiles.size();
  a.nv = (uint32_t)g->nv;
  a.wshift = g->wshift;
  int bpsm = 0;
  if (push)
    THV_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bpsm, g->esz == 8 ? pr_ref_push_kernel<8> : pr_ref_push_kernel<4>, kPrThreads, 0));
  else
    THV_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bpsm, g->esz == 8 ? pr_ref_pull_kernel<8> : pr_ref_pull_kernel<4>, kPrThreads, 0));
  const int grid = std::max(1, bpsm) * g->num_sms;
  const int ugrid = std::max(1, std::min<int>(g->num_sms * 8, (int)((g->nv + kPrThreads - 1) / kPrThreads)));
  const size_t nsplit = std::max<size_t>(1, tiles.split_parts.size());
  uint32_t launches = 0, rounds = 0;
  uint64_t edges = 0;
  THV_CUDA(cudaEventRecord(p->ev0, st));
  THV_CUDA(cudaMemsetAsync(p->d_split_acc, 0, nsplit * 8, st));
  THV_CUDA(cudaMemsetAsync(p->d_split_done, 0, nsplit * 4, st));
  THV_CUDA(cudaMemsetAsync(p->d_cnt, 0, 16, st));
  pr_ref_init<<<ugrid, kPrThreads, 0, st>>>(a, push ? 1 : 0);
  THV_CUDA(cudaGetLastError());
  launches++;
  THV_CUDA(cudaMemcpyAsync(p->h_cnt, p->d_cnt, 16, cudaMemcpyDeviceToHost, st));
  THV_CUDA(cudaStreamSynchronize(st));
  while (p->h_cnt[0]) {
    if (rounds == max_rounds) return fail(THV_ETIMEOUT, "PageRank did not converge in %u rounds", max_rounds);
    edges += p->h_cnt[1];
    THV_CUDA(cudaMemsetAsync(p->d_tile_ctr, 0, 4, st));
    THV_CUDA(cudaMemsetAsync(p->d_cnt, 0, 16, st));
    if (push) {
      if (g->esz == 8) pr_ref_push_kernel<8><<<grid, kPrThreads, 0, st>>>(a);
      else pr_ref_push_kernel<4><<<grid, kPrThreads, 0, st>>>(a);
      pr_ref_push_update<<<ugrid, kPrThreads, 0, st>>>(a);
    } else {
      if (g->esz == 8) pr_ref_pull_kernel<8><<<grid, kPrThreads, 0, st>>>(a);
      else pr_ref_pull_kernel<4><<<grid, kPrThreads, 0, st>>>(a);
      pr_ref_pull_update<<<ugrid, kPrThreads, 0, st>>>(a);
    }
    THV_CUDA(cudaGetLastError());
    launches += 2;
    THV_CUDA(cudaMemcpyAsync(p->h_cnt, p->d_cnt, 16, cudaMemcpyDeviceToHost, st));
    THV_CUDA(cudaStreamSynchronize(st));
    rounds++;
  }
  THV_CUDA(cudaEventRecord(p->ev1, st));
  THV_CUDA(cudaStreamSynchronize(st));
  g->last_algo = algo;
  if (stats) {
    float ms_ = 0.f;
    cudaEventElapsedTime(&ms_, p->ev0, p->ev1);
    stats->device_ms = ms_;
    stats->iterations = rounds;
    stats->edges_expanded = edges;
    stats->kernel_launches = launches;
  }
  return THV_OK;
}

thv_status run_pagerank(thv_graph *g, thv_algo algo, const thv_run_opts *o,
                        cudaStream_t st, thv_stats *stats) {
  const bool push = algo == THV_ALGO_PR_PUSH;
  if (push && g->fmt == THV_FMT_CSC)
    return fail(THV_EINVAL, "push PageRank needs out-edges (CSR), got CSC");
  if (!push && g->fmt != THV_FMT_CSC)
    return fail(THV_EINVAL, "pull PageRank needs in-edges (CSC)");
  if (g->nv == 0) return fail(THV_EINVAL, "empty graph");
  if (o && (o->flags & THV_RUN_PR_REFERENCE)) return run_pagerank_ref(g, algo, o, st, stats);
  const uint32_t iters = o && o->pr_iters ? o->pr_iters : 20u;
  const double damping = o && o->pr_damping > 0 ? o->pr_damping : 0.85;
  THV_TRY(ensure_plan(g));
  const uint64_t warps = (uint64_t)kPushCtas * g->num_sms * kPrWarps;
  const uint64_t warp_tiles =
      std::max(g->ne / kTileShape[kWarpTiles].edges, g->nv / kTileShape[kWarpTiles].verts);
  const PrTileKind kind = push && g->plan.host_edge_bytes == 0 && warp_tiles > kPushWarpTiles * warps
                              ? kCtaTiles
                              : kWarpTiles;
  THV_TRY(build_tiles(g, kind));
  const PrTiles &tiles = g->plan.tiles[kind];
  THV_TRY(ensure_pr_state(g, push, iters, false, tiles));
  PrState *p = g->ps;
  p->iters = iters;

  PrArgs a{};
  a.tiles = tiles.d_tiles;
  a.blk_base = g->plan.d_base;
  a.off = g->d_off;
  a.outdeg = g->fmt == THV_FMT_CSC ? g->d_outdeg : nullptr;
  a.rank = p->d_rank;
  a.sum = p->d_sum;
  a.split_acc = p->d_split_acc;
  a.split_done = p->d_split_done;
  a.split_parts = tiles.d_split_parts;
  a.dang = p->d_dang;
  a.tile_ctr = p->d_tile_ctr;
  a.ntiles = (uint32_t)tiles.tiles.size();
  a.nv = (uint32_t)g->nv;
  a.damping = damping;
  a.inv_n = 1.0 / (double)g->nv;
  a.wshift = g->wshift;

  uint32_t launches = 0;
  THV_CUDA(cudaEventRecord(p->ev0, st));
  THV_CUDA(cudaMemsetAsync(p->d_dang, 0, (iters + 1) * 8, st));
  THV_CUDA(cudaMemsetAsync(p->d_tile_ctr, 0, iters * 4, st));
  const size_t nsplit = std::max<size_t>(1, tiles.split_parts.size());
  THV_CUDA(cudaMemsetAsync(p->d_split_acc, 0, nsplit * 8, st));
  THV_CUDA(cudaMemsetAsync(p->d_split_done, 0, nsplit * 4, st));
  const int ugrid = std::max(1, std::min<int>(g->num_sms * 8, (int)((g->nv + kPrThreads - 1) / kPrThreads)));
  pr_init<<<ugrid, kPrThreads, 0, st>>>(a, p->d_c[0]);
  THV_CUDA(cudaGetLastError());
  launches++;
  thv_status s = g->esz == 8 ? pr_iterate<8>(g, a, push, kind, iters, st, launches)
                             : pr_iterate<4>(g, a, push, kind, iters, st, launches);
  if (s != THV_OK) return s;
  THV_CUDA(cudaEventRecord(p->ev1, st));
  THV_CUDA(cudaStreamSynchronize(st));
  g->last_algo = algo;
  if (stats) {
    float ms_ = 0.f;
    cudaEventElapsedTime(&ms_, p->ev0, p->ev1);
    stats->device_ms = ms_;
    stats->iterations = iters;
    stats->edges_expanded = g->ne * iters;
    uint64_t hbm = 0, link = 0;  // whole blocks: PageRank does not read the small-list cache
    for (const Block &b : g->plan.blocks) (b.resident ? hbm : link) += (b.eend - b.ebegin) * g->esz;
    stats->hbm_edge_bytes = hbm * iters;
    stats->link_edge_bytes = link * iters;
    stats->kernel_launches = launches;
  }
  return THV_OK;
}

thv_status pagerank_values(thv_graph *g, double *out, cudaStream_t st) {
  if (!g->ps) return fail(THV_EINVAL, "no PageRank values");
  if (g->ps->ref) {
    THV_CUDA(cudaMemcpyAsync(out, g->ps->d_val, g->nv * 8, cudaMemcpyDeviceToHost, st));
    THV_CUDA(cudaStreamSynchronize(st));
    return THV_OK;
  }
  PrState *p = g->ps;
  const uint64_t half = (g->nv + 1) / 2;
  double *lo = (double *)p->d_c[0], *hi = (double *)p->d_c[1];
  const int grid = std::max(1, std::min<int>(g->num_sms * 8, (int)((half + kPrThreads - 1) / kPrThreads)));
  pr_widen<<<grid, kPrThreads, 0, st>>>(p->d_rank, g->nv, half, lo, hi);
  THV_CUDA(cudaGetLastError());
  THV_CUDA(cudaMemcpyAsync(out, lo, half * 8, cudaMemcpyDeviceToHost, st));
  if (g->nv > half)
    THV_CUDA(cudaMemcpyAsync(out + half, hi, (g->nv - half) * 8, cudaMemcpyDeviceToHost, st));
  THV_CUDA(cudaStreamSynchronize(st));
  return THV_OK;
}

}  // namespace thv
