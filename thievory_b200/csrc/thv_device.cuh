// Device-side helpers: coherent loads, warp collectives, bounded grid barrier.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "thv_internal.h"

namespace thv {

constexpr unsigned kFull = 0xFFFFFFFFu;

// Device error codes (0 = ok); a launch's control word holds bit code - 1.
enum : unsigned {
  kDevOk = 0,
  kDevErrBarrier = 1,   // a grid barrier wait ran out of time
  kDevErrIters = 2,     // iteration cap reached
  kDevErrQueue = 3,     // work queue capacity exceeded
  kDevErrDepth = 4,     // batched BFS level exceeded the u8 range
};

// L2-coherent load (bypasses the non-coherent L1) for data other SMs write.
__device__ __forceinline__ uint32_t ldcg(const uint32_t *p) { return __ldcg(p); }
__device__ __forceinline__ unsigned long long ldcg(const unsigned long long *p) {
  return __ldcg(p);
}
__device__ __forceinline__ double ldcg(const double *p) { return __ldcg(p); }

// Read-only 16-byte load; works for HBM and for host-mapped pinned memory.
__device__ __forceinline__ uint4 ld_nc_v4(uintptr_t addr) {
  return __ldg(reinterpret_cast<const uint4 *>(addr));
}
__device__ __forceinline__ uint32_t ld_nc_u32(uintptr_t addr) {
  return __ldg(reinterpret_cast<const uint32_t *>(addr));
}
__device__ __forceinline__ uint2 ld_nc_u2(uintptr_t addr) {
  return __ldg(reinterpret_cast<const uint2 *>(addr));
}

// L2 eviction priorities (createpolicy + .L2::cache_hint): streaming data
// read once (edges, queue items) is marked evict-first so that it does not
// push the randomly probed per-vertex values out of L2; those are marked
// evict-last.  A hint only orders evictions; results do not depend on it.
__device__ __forceinline__ unsigned long long l2_evict_first() {
  unsigned long long p;
  asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ unsigned long long l2_evict_last() {
  unsigned long long p;
  asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}
// Read-only 16 / 4 / 8-byte streaming loads with an L2 policy, not kept in L1.
__device__ __forceinline__ uint4 ld_stream_v4(uintptr_t addr, unsigned long long pol) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.v4.u32 {%0, %1, %2, %3}, [%4], %5;"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(addr), "l"(pol));
  return v;
}
__device__ __forceinline__ uint32_t ld_stream_u32(uintptr_t addr, unsigned long long pol) {
  uint32_t v;
  asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.u32 %0, [%1], %2;"
               : "=r"(v)
               : "l"(addr), "l"(pol));
  return v;
}
__device__ __forceinline__ uint2 ld_stream_u2(uintptr_t addr, unsigned long long pol) {
  uint2 v;
  asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.v2.u32 {%0, %1}, [%2], %3;"
               : "=r"(v.x), "=r"(v.y)
               : "l"(addr), "l"(pol));
  return v;
}
// L2-coherent load / atomic min of a value other SMs write, with an L2 policy.
__device__ __forceinline__ uint32_t ldcg_hint(const uint32_t *p, unsigned long long pol) {
  uint32_t v;
  asm volatile("ld.global.cg.L2::cache_hint.u32 %0, [%1], %2;" : "=r"(v) : "l"(p), "l"(pol));
  return v;
}
// atomicMin whose old value nobody waits for (a reduction).
__device__ __forceinline__ void red_min_hint(uint32_t *p, uint32_t x, unsigned long long pol) {
  asm volatile("red.global.min.L2::cache_hint.u32 [%0], %1, %2;" : : "l"(p), "r"(x), "l"(pol)
               : "memory");
}
__device__ __forceinline__ uint32_t atomic_min_hint(uint32_t *p, uint32_t x, unsigned long long pol) {
  uint32_t old;
  asm volatile("atom.global.min.L2::cache_hint.u32 %0, [%1], %2, %3;"
               : "=r"(old)
               : "l"(p), "r"(x), "l"(pol)
               : "memory");
  return old;
}

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ unsigned lane_id() { return threadIdx.x & 31u; }

__device__ __forceinline__ unsigned lanemask_lt() {
  unsigned m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

template <typename T>
__device__ __forceinline__ T warp_incl_scan(T x) {
  const unsigned lane = lane_id();
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    T y = __shfl_up_sync(kFull, x, d);
    if (lane >= (unsigned)d) x += y;
  }
  return x;
}

template <typename T>
__device__ __forceinline__ T warp_sum(T x) {
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) x += __shfl_xor_sync(kFull, x, d);
  return x;
}

__device__ __forceinline__ unsigned long long warp_or(unsigned long long x) {
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) x |= __shfl_xor_sync(kFull, x, d);
  return x;
}

__device__ __forceinline__ unsigned warp_min(unsigned x) {
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) x = min(x, __shfl_xor_sync(kFull, x, d));
  return x;
}

__device__ __forceinline__ unsigned long long shfl64(unsigned long long x,
                                                     int src) {
  return __shfl_sync(kFull, x, src);
}

// Largest lane l with excl[l] <= t, for excl non-decreasing across the warp.
__device__ __forceinline__ int warp_owner(unsigned excl, unsigned t) {
  int pos = 0;
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) {
    const unsigned e = __shfl_sync(kFull, excl, pos + s);
    if (e <= t) pos += s;
  }
  return pos;
}

// Frontier work item: the adjacency of vertex v (or one chunk of it) at a
// device or host-mapped address.
struct __align__(16) WorkItem {
  uint64_t eaddr;
  uint32_t v;
  uint32_t cnt;
};

constexpr uint32_t kSmemBlocks = 2048;  // block tables up to this size go to smem

// Edge block of vertex v: largest b with vb[b] <= v (vb has nblk+1 entries).
__device__ __forceinline__ uint32_t find_block(const uint32_t *vb, uint32_t nblk,
                                               uint32_t v) {
  uint32_t lo = 0, hi = nblk;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (vb[mid] <= v) lo = mid;
    else hi = mid;
  }
  return lo;
}

// A 4-byte edge: the neighbour id in the high bits and, for packed weighted
// graphs, w - wbase in the low wshift bits (wshift = 0: an id-only edge).
__device__ __forceinline__ uint32_t edge_dst(uint32_t e, uint32_t wshift) { return e >> wshift; }
__device__ __forceinline__ uint32_t edge_wt(uint32_t e, uint32_t wshift, uint32_t wbase) {
  return (e & ((1u << wshift) - 1u)) + wbase;
}

// Device address of the first edge of v's list, given its block's base and
// its first edge index s0; *host says whether it is read over the host link.
__device__ __forceinline__ unsigned long long list_addr(const ListCache &lc,
                                                       unsigned long long block_base,
                                                       unsigned long long host_base, uint32_t v,
                                                       uint64_t s0, uint32_t deg, uint32_t esz,
                                                       bool *host) {
  const bool on_host = block_base == host_base;
  if (on_host && deg < lc.deg_lt && deg > 0) {
    *host = false;
    return lc.base + (unsigned long long)__ldg(lc.idx + v) * esz;
  }
  *host = on_host;
  return block_base + s0 * esz;
}

// Grid-wide barrier for a cooperative launch: one 64-bit word, arrivals in
// the high half and the launch's error bits in the low one.  Every block adds
// 1 to the arrivals, block 0 what is missing to 2^31, so their top bit flips
// when the last one arrives and no block resets anything (the arrival scheme
// of cooperative groups' grid barrier); what overflows leaves at the top of
// the word, so the error bits never change by it.  The wait is bounded by
// timeout_ns of %globaltimer; a block whose wait runs out sets its error bit,
// and every block that sees an error leaves at once through the false return
// (the whole block alike).
//
// The word is only ever accessed whole: PTX's memory model gives no order to
// racing accesses that overlap in part, so a release-add on one half would
// not synchronise with a poll of both.
//
// One barrier is a release-add and the polls, which read arrivals and errors
// together.  (With a counter reset and a generation bump by the
// last block, a 32 ns sleep between polls and the error word read by every
// thread after the barrier, it took four dependent L2 round trips more.
// SSSP of 700 K vertices, 46 phases: 1,113 -> 992 us; BFS of 4,999 vertices
// 68.5 -> 59.6 us, of 1 M 146 -> 134; label propagation of 1 M, 26
// iterations: 769 -> 668 us.)
struct GridBar {
  unsigned long long word;
  // code of the launch's error, the lowest of several (host, after the launch)
  unsigned error() const { return (unsigned)__builtin_ffs((int)(unsigned)word); }
};

__device__ __forceinline__ void flag_error(GridBar *bar, unsigned code) {
  atomicOr(&bar->word, 1ull << (code - 1u));
}

// The control block's counters sit in a few cache lines, so a phase must not
// have every warp touch them: thread 0 of each block runs before() ahead of
// its arrival (what the block gathered in shared memory goes out as one
// reduction per counter) and after() behind the wait (counters come in as one
// load each, into shared memory for the block).  With 4,736 warps reading
// two to six counters per phase and adding their own statistics, the one L2
// slice those lines live in took 3 to 10 us of each phase.  Before and after:
// SSSP of 700 K vertices in 46 phases 985 and 668 us, of 20,000 281 and 214;
// BFS of 1 M 140 and 94, of 4,999 65 and 51; label propagation of 1 M 664 and
// 558; 64-source BFS of 262 K 550 and 494.
template <class Before, class After>
__device__ __forceinline__ bool grid_sync(GridBar *bar, unsigned long long timeout_ns, Before before,
                                          After after) {
  __syncthreads();
  unsigned err = 0;
  if (threadIdx.x == 0) {
    before();
    const unsigned nblocks = gridDim.x * gridDim.y * gridDim.z;
    const unsigned add = blockIdx.x + blockIdx.y + blockIdx.z == 0 ? 0x80000000u - (nblocks - 1u) : 1u;
    unsigned long long old;
    // release: the block's writes, ordered before by the block barrier
    asm volatile("atom.add.release.gpu.global.u64 %0, [%1], %2;"
                 : "=l"(old)
                 : "l"(&bar->word), "l"((unsigned long long)add << 32)
                 : "memory");
    const unsigned long long t0 = global_ns();
    for (unsigned spins = 1;; spins++) {
      unsigned long long w;
      asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(&bar->word) : "memory");
      err = (unsigned)w;
      if (err || (long long)(w ^ old) < 0) break;
      if ((spins & 63u) == 0 && global_ns() - t0 > timeout_ns) {
        flag_error(bar, kDevErrBarrier);
        err = kDevErrBarrier;
        break;
      }
    }
    // acquire: the other blocks' writes, for the whole block after its barrier
    asm volatile("fence.acq_rel.gpu;" : : : "memory");
    if (!err) after();
  }
  return __syncthreads_or((int)err) == 0;
}
__device__ __forceinline__ bool grid_sync(GridBar *bar, unsigned long long timeout_ns) {
  return grid_sync(bar, timeout_ns, [] {}, [] {});
}

// A block's share of a launch's statistics and of a phase's counters, in
// shared memory (lane 0 of a warp adds, thread 0 hands them on at a barrier),
// and the counters thread 0 read for the block after it.
struct BlockCounts {
  unsigned long long edges, hbm, link, items;  // whole launch
  unsigned long long keep, extra;              // this phase
  unsigned least, pad;
  unsigned long long ns, nb, nh, rem, other;  // read after the barrier
  unsigned mk, pad2;
};
__device__ __forceinline__ void counts_clear(BlockCounts &b) {  // before a __syncthreads
  if (threadIdx.x == 0) {
    b = BlockCounts{};
    b.least = 0xFFFFFFFFu;
  }
}
// A warp's kept vertices and their least value into the block's.
__device__ __forceinline__ void counts_kept(BlockCounts &b, unsigned long long keep, unsigned least) {
  if (keep) atomicAdd(&b.keep, keep);
  if (least != 0xFFFFFFFFu) atomicMin(&b.least, least);
}
// The block's kept vertices on to the phase's counters (thread 0).
__device__ __forceinline__ void counts_pass_kept(BlockCounts &b, unsigned long long *remaining,
                                                 unsigned *minkept) {
  if (b.keep) atomicAdd(remaining, b.keep);
  if (b.least != 0xFFFFFFFFu) atomicMin(minkept, b.least);
  b.keep = 0;
  b.least = 0xFFFFFFFFu;
}

}  // namespace thv
