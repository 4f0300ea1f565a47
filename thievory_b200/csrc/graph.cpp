// Graph container: loading (converter byte formats), placement plan, C ABI.
//
// Replaces CSR<E> of the reference (src/graph.cuh:11-925):
//   ReadInputFile (:641-815)  -> thv_open: header, offsets, and edges read
//                                straight into pinned, mapped host memory;
//                                errors are returned, never exit().
//   SetPartitionsConfig (:270-304) -> Plan::blocks: greedy split of the vertex
//                                range into edge blocks of <= block_bytes.
//   SetNumStaticEdges (:306-341) -> Plan residency: the caller's HBM budget
//                                (not 90% of free memory), filled up front by
//                                the densest blocks (or the prefix, as the
//                                reference does), instead of an empty region
//                                filled lazily by filter copies.
//   DumpValues (:817-852)     -> thv_write_values: one write per array.
#include <sys/stat.h>

#include <algorithm>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <memory>
#include <numeric>

#include "thv_internal.h"

namespace thv {

static thread_local std::string g_last_error;
static uint32_t g_fail_alloc_after = 0;  // test hook; 0 = off

thv_status fail(thv_status s, const char *fmt, ...) {
  char buf[1024];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  g_last_error = buf;
  return s;
}

bool alloc_should_fail() {
  if (g_fail_alloc_after == 0) return false;
  if (--g_fail_alloc_after == 0) return true;
  return false;
}

thv_status dev_alloc(void **p, size_t bytes, const char *what) {
  *p = nullptr;
  if (alloc_should_fail())
    return fail(THV_ENOMEM, "injected failure allocating %s", what);
  cudaError_t e = cudaMalloc(p, std::max<size_t>(bytes, 16));
  if (e != cudaSuccess) {
    cudaGetLastError();
    *p = nullptr;
    return fail(THV_ENOMEM, "cudaMalloc(%zu) for %s: %s", bytes, what,
                cudaGetErrorString(e));
  }
  return THV_OK;
}

thv_status pinned_alloc(void **p, size_t bytes, const char *what) {
  *p = nullptr;
  if (alloc_should_fail())
    return fail(THV_ENOMEM, "injected failure allocating %s", what);
  cudaError_t e = cudaHostAlloc(p, std::max<size_t>(bytes, 16),
                                cudaHostAllocMapped | cudaHostAllocPortable);
  if (e != cudaSuccess) {
    cudaGetLastError();
    *p = nullptr;
    return fail(THV_ENOMEM, "cudaHostAlloc(%zu) for %s: %s", bytes, what,
                cudaGetErrorString(e));
  }
  return THV_OK;
}

void dev_free(void *p) {
  if (p) cudaFree(p);
}
void pinned_free(void *p) {
  if (p) cudaFreeHost(p);
}

double now_ms() {
  timespec ts;
  clock_gettime(CLOCK_MONOTONIC, &ts);
  return ts.tv_sec * 1e3 + ts.tv_nsec * 1e-6;
}

// ----------------------------------------------------------- device init --

thv_status graph_init_device(thv_graph *g) {
  THV_CUDA(cudaSetDevice(g->device));
  cudaDeviceProp prop;
  THV_CUDA(cudaGetDeviceProperties(&prop, g->device));
  g->num_sms = prop.multiProcessorCount;
  if (!prop.cooperativeLaunch)
    return fail(THV_EUNSUPPORTED, "device %d lacks cooperative launch", g->device);
  THV_CUDA(cudaStreamCreateWithFlags(&g->stream, cudaStreamNonBlocking));
  THV_TRY(dev_alloc((void **)&g->d_off, (g->nv + 1) * 8 + 64, "offsets"));
  THV_CUDA(cudaMemcpy(g->d_off, g->off.data(), (g->nv + 1) * 8,
                      cudaMemcpyHostToDevice));
  g->device_bytes += (g->nv + 1) * 8;
  if (g->fmt == THV_FMT_CSC) {
    THV_TRY(dev_alloc((void **)&g->d_outdeg, g->nv * 4 + 64, "out-degrees"));
    THV_CUDA(cudaMemcpy(g->d_outdeg, g->outdeg.data(), g->nv * 4,
                        cudaMemcpyHostToDevice));
    g->device_bytes += g->nv * 4;
  }
  void *dp = nullptr;
  THV_CUDA(cudaHostGetDevicePointer(&dp, g->h_edges, 0));
  g->h_edges_dev = (uint64_t)dp;
  return THV_OK;
}

static void graph_destroy(thv_graph *g) {
  if (!g) return;
  cudaSetDevice(g->device);
  if (g->stream) cudaStreamSynchronize(g->stream);
  batch_free(g);
  minprop_free(g);
  pagerank_free(g);
  transpose_free(g);
  plan_free(g);
  dev_free(g->d_off);
  dev_free(g->d_outdeg);
  pinned_free(g->h_edges);
  if (g->stream) cudaStreamDestroy(g->stream);
  delete g;
}

// Validate offsets / ids so a malformed file is an error, not a fault.
static thv_status validate(thv_graph *g) {
  const uint64_t nv = g->nv, ne = g->ne;
  if (nv && g->off[0] != 0) return fail(THV_EFORMAT, "offset[0] = %llu, expected 0",
                                        (unsigned long long)g->off[0]);
  for (uint64_t v = 0; v < nv; v++)
    if (g->off[v] > g->off[v + 1])
      return fail(THV_EFORMAT, "offsets decrease at vertex %llu", (unsigned long long)v);
  const uint32_t stride = g->esz / 4;
  const uint32_t *e = (const uint32_t *)g->h_edges;
  int64_t bad_at = -1;
#pragma omp parallel for schedule(static) reduction(max : bad_at)
  for (int64_t i = 0; i < (int64_t)ne; i++)
    if (e[(uint64_t)i * stride] >= nv) bad_at = std::max<int64_t>(bad_at, i);
  if (bad_at >= 0)
    return fail(THV_EFORMAT, "edge %lld has neighbour id >= n=%llu",
                (long long)bad_at, (unsigned long long)nv);
  // sorted lists (the converter's order) allow reading only part of a list
  int64_t unsorted = 0;
#pragma omp parallel for schedule(dynamic, 4096) reduction(+ : unsorted)
  for (int64_t v = 0; v < (int64_t)nv; v++)
    for (uint64_t i = g->off[v] + 1; i < g->off[v + 1]; i++)
      unsorted += e[i * stride] < e[(i - 1) * stride];
  g->sorted = unsorted == 0;
  return THV_OK;
}

static uint32_t bit_width(uint32_t x) { return x ? 32u - (uint32_t)__builtin_clz(x) : 0u; }

// Weighted edges are stored in 4 bytes, dst << wshift | (w - wbase), when
// the id bits and the bits of the weight range fit 32 (lossless); the
// {dst, w} pairs are restored for save and the host view.
thv_status set_packing(thv_graph *g, bool on) {
  if (!g->weighted || on == g->packed) return THV_OK;
  THV_CUDA(cudaSetDevice(g->device));
  if (g->stream) THV_CUDA(cudaStreamSynchronize(g->stream));
  batch_free(g);
  minprop_free(g);
  pagerank_free(g);
  plan_free(g);
  const uint64_t ne = g->ne;
  const uint32_t *e = (const uint32_t *)g->h_edges;
  void *nb = nullptr;
  if (on) {
    uint32_t wmin = 0xFFFFFFFFu, wmax = 0;
    uint64_t wsum = 0;  // of weights cut off at 2^22, which no window exceeds
#pragma omp parallel for schedule(static) reduction(min : wmin) reduction(max : wmax) reduction(+ : wsum)
    for (int64_t i = 0; i < (int64_t)ne; i++) {
      wmin = std::min(wmin, e[2 * i + 1]);
      wmax = std::max(wmax, e[2 * i + 1]);
      wsum += std::min(e[2 * i + 1], 1u << 22);
    }
    if (!ne) wmin = wmax = 0;
    g->wtyp = ne ? (uint32_t)std::min<uint64_t>(wmax, (2 * wsum + ne - 1) / ne) : 0;
    const uint32_t ib = bit_width(g->nv ? (uint32_t)(g->nv - 1) : 0u);
    const uint32_t wb = bit_width(wmax - wmin);
    if (wb >= 32 || ib + wb > 32) return THV_OK;  // does not fit: keep pairs
    const size_t bytes = ne * 4 + kEdgePad;
    THV_TRY(pinned_alloc(&nb, bytes, "pinned packed edges"));
    uint32_t *p = (uint32_t *)nb;
#pragma omp parallel for schedule(static)
    for (int64_t i = 0; i < (int64_t)ne; i++) p[i] = (e[2 * i] << wb) | (e[2 * i + 1] - wmin);
    memset(p + ne, 0, kEdgePad);
    g->esz = 4;
    g->wshift = wb;
    g->wbase = wmin;
    g->h_edges_bytes = bytes;
  } else {
    const size_t bytes = ne * 8 + kEdgePad;
    THV_TRY(pinned_alloc(&nb, bytes, "pinned edges"));
    uint32_t *p = (uint32_t *)nb;
    const uint32_t wb = g->wshift, base = g->wbase, mask = (1u << wb) - 1u;
#pragma omp parallel for schedule(static)
    for (int64_t i = 0; i < (int64_t)ne; i++) {
      p[2 * i] = e[i] >> wb;
      p[2 * i + 1] = (e[i] & mask) + base;
    }
    memset(p + 2 * ne, 0, kEdgePad);
    g->esz = 8;
    g->wshift = g->wbase = 0;
    g->h_edges_bytes = bytes;
  }
  pinned_free(g->h_edges);
  g->h_edges = nb;
  g->packed = on;
  g->h_unpacked.clear();
  g->h_unpacked.shrink_to_fit();
  void *dp = nullptr;
  THV_CUDA(cudaHostGetDevicePointer(&dp, g->h_edges, 0));
  g->h_edges_dev = (uint64_t)dp;
  return THV_OK;
}

// {dst, w} of edge i whatever the in-memory layout.
static inline void edge_at(const thv_graph *g, uint64_t i, uint32_t *dst, uint32_t *w) {
  const uint32_t *e = (const uint32_t *)g->h_edges;
  if (g->packed) {
    *dst = e[i] >> g->wshift;
    *w = (e[i] & ((1u << g->wshift) - 1u)) + g->wbase;
  } else if (g->esz == 8) {
    *dst = e[2 * i];
    *w = e[2 * i + 1];
  } else {
    *dst = e[i];
    *w = 20u;  // converter.cpp writes weight 20 for unweighted inputs
  }
}

static thv_status alloc_host_edges(thv_graph *g) {
  g->h_edges_bytes = g->ne * g->esz + kEdgePad;
  THV_TRY(pinned_alloc(&g->h_edges, g->h_edges_bytes, "pinned edges"));
  memset((char *)g->h_edges + g->ne * g->esz, 0, kEdgePad);
  return THV_OK;
}

struct FileCloser {
  void operator()(FILE *f) const { if (f) fclose(f); }
};

static thv_status open_file(const char *path, thv_format fmt, uint32_t flags,
                            int device, thv_graph **out) {
  if (!path || !out) return fail(THV_EINVAL, "null argument");
  std::unique_ptr<FILE, FileCloser> f(fopen(path, "rb"));
  if (!f) return fail(THV_EIO, "cannot open %s: %s", path, strerror(errno));
  struct stat st;
  if (fstat(fileno(f.get()), &st) != 0) return fail(THV_EIO, "cannot stat %s", path);
  const uint64_t size = (uint64_t)st.st_size;
  uint64_t hdr[2];
  if (fread(hdr, 8, 2, f.get()) != 2)
    return fail(THV_EFORMAT, "%s: truncated header", path);
  const uint64_t nv = hdr[0], ne = hdr[1];
  const bool want_w = fmt == THV_FMT_WCSR || (fmt == THV_FMT_CSR && (flags & THV_OPEN_WEIGHTS));
  // bytes needed after the header
  __uint128_t need = (__uint128_t)nv * 8;
  if (fmt == THV_FMT_WCSR) need += (__uint128_t)ne * 8;
  else need += (__uint128_t)ne * 4;
  if (fmt == THV_FMT_CSR && want_w) need += (__uint128_t)ne * 4;
  if (fmt == THV_FMT_CSC) need += (__uint128_t)nv * 4;
  if (need + 16 > size)
    return fail(THV_EFORMAT, "%s: file has %llu bytes, header (n=%llu, m=%llu) "
                "needs %llu", path, (unsigned long long)size,
                (unsigned long long)nv, (unsigned long long)ne,
                (unsigned long long)(need + 16));
  if (nv >= 0xFFFFFFFFull) return fail(THV_EUNSUPPORTED, "n=%llu too large", (unsigned long long)nv);

  std::unique_ptr<thv_graph, void (*)(thv_graph *)> g(new thv_graph(), graph_destroy);
  g->nv = nv;
  g->ne = ne;
  g->fmt = fmt;
  g->device = device;
  g->weighted = want_w;
  g->esz = want_w ? 8 : 4;
  g->off.resize(nv + 1);
  if (nv && fread(g->off.data(), 8, nv, f.get()) != nv)
    return fail(THV_EFORMAT, "%s: truncated offsets", path);
  g->off[nv] = ne;  // the file has no trailing entry (src/graph.cuh:731)
  THV_TRY(alloc_host_edges(g.get()));
  if (fmt == THV_FMT_WCSR) {
    if (ne && fread(g->h_edges, 8, ne, f.get()) != ne)
      return fail(THV_EFORMAT, "%s: truncated edges", path);
  } else if (want_w) {  // CSR + trailing weights -> interleaved {dst, w}
    std::vector<uint32_t> tmp(std::min<uint64_t>(ne, 1ull << 24));
    uint32_t *e = (uint32_t *)g->h_edges;
    for (uint64_t i = 0; i < ne;) {
      const uint64_t k = std::min<uint64_t>(tmp.size(), ne - i);
      if (fread(tmp.data(), 4, k, f.get()) != k)
        return fail(THV_EFORMAT, "%s: truncated edges", path);
      for (uint64_t j = 0; j < k; j++) e[2 * (i + j)] = tmp[j];
      i += k;
    }
    for (uint64_t i = 0; i < ne;) {
      const uint64_t k = std::min<uint64_t>(tmp.size(), ne - i);
      if (fread(tmp.data(), 4, k, f.get()) != k)
        return fail(THV_EFORMAT, "%s: truncated weights", path);
      for (uint64_t j = 0; j < k; j++) e[2 * (i + j) + 1] = tmp[j];
      i += k;
    }
  } else {
    if (ne && fread(g->h_edges, 4, ne, f.get()) != ne)
      return fail(THV_EFORMAT, "%s: truncated edges", path);
  }
  if (fmt == THV_FMT_CSC) {
    g->outdeg.resize(nv);
    if (nv && fread(g->outdeg.data(), 4, nv, f.get()) != nv)
      return fail(THV_EFORMAT, "%s: truncated out-degrees", path);
  }
  THV_TRY(validate(g.get()));
  THV_TRY(graph_init_device(g.get()));
  THV_TRY(set_packing(g.get(), true));
  *out = g.release();
  return THV_OK;
}

// ------------------------------------------------------------------ plan --

// Access bytes of old blocks [ovb[i], ovb[i+1]) spread over new blocks by
// vertex overlap.
static std::vector<uint64_t> spread_access(const std::vector<uint32_t> &ovb,
                                           const std::vector<uint64_t> &ob,
                                           const std::vector<uint32_t> &nvb) {
  std::vector<uint64_t> out(nvb.empty() ? 0 : nvb.size() - 1, 0);
  size_t j = 0;
  for (size_t i = 0; i < ob.size(); i++) {
    const uint64_t a = ovb[i], b = ovb[i + 1];
    if (b <= a || !ob[i]) continue;
    while (j + 1 < nvb.size() && nvb[j + 1] <= a) j++;
    for (size_t k = j; k + 1 < nvb.size() && nvb[k] < b; k++) {
      const uint64_t lo = std::max<uint64_t>(a, nvb[k]), hi = std::min<uint64_t>(b, nvb[k + 1]);
      if (hi > lo) out[k] += (uint64_t)((__uint128_t)ob[i] * (hi - lo) / (b - a));
    }
  }
  return out;
}

// Folds the counters of a tracked plan into the graph's access history.
static void fold_access(thv_graph *g) {
  Plan &p = g->plan;
  if (!p.d_access || p.blocks.empty()) return;
  std::vector<uint64_t> cur(p.blocks.size(), 0);
  if (cudaMemcpy(cur.data(), p.d_access, cur.size() * 8, cudaMemcpyDeviceToHost) != cudaSuccess) {
    cudaGetLastError();
    return;
  }
  std::vector<uint32_t> vb(p.vbegin.begin(), p.vbegin.end());
  if (!g->access_bytes.empty()) {
    const std::vector<uint64_t> old = spread_access(g->access_vb, g->access_bytes, vb);
    for (size_t i = 0; i < cur.size(); i++) cur[i] += old[i];
  }
  g->access_vb = vb;
  g->access_bytes = cur;
}

void plan_free(thv_graph *g) {
  Plan &p = g->plan;
  fold_access(g);
  dev_free(p.d_access);
  dev_free(p.d_resident);
  dev_free(p.d_lists);
  dev_free(p.d_list_idx);
  dev_free(p.d_vbegin);
  dev_free(p.d_base);
  for (PrTiles &t : p.tiles) {
    dev_free(t.d_tiles);
    dev_free(t.d_split_parts);
  }
  p = Plan();
}

// Packs the lists with 0 < deg < ldeg of every host block into d_lists, in
// vertex order, through a pinned staging buffer.
static thv_status build_list_cache(thv_graph *g, uint32_t ldeg) {
  Plan &p = g->plan;
  p.list_deg = ldeg;
  if (!ldeg) return THV_OK;
  const uint64_t esz = g->esz;
  std::vector<uint32_t> idx(g->nv, 0);
  uint64_t cursor = 0, verts = 0;
  for (const Block &b : p.blocks) {
    if (b.resident) continue;
    for (uint64_t v = b.vbegin; v < b.vend; v++) {
      const uint64_t d = g->off[v + 1] - g->off[v];
      if (d > 0 && d < ldeg) {
        idx[v] = (uint32_t)cursor;
        cursor += d;
        verts++;
      }
    }
  }
  p.list_bytes = cursor * esz;
  p.list_vertices = verts;
  if (!cursor) {
    p.list_deg = 0;
    return THV_OK;
  }
  p.d_lists_bytes = kListLead + cursor * esz + kEdgePad;
  THV_TRY(dev_alloc((void **)&p.d_lists, p.d_lists_bytes, "small-list cache"));
  THV_TRY(dev_alloc((void **)&p.d_list_idx, g->nv * 4, "small-list index"));
  THV_CUDA(cudaMemset(p.d_lists, 0, p.d_lists_bytes));
  THV_CUDA(cudaMemcpy(p.d_list_idx, idx.data(), g->nv * 4, cudaMemcpyHostToDevice));
  // stage vertex ranges of at most kStage bytes; lists are copied in parallel
  constexpr uint64_t kStage = 64ull << 20;
  char *stage = nullptr;
  THV_TRY(pinned_alloc((void **)&stage, kStage, "list staging"));
  std::vector<uint32_t> vs;  // cached vertices in cache order
  vs.reserve(verts);
  for (const Block &b : p.blocks) {
    if (b.resident) continue;
    for (uint64_t v = b.vbegin; v < b.vend; v++) {
      const uint64_t d = g->off[v + 1] - g->off[v];
      if (d > 0 && d < ldeg) vs.push_back((uint32_t)v);
    }
  }
  thv_status st = THV_OK;
  const char *src = (const char *)g->h_edges;
  for (size_t i = 0; i < vs.size() && st == THV_OK;) {
    const uint64_t e0 = idx[vs[i]];
    size_t j = i;
    while (j < vs.size() && (idx[vs[j]] - e0 + (g->off[vs[j] + 1] - g->off[vs[j]])) * esz <= kStage)
      j++;
#pragma omp parallel for schedule(static, 4096)
    for (size_t k = i; k < j; k++) {
      const uint32_t v = vs[k];
      memcpy(stage + (idx[v] - e0) * esz, src + g->off[v] * esz,
             (g->off[v + 1] - g->off[v]) * esz);
    }
    const uint64_t last = vs[j - 1];
    const uint64_t bytes = (idx[last] - e0 + (g->off[last + 1] - g->off[last])) * esz;
    if (cudaMemcpy(p.d_lists + kListLead + e0 * esz, stage, bytes, cudaMemcpyHostToDevice) !=
        cudaSuccess)
      st = fail(THV_ECUDA, "small-list cache copy failed");
    i = j;
  }
  pinned_free(stage);
  return st;
}

// force: an explicit resident flag per block (a loaded plan), or null.
static thv_status do_plan(thv_graph *g, const thv_plan_opts *o,
                          const std::vector<uint8_t> *force = nullptr) {
  THV_CUDA(cudaSetDevice(g->device));
  if (g->stream) THV_CUDA(cudaStreamSynchronize(g->stream));
  batch_free(g);  // its captured launch graphs hold the old plan's tables
  plan_free(g);
  Plan &p = g->plan;
  const uint64_t esz = g->esz;
  p.block_bytes = o && o->block_bytes ? o->block_bytes : kDefaultBlockBytes;
  p.policy = o ? o->policy : THV_PLACE_DENSEST;
  p.flags = o ? o->flags : 0;
  if (p.policy > THV_PLACE_ACCESS) return fail(THV_EINVAL, "unknown placement policy %u", p.policy);
  const uint64_t max_edges = std::max<uint64_t>(1, p.block_bytes / esz);
  // blocks on vertex boundaries (src/graph.cuh:270-304)
  uint32_t begin = 0;
  uint64_t cur = 0;
  for (uint64_t v = 0; v < g->nv; v++) {
    const uint64_t d = g->off[v + 1] - g->off[v];
    if (cur + d <= max_edges || v == begin) {
      cur += d;
    } else {
      p.blocks.push_back(Block{begin, (uint32_t)v, g->off[begin], g->off[v], false, 0});
      begin = (uint32_t)v;
      cur = d;
    }
  }
  p.blocks.push_back(Block{begin, (uint32_t)g->nv, g->off[begin], g->off[g->nv], false, 0});
  const uint64_t total = g->ne * esz;
  uint64_t budget = o ? o->hbm_budget_bytes : UINT64_MAX;
  if (budget == UINT64_MAX) {
    size_t fr = 0, tot = 0;
    THV_CUDA(cudaMemGetInfo(&fr, &tot));
    const uint64_t reserve = 96ull * g->nv + g->ne + (2ull << 30);
    budget = fr > reserve ? std::min<uint64_t>(total, fr - reserve) : 0;
  }
  p.budget_bytes = budget;
  // Small-list cache threshold: the largest t <= the requested one whose
  // lists (0 < deg < t) fit the budget and 2^32 cached elements.
  uint32_t ldeg = o && o->small_list_degree ? o->small_list_degree
                                            : (g->fmt == THV_FMT_CSC ? 1u : kDefaultListDeg);
  ldeg = (uint32_t)std::min<uint64_t>(ldeg, g->nv + 1);
  if (ldeg > 1) {
    std::vector<uint64_t> by_deg(ldeg, 0);  // edges in lists of each degree
    for (uint64_t v = 0; v < g->nv; v++) {
      const uint64_t d = g->off[v + 1] - g->off[v];
      if (d > 0 && d < ldeg) by_deg[d] += d;
    }
    uint64_t acc = 0;
    uint32_t t = 1;
    while (t < ldeg && (acc + by_deg[t]) * esz <= budget && acc + by_deg[t] < (1ull << 32)) {
      acc += by_deg[t];
      t++;
    }
    ldeg = t;
  }
  if (ldeg <= 1) ldeg = 0;
  // per-block bytes of small lists; a resident block needs none of them cached
  std::vector<uint64_t> small_b(p.blocks.size(), 0);
  uint64_t small_total = 0;
  if (ldeg) {
    for (size_t b = 0; b < p.blocks.size(); b++) {
      uint64_t s = 0;
      for (uint64_t v = p.blocks[b].vbegin; v < p.blocks[b].vend; v++) {
        const uint64_t d = g->off[v + 1] - g->off[v];
        if (d > 0 && d < ldeg) s += d;
      }
      small_b[b] = s * esz;
      small_total += s * esz;
    }
  }
  std::vector<uint32_t> order(p.blocks.size());
  std::iota(order.begin(), order.end(), 0u);
  auto denser = [&](uint32_t x, uint32_t y) {
    const Block &a = p.blocks[x], &b = p.blocks[y];
    // edges per vertex, compared without division
    const __uint128_t l = (__uint128_t)(a.eend - a.ebegin) * std::max<uint64_t>(1, b.vend - b.vbegin);
    const __uint128_t r = (__uint128_t)(b.eend - b.ebegin) * std::max<uint64_t>(1, a.vend - a.vbegin);
    return l > r;
  };
  if (p.policy == THV_PLACE_DENSEST) {
    std::stable_sort(order.begin(), order.end(), denser);
  } else if (p.policy == THV_PLACE_ACCESS) {
    // most adjacency bytes read per byte of HBM the block would take (its
    // long lists)
    std::vector<uint32_t> vb(p.blocks.size() + 1);
    for (size_t b = 0; b < p.blocks.size(); b++) vb[b] = p.blocks[b].vbegin;
    vb[p.blocks.size()] = (uint32_t)g->nv;
    const std::vector<uint64_t> hot =
        g->access_bytes.empty() ? std::vector<uint64_t>(p.blocks.size(), 0)
                                : spread_access(g->access_vb, g->access_bytes, vb);
    std::stable_sort(order.begin(), order.end(), [&](uint32_t x, uint32_t y) {
      const uint64_t cx = std::max<uint64_t>(1, (p.blocks[x].eend - p.blocks[x].ebegin) * esz - small_b[x]);
      const uint64_t cy = std::max<uint64_t>(1, (p.blocks[y].eend - p.blocks[y].ebegin) * esz - small_b[y]);
      const __uint128_t l = (__uint128_t)hot[x] * cy, r = (__uint128_t)hot[y] * cx;
      if (l != r) return l > r;
      return denser(x, y);
    });
  }
  // the cache is paid first; a block then costs only its long lists
  uint64_t used = small_total;
  if (force) {
    if (force->size() != p.blocks.size()) return fail(THV_EINVAL, "plan has a different block split");
    for (size_t b = 0; b < p.blocks.size(); b++) {
      if (!(*force)[b]) continue;
      p.blocks[b].resident = true;
      used += (p.blocks[b].eend - p.blocks[b].ebegin) * esz - small_b[b];
    }
    if (used > budget) return fail(THV_EINVAL, "loaded plan exceeds its budget");
  } else {
    for (uint32_t b : order) {
      const uint64_t bytes = (p.blocks[b].eend - p.blocks[b].ebegin) * esz;
      if (bytes == 0) continue;
      const uint64_t cost = bytes - small_b[b];
      if (used + cost <= budget) {
        p.blocks[b].resident = true;
        used += cost;
      } else if (p.policy == THV_PLACE_PREFIX) {
        break;
      }
    }
  }
  // pack resident blocks; element offsets keep the edge index's position
  // inside a 128-byte line so aligned loads stay aligned in HBM
  const uint64_t A = 128 / esz;
  uint64_t cursor = 0;
  for (Block &b : p.blocks) {
    if (!b.resident) continue;
    const uint64_t d = (cursor + A - 1) / A * A + (b.ebegin % A);
    b.dev_elem = d;
    cursor = d + (b.eend - b.ebegin);
  }
  p.d_resident_bytes = cursor * esz + kEdgePad;
  if (used) {
    THV_TRY(dev_alloc((void **)&p.d_resident, p.d_resident_bytes, "resident edge blocks"));
    for (const Block &b : p.blocks) {
      if (!b.resident) continue;
      THV_CUDA(cudaMemcpy(p.d_resident + b.dev_elem * esz,
                          (char *)g->h_edges + b.ebegin * esz,
                          (b.eend - b.ebegin) * esz, cudaMemcpyHostToDevice));
    }
  }
  THV_TRY(build_list_cache(g, ldeg));
  p.resident_edge_bytes = used;
  p.host_edge_bytes = total - used;
  const size_t nb = p.blocks.size();
  p.vbegin.resize(nb + 1);
  p.base.resize(nb);
  for (size_t i = 0; i < nb; i++) {
    const Block &b = p.blocks[i];
    p.vbegin[i] = b.vbegin;
    p.base[i] = b.resident ? (uint64_t)p.d_resident + b.dev_elem * esz - b.ebegin * esz
                           : g->h_edges_dev;
  }
  p.vbegin[nb] = (uint32_t)g->nv;
  THV_TRY(dev_alloc((void **)&p.d_vbegin, (nb + 1) * 4, "block table"));
  THV_TRY(dev_alloc((void **)&p.d_base, nb * 8, "block table"));
  THV_CUDA(cudaMemcpy(p.d_vbegin, p.vbegin.data(), (nb + 1) * 4, cudaMemcpyHostToDevice));
  THV_CUDA(cudaMemcpy(p.d_base, p.base.data(), nb * 8, cudaMemcpyHostToDevice));
  if (p.flags & THV_PLAN_TRACK_ACCESS) {
    THV_TRY(dev_alloc((void **)&p.d_access, nb * 8, "block access counters"));
    THV_CUDA(cudaMemset(p.d_access, 0, nb * 8));
  }
  p.valid = true;
  return THV_OK;
}

// Re-places blocks by the measured access with the current plan's budget,
// block size, small-list threshold and flags.
thv_status replan_by_access(thv_graph *g) {
  if (!g->plan.valid) return THV_OK;
  thv_plan_opts o{};
  o.hbm_budget_bytes = g->plan.budget_bytes;
  o.block_bytes = g->plan.block_bytes;
  o.policy = THV_PLACE_ACCESS;
  o.small_list_degree = g->plan.list_deg ? g->plan.list_deg : 1u;
  o.flags = g->plan.flags;
  return do_plan(g, &o);
}

// ---- plan files: magic, sizes, options, block split, resident set, access
static constexpr char kPlanMagic[8] = {'T', 'H', 'V', 'P', 'L', 'A', 'N', '1'};

static thv_status save_plan(const thv_graph *g, const char *path) {
  const Plan &p = g->plan;
  if (!p.valid) return fail(THV_EINVAL, "graph has no plan yet");
  std::vector<uint64_t> acc(p.blocks.size(), 0);
  if (p.d_access)
    THV_CUDA(cudaMemcpy(acc.data(), p.d_access, acc.size() * 8, cudaMemcpyDeviceToHost));
  if (!g->access_bytes.empty()) {
    std::vector<uint32_t> vb(p.vbegin.begin(), p.vbegin.end());
    const std::vector<uint64_t> old = spread_access(g->access_vb, g->access_bytes, vb);
    for (size_t i = 0; i < acc.size(); i++) acc[i] += old[i];
  }
  std::unique_ptr<FILE, FileCloser> f(fopen(path, "wb"));
  if (!f) return fail(THV_EIO, "cannot create %s: %s", path, strerror(errno));
  const uint64_t hdr[8] = {g->nv, g->ne, g->esz, p.block_bytes, p.budget_bytes,
                           p.list_deg ? p.list_deg : 1u, p.flags, p.blocks.size()};
  std::vector<uint8_t> res(p.blocks.size());
  for (size_t i = 0; i < res.size(); i++) res[i] = p.blocks[i].resident ? 1 : 0;
  bool ok = fwrite(kPlanMagic, 1, 8, f.get()) == 8 && fwrite(hdr, 8, 8, f.get()) == 8 &&
            fwrite(p.vbegin.data(), 4, p.vbegin.size(), f.get()) == p.vbegin.size() &&
            fwrite(res.data(), 1, res.size(), f.get()) == res.size() &&
            fwrite(acc.data(), 8, acc.size(), f.get()) == acc.size();
  if (!ok) return fail(THV_EIO, "write to %s failed", path);
  return THV_OK;
}

static thv_status load_plan(thv_graph *g, const char *path) {
  std::unique_ptr<FILE, FileCloser> f(fopen(path, "rb"));
  if (!f) return fail(THV_EIO, "cannot open %s: %s", path, strerror(errno));
  char magic[8];
  uint64_t hdr[8];
  if (fread(magic, 1, 8, f.get()) != 8 || memcmp(magic, kPlanMagic, 8) != 0 ||
      fread(hdr, 8, 8, f.get()) != 8)
    return fail(THV_EFORMAT, "%s: not a plan file", path);
  if (hdr[0] != g->nv || hdr[1] != g->ne || hdr[2] != g->esz)
    return fail(THV_EINVAL, "%s: plan of another graph (n=%llu m=%llu edge size %llu)", path,
                (unsigned long long)hdr[0], (unsigned long long)hdr[1],
                (unsigned long long)hdr[2]);
  const uint64_t nb = hdr[7];
  if (nb == 0 || nb > g->nv + 1) return fail(THV_EFORMAT, "%s: bad block count", path);
  std::vector<uint32_t> vb(nb + 1);
  std::vector<uint8_t> res(nb);
  std::vector<uint64_t> acc(nb);
  if (fread(vb.data(), 4, nb + 1, f.get()) != nb + 1 || fread(res.data(), 1, nb, f.get()) != nb ||
      fread(acc.data(), 8, nb, f.get()) != nb)
    return fail(THV_EFORMAT, "%s: truncated plan", path);
  thv_plan_opts o{};
  o.block_bytes = hdr[3];
  o.hbm_budget_bytes = hdr[4];
  o.small_list_degree = (uint32_t)hdr[5];
  o.flags = (uint32_t)hdr[6];
  o.policy = THV_PLACE_DENSEST;
  THV_TRY(do_plan(g, &o, &res));
  if (g->plan.vbegin != vb) return fail(THV_EINVAL, "%s: block split differs from this graph's", path);
  g->access_vb = vb;
  g->access_bytes = acc;
  return THV_OK;
}

thv_status ensure_plan(thv_graph *g) {
  if (g->plan.valid) return THV_OK;
  return do_plan(g, nullptr);
}

static uint64_t mix64_host(uint64_t x) {
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}

// Whether every edge has its reverse, as often as it occurs itself: the sum
// of hash(u, w) - hash(w, u) over all edges is zero mod 2^64 then, and
// otherwise but for one case in 2^64.  One pass, once per graph (62 M edges:
// about 12 ms on 16 cores, beside 150 ms to open the graph).
bool edges_mirrored(const thv_graph *g) {
  const uint32_t *e = (const uint32_t *)g->h_edges;
  const uint32_t step = g->esz / 4, shift = g->packed ? g->wshift : 0;
  uint64_t sum = 0;
#pragma omp parallel for schedule(dynamic, 4096) reduction(+ : sum)
  for (int64_t v = 0; v < (int64_t)g->nv; v++)
    for (uint64_t i = g->off[v]; i < g->off[v + 1]; i++) {
      const uint64_t w = e[step * i] >> shift;
      sum += mix64_host((uint64_t)v << 32 | w) - mix64_host(w << 32 | (uint64_t)v);
    }
  return sum == 0;
}

// hub_reach is estimated from up to kReachSample evenly spaced neighbours (a
// few random reads per thread; hubs of RMAT graphs have up to a million).
constexpr uint64_t kReachSample = 16384;

}  // namespace thv

uint32_t thv_graph::hub_vertex() {
  if (hub >= 0) return (uint32_t)hub;
  hub = 0;
  for (uint64_t v = 1; v < nv; v++)
    if (off[v + 1] - off[v] > off[hub + 1] - off[hub]) hub = (int64_t)v;
  const uint64_t deg = off[hub + 1] - off[hub];
  const uint64_t n = std::min(deg, thv::kReachSample);
  const uint32_t *e = (const uint32_t *)h_edges;
  const uint32_t step = esz / 4, shift = packed ? wshift : 0;
  uint64_t sum = 0;
#pragma omp parallel for schedule(static) reduction(+ : sum)
  for (int64_t i = 0; i < (int64_t)n; i++) {
    const uint64_t w = e[step * (off[hub] + (uint64_t)i * deg / n)] >> shift;
    sum += off[w + 1] - off[w];
  }
  if (n) hub_reach = (double)sum / (double)n * (double)deg / (double)ne;
  return (uint32_t)hub;
}

namespace thv {

// PageRank tiles within the bounds of kTileShape[kind], never crossing a
// block; a vertex of more than split_deg edges is cut into parts of at most
// part_edges edges whose partial sums are combined atomically.
thv_status build_tiles(thv_graph *g, PrTileKind kind) {
  const Plan &plan = g->plan;
  const PrTileShape &sh = kTileShape[kind];
  PrTiles &p = g->plan.tiles[kind];
  if (p.valid) return THV_OK;
  p.tiles.clear();
  p.split_parts.clear();
  for (uint32_t bi = 0; bi < plan.blocks.size(); bi++) {
    const Block &b = plan.blocks[bi];
    uint32_t start = b.vbegin;
    uint64_t edges = 0;
    auto close = [&](uint32_t end) {
      if (end > start)
        p.tiles.push_back(PrTile{g->off[start], g->off[end], start, end, bi, 0});
    };
    for (uint32_t v = b.vbegin; v < b.vend; v++) {
      const uint64_t d = g->off[v + 1] - g->off[v];
      if (d > sh.split_deg) {
        close(v);
        const uint32_t parts = (uint32_t)((d + sh.part_edges - 1) / sh.part_edges);
        const uint32_t sidx = (uint32_t)p.split_parts.size();
        p.split_parts.push_back(parts);
        for (uint32_t k = 0; k < parts; k++) {
          const uint64_t e0 = g->off[v] + (uint64_t)k * sh.part_edges;
          const uint64_t e1 = std::min<uint64_t>(g->off[v + 1], e0 + sh.part_edges);
          p.tiles.push_back(PrTile{e0, e1, v, v + 1, bi, sidx + 1});
        }
        start = v + 1;
        edges = 0;
      } else if (edges + d > sh.edges || v - start >= sh.verts) {
        close(v);
        start = v;
        edges = d;
      } else {
        edges += d;
      }
    }
    close(b.vend);
  }
  // Interleave host-block and HBM-block tiles in proportion to their edges.
  // Tiles are taken in this order, drawn or a round at a time, so the host
  // link stays busy for the whole iteration while the HBM tiles are done
  // beside it; in block order the GPU would work through host blocks with HBM idle, then
  // HBM blocks with the link idle.  Results do not depend on the order.
  {
    std::vector<PrTile> host, hbm;
    uint64_t eh = 0, er = 0;
    for (const PrTile &t : p.tiles) {
      if (plan.blocks[t.block].resident) { hbm.push_back(t); er += t.eend - t.ebegin; }
      else { host.push_back(t); eh += t.eend - t.ebegin; }
    }
    size_t i = 0, j = 0;
    uint64_t dh = 0, dr = 0;
    p.tiles.clear();
    while (i < host.size() || j < hbm.size()) {
      // take from the side that is behind its share (dh / eh vs dr / er)
      const bool take_host =
          j == hbm.size() || (i < host.size() && (unsigned __int128)dh * er <= (unsigned __int128)dr * eh);
      const PrTile &t = take_host ? host[i++] : hbm[j++];
      (take_host ? dh : dr) += t.eend - t.ebegin;
      p.tiles.push_back(t);
    }
  }
  THV_TRY(dev_alloc((void **)&p.d_tiles, std::max<size_t>(1, p.tiles.size()) * sizeof(PrTile), "tiles"));
  THV_TRY(dev_alloc((void **)&p.d_split_parts, std::max<size_t>(1, p.split_parts.size()) * 4, "split table"));
  if (!p.tiles.empty())
    THV_CUDA(cudaMemcpy(p.d_tiles, p.tiles.data(), p.tiles.size() * sizeof(PrTile),
                        cudaMemcpyHostToDevice));
  if (!p.split_parts.empty())
    THV_CUDA(cudaMemcpy(p.d_split_parts, p.split_parts.data(), p.split_parts.size() * 4,
                        cudaMemcpyHostToDevice));
  p.valid = true;
  return THV_OK;
}

static thv_status from_arrays(uint64_t nv, uint64_t ne, const uint64_t *off,
                              const void *edges, uint32_t esz, thv_format fmt,
                              const uint32_t *outdeg, int device,
                              thv_graph **out) {
  if (!out || (!off && nv) || (!edges && ne)) return fail(THV_EINVAL, "null argument");
  if (esz != 4 && esz != 8) return fail(THV_EINVAL, "edge size must be 4 or 8");
  if (fmt == THV_FMT_CSC && (!outdeg || esz != 4))
    return fail(THV_EINVAL, "CSC needs 4-byte ids and out-degrees");
  if (fmt == THV_FMT_WCSR && esz != 8) return fail(THV_EINVAL, "WCSR needs 8-byte edges");
  if (nv >= 0xFFFFFFFFull) return fail(THV_EUNSUPPORTED, "n too large");
  if (nv && off[nv] != ne) return fail(THV_EFORMAT, "off[n] != m");
  std::unique_ptr<thv_graph, void (*)(thv_graph *)> g(new thv_graph(), graph_destroy);
  g->nv = nv;
  g->ne = ne;
  g->fmt = fmt;
  g->esz = esz;
  g->weighted = esz == 8;
  g->device = device;
  g->off.assign(off, off + nv + 1);
  if (!nv) g->off.assign(1, 0);
  THV_TRY(alloc_host_edges(g.get()));
  if (ne) memcpy(g->h_edges, edges, ne * esz);
  if (fmt == THV_FMT_CSC) g->outdeg.assign(outdeg, outdeg + nv);
  THV_TRY(validate(g.get()));
  THV_TRY(graph_init_device(g.get()));
  THV_TRY(set_packing(g.get(), true));
  *out = g.release();
  return THV_OK;
}

thv_status graph_adopt(uint64_t nv, uint64_t ne, thv_format fmt, uint32_t esz,
                       std::vector<uint64_t> &off, const void *d_edges,
                       std::vector<uint32_t> &outdeg, bool symmetric, int device,
                       thv_graph **out) {
  std::unique_ptr<thv_graph, void (*)(thv_graph *)> g(new thv_graph(), graph_destroy);
  g->nv = nv;
  g->ne = ne;
  g->fmt = fmt;
  g->esz = esz;
  g->weighted = esz == 8;
  g->sorted = true;  // the generator sorts by (src, dst)
  g->symmetric = symmetric;
  if (symmetric) g->mirrored = 1;  // the generator inserts every edge both ways
  g->device = device;
  g->off.swap(off);
  g->outdeg.swap(outdeg);
  THV_TRY(alloc_host_edges(g.get()));
  if (ne) THV_CUDA(cudaMemcpy(g->h_edges, d_edges, ne * esz, cudaMemcpyDeviceToHost));
  THV_TRY(graph_init_device(g.get()));
  THV_TRY(set_packing(g.get(), true));
  *out = g.release();
  return THV_OK;
}

static thv_status save(const thv_graph *g, const char *path) {
  std::unique_ptr<FILE, FileCloser> f(fopen(path, "wb"));
  if (!f) return fail(THV_EIO, "cannot create %s: %s", path, strerror(errno));
  bool ok = fwrite(&g->nv, 8, 1, f.get()) == 1 && fwrite(&g->ne, 8, 1, f.get()) == 1;
  ok = ok && (g->nv == 0 || fwrite(g->off.data(), 8, g->nv, f.get()) == g->nv);
  const uint64_t ne = g->ne;
  std::vector<uint32_t> buf;
  buf.reserve(1 << 20);
  auto flush = [&]() {
    ok = ok && (buf.empty() || fwrite(buf.data(), 4, buf.size(), f.get()) == buf.size());
    buf.clear();
  };
  uint32_t d, w;
  if (g->fmt == THV_FMT_WCSR) {
    for (uint64_t i = 0; ok && i < ne; i++) {
      edge_at(g, i, &d, &w);
      buf.push_back(d);
      buf.push_back(w);
      if (buf.size() >= (1u << 20)) flush();
    }
    flush();
  } else {
    for (uint64_t i = 0; ok && i < ne; i++) {
      edge_at(g, i, &d, &w);
      buf.push_back(d);
      if (buf.size() == (1u << 20)) flush();
    }
    flush();
    if (g->fmt == THV_FMT_CSR) {  // trailing weight section
      for (uint64_t i = 0; ok && i < ne; i++) {
        edge_at(g, i, &d, &w);
        buf.push_back(w);
        if (buf.size() == (1u << 20)) flush();
      }
      flush();
    } else {
      ok = ok && (g->nv == 0 || fwrite(g->outdeg.data(), 4, g->nv, f.get()) == g->nv);
    }
  }
  if (!ok) return fail(THV_EIO, "write to %s failed", path);
  return THV_OK;
}

}  // namespace thv

// ===================================================================== ABI

using namespace thv;

#define THV_GUARD_BEGIN try {
#define THV_GUARD_END                                                   \
  }                                                                     \
  catch (const std::bad_alloc &) {                                      \
    return fail(THV_ENOMEM, "host allocation failed");                  \
  }                                                                     \
  catch (const std::exception &ex) {                                    \
    return fail(THV_EINVAL, "exception: %s", ex.what());                \
  }                                                                     \
  catch (...) {                                                         \
    return fail(THV_EINVAL, "unknown exception");                       \
  }

extern "C" {

thv_status thv_open(const char *path, thv_format fmt, uint32_t flags,
                    int device, thv_graph **out) {
  THV_GUARD_BEGIN
  if (fmt != THV_FMT_CSR && fmt != THV_FMT_CSC && fmt != THV_FMT_WCSR)
    return fail(THV_EINVAL, "unknown format %d", (int)fmt);
  return open_file(path, fmt, flags, device, out);
  THV_GUARD_END
}

thv_status thv_from_arrays(uint64_t nv, uint64_t ne, const uint64_t *off,
                           const void *edges, uint32_t esz, thv_format fmt,
                           const uint32_t *outdeg, int device,
                           thv_graph **out) {
  THV_GUARD_BEGIN
  return from_arrays(nv, ne, off, edges, esz, fmt, outdeg, device, out);
  THV_GUARD_END
}

thv_status thv_generate_rmat(const thv_rmat_opts *o, thv_format fmt,
                             int device, thv_graph **out) {
  THV_GUARD_BEGIN
  if (!o || !out) return fail(THV_EINVAL, "null argument");
  return generate_rmat(o, fmt, device, out);
  THV_GUARD_END
}

thv_status thv_save(const thv_graph *g, const char *path) {
  THV_GUARD_BEGIN
  if (!g || !path) return fail(THV_EINVAL, "null argument");
  return save(g, path);
  THV_GUARD_END
}

thv_status thv_close(thv_graph *g) {
  THV_GUARD_BEGIN
  graph_destroy(g);
  return THV_OK;
  THV_GUARD_END
}

thv_status thv_info(const thv_graph *g, thv_graph_info *o) {
  if (!g || !o) return fail(THV_EINVAL, "null argument");
  o->nv = g->nv;
  o->ne = g->ne;
  o->fmt = g->fmt;
  o->esz = g->packed ? 8 : g->esz;
  o->device = (uint32_t)g->device;
  o->weighted = g->weighted;
  o->mem_esz = g->esz;
  o->weight_bits = g->packed ? g->wshift : 0;
  o->sorted = g->sorted;
  o->symmetric = g->symmetric;
  return THV_OK;
}

thv_status thv_convert(const char *txt_path, const char *out_path, thv_format fmt,
                       uint32_t skip_lines, uint32_t flags, int device, uint64_t *nv_out,
                       uint64_t *ne_out) {
  THV_GUARD_BEGIN
  return convert_edge_list(txt_path, out_path, fmt, skip_lines, flags, device, nv_out, ne_out);
  THV_GUARD_END
}

thv_status thv_set_symmetric(thv_graph *g, int symmetric) {
  THV_GUARD_BEGIN
  if (!g) return fail(THV_EINVAL, "null graph");
  g->symmetric = symmetric != 0;
  if (g->symmetric && g->mirrored < 0) g->mirrored = edges_mirrored(g);
  return THV_OK;
  THV_GUARD_END
}

thv_status thv_set_edge_packing(thv_graph *g, int packed) {
  THV_GUARD_BEGIN
  if (!g) return fail(THV_EINVAL, "null graph");
  return set_packing(g, packed != 0);
  THV_GUARD_END
}

thv_status thv_host_arrays(const thv_graph *g, const uint64_t **off,
                           const void **edges, const uint32_t **outdeg) {
  if (!g) return fail(THV_EINVAL, "null argument");
  if (off) *off = g->off.data();
  if (edges && g->packed && g->h_unpacked.size() != 2 * g->ne) {
    g->h_unpacked.resize(2 * g->ne);
    uint32_t *u = g->h_unpacked.data();
#pragma omp parallel for schedule(static)
    for (int64_t i = 0; i < (int64_t)g->ne; i++) edge_at(g, i, &u[2 * i], &u[2 * i + 1]);
  }
  if (edges) *edges = g->packed ? (const void *)g->h_unpacked.data() : g->h_edges;
  if (outdeg) *outdeg = g->fmt == THV_FMT_CSC ? g->outdeg.data() : nullptr;
  return THV_OK;
}

thv_status thv_plan(thv_graph *g, const thv_plan_opts *o) {
  THV_GUARD_BEGIN
  if (!g) return fail(THV_EINVAL, "null graph");
  return do_plan(g, o);
  THV_GUARD_END
}

thv_status thv_get_plan(const thv_graph *g, thv_plan_info *o) {
  if (!g || !o) return fail(THV_EINVAL, "null argument");
  if (!g->plan.valid) return fail(THV_EINVAL, "graph has no plan yet");
  const Plan &p = g->plan;
  o->num_blocks = p.blocks.size();
  o->resident_blocks = 0;
  for (const Block &b : p.blocks) o->resident_blocks += b.resident;
  o->resident_edge_bytes = p.resident_edge_bytes;
  o->host_edge_bytes = p.host_edge_bytes;
  o->device_bytes = g->device_bytes + p.d_resident_bytes +
                    (p.d_lists ? p.d_lists_bytes + g->nv * 4 : 0);
  o->small_list_degree = p.list_deg;
  o->small_list_bytes = p.list_bytes;
  o->small_list_vertices = p.list_vertices;
  return THV_OK;
}

thv_status thv_get_block_access(const thv_graph *g, uint64_t cap, uint64_t *link_bytes,
                                uint64_t *nb) {  // link_bytes: all adjacency bytes read
  if (!g || !nb) return fail(THV_EINVAL, "null argument");
  if (!g->plan.valid) return fail(THV_EINVAL, "graph has no plan yet");
  const Plan &p = g->plan;
  *nb = p.blocks.size();
  if (!link_bytes) return THV_OK;
  if (!p.d_access) return fail(THV_EINVAL, "plan does not track access (THV_PLAN_TRACK_ACCESS)");
  if (cap < p.blocks.size()) return fail(THV_EINVAL, "capacity %llu < %zu blocks",
                                         (unsigned long long)cap, p.blocks.size());
  THV_CUDA(cudaMemcpy(link_bytes, p.d_access, p.blocks.size() * 8, cudaMemcpyDeviceToHost));
  return THV_OK;
}

thv_status thv_save_plan(const thv_graph *g, const char *path) {
  THV_GUARD_BEGIN
  if (!g || !path) return fail(THV_EINVAL, "null argument");
  return save_plan(g, path);
  THV_GUARD_END
}

thv_status thv_load_plan(thv_graph *g, const char *path) {
  THV_GUARD_BEGIN
  if (!g || !path) return fail(THV_EINVAL, "null argument");
  return load_plan(g, path);
  THV_GUARD_END
}

thv_status thv_get_blocks(const thv_graph *g, uint64_t cap, uint32_t *vbegin,
                          uint8_t *resident, uint64_t *nb) {
  if (!g || !nb) return fail(THV_EINVAL, "null argument");
  if (!g->plan.valid) return fail(THV_EINVAL, "graph has no plan yet");
  const Plan &p = g->plan;
  *nb = p.blocks.size();
  if (cap < p.blocks.size()) return vbegin || resident ? fail(THV_EINVAL, "capacity %llu < %zu blocks",
                                                              (unsigned long long)cap, p.blocks.size())
                                                       : THV_OK;
  for (size_t i = 0; i < p.blocks.size(); i++) {
    if (vbegin) vbegin[i] = p.blocks[i].vbegin;
    if (resident) resident[i] = p.blocks[i].resident ? 1 : 0;
  }
  if (vbegin) vbegin[p.blocks.size()] = (uint32_t)g->nv;
  return THV_OK;
}

thv_status thv_run(thv_graph *g, thv_algo algo, const thv_run_opts *o,
                   void *out_values, thv_stats *stats) {
  THV_GUARD_BEGIN
  if (!g) return fail(THV_EINVAL, "null graph");
  const double t0 = now_ms();
  THV_CUDA(cudaSetDevice(g->device));
  thv_stats local{};
  cudaStream_t st = o && o->stream ? (cudaStream_t)o->stream : g->stream;
  thv_status s;
  switch (algo) {
    case THV_ALGO_BFS:
    case THV_ALGO_CC:
    case THV_ALGO_SSSP:
      s = run_minprop(g, algo, o, st, &local, (uint32_t *)out_values);
      if (s == THV_OK && out_values) local.d2h_bytes += g->nv * 4;
      break;
    case THV_ALGO_PR_PUSH:
    case THV_ALGO_PR_PULL:
      s = run_pagerank(g, algo, o, st, &local);
      if (s == THV_OK && out_values) {
        s = pagerank_values(g, (double *)out_values, st);
        local.d2h_bytes += g->nv * 8;
      }
      break;
    default:
      return fail(THV_EINVAL, "unknown algorithm %d", (int)algo);
  }
  local.wall_ms = now_ms() - t0;
  if (stats) *stats = local;
  return s;
  THV_GUARD_END
}

thv_status thv_values(thv_graph *g, void *out) {
  THV_GUARD_BEGIN
  if (!g || !out) return fail(THV_EINVAL, "null argument");
  THV_CUDA(cudaSetDevice(g->device));
  if (g->last_algo == THV_ALGO_PR_PUSH || g->last_algo == THV_ALGO_PR_PULL)
    return pagerank_values(g, (double *)out, g->stream);
  if (g->last_algo < 0) return fail(THV_EINVAL, "no values: nothing ran");
  return minprop_values(g, (uint32_t *)out, g->stream);
  THV_GUARD_END
}

thv_status thv_write_values(const char *path, const void *values, uint64_t n,
                            uint32_t elem_size) {
  THV_GUARD_BEGIN
  if (!path || (!values && n)) return fail(THV_EINVAL, "null argument");
  std::unique_ptr<FILE, FileCloser> f(fopen(path, "wb"));
  if (!f) return fail(THV_EIO, "cannot create %s: %s", path, strerror(errno));
  if (n && fwrite(values, elem_size, n, f.get()) != n)
    return fail(THV_EIO, "write to %s failed", path);
  return THV_OK;
  THV_GUARD_END
}

thv_status thv_batch_run(thv_graph *g, thv_algo algo, const uint32_t *sources,
                         uint32_t n, const thv_batch_opts *o, uint32_t *out,
                         uint64_t *checksums, thv_stats *stats) {
  THV_GUARD_BEGIN
  if (!g || (!sources && n)) return fail(THV_EINVAL, "null argument");
  THV_CUDA(cudaSetDevice(g->device));
  return run_batch(g, algo, sources, n, o, out, checksums, stats);
  THV_GUARD_END
}

thv_status thv_batch_tuned(thv_graph *g, thv_algo algo, thv_batch_config *out) {
  THV_GUARD_BEGIN
  if (!g || !out) return fail(THV_EINVAL, "null argument");
  THV_CUDA(cudaSetDevice(g->device));
  return batch_config(g, algo, out);
  THV_GUARD_END
}

thv_status thv_pick_sources(const thv_graph *g, uint64_t seed, uint32_t n, uint32_t *out) {
  if (!g || (!out && n)) return fail(THV_EINVAL, "null argument");
  if (g->nv == 0) return fail(THV_EINVAL, "empty graph");
  const uint64_t key = mix64_host(seed ^ 0x534F555243455331ull);
  for (uint32_t j = 0; j < n; j++) {
    bool found = false;
    for (uint64_t t = 0; t < (1ull << 24) && !found; t++) {
      const uint64_t c = mix64_host(key ^ (((uint64_t)j << 24) | t)) % g->nv;
      if (g->off[c + 1] > g->off[c]) {
        out[j] = (uint32_t)c;
        found = true;
      }
    }
    if (!found) return fail(THV_EINVAL, "no vertex with out-degree > 0");
  }
  return THV_OK;
}

const char *thv_last_error(void) { return g_last_error.c_str(); }

const char *thv_status_str(thv_status s) {
  switch (s) {
    case THV_OK: return "ok";
    case THV_EINVAL: return "invalid argument";
    case THV_EIO: return "i/o error";
    case THV_EFORMAT: return "malformed graph file";
    case THV_ENOMEM: return "out of memory";
    case THV_ECUDA: return "cuda error";
    case THV_ETIMEOUT: return "timeout";
    case THV_EUNSUPPORTED: return "unsupported";
    case THV_EBUSY: return "busy";
    case THV_ENOTREADY: return "not ready";
    case THV_EDEVICE: return "device error";
  }
  return "unknown status";
}

uint32_t thv_abi_version(void) { return THV_ABI_VERSION; }

void thv_debug_fail_alloc_after(uint32_t n) { g_fail_alloc_after = n; }

}  // extern "C"
