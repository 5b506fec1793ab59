// Many graphs in one call: BFS over a batch of independent graphs of uneven
// size.  The graphs live in one device arena as one union graph (vertices and
// edges numbered consecutively), which the all-levels BFS loop traverses with
// every CTA of the GPU on every level, top-down or bottom-up (gg_loop.cu): a
// level's edges are spread over the GPU whatever graph they belong to, where
// one CTA per graph would leave the GPU waiting for the largest one (256
// R-MAT graphs of scale 10-16, 90M edges: 8.5 ms, of which the largest graph
// alone).  Once the frontier has fewer than a window of edges per graph and grows
// by less than four times a level, a persistent kernel takes over, for the rest
// of the traversal, whose CTAs take whole graphs from a device work queue (largest
// first) and finish each inside the CTA without grid barriers: its
// level-synchronous top-down traversal of app/BFS.C:77-101 balances a
// frontier's edges over the CTA's threads by a block prefix sum over the
// frontier's degrees.  Batches past 2^31 vertices or 2^32 - 64 edges, those whose
// in-edges do not fit beside them, and small graphs that are all resident at
// once run in that kernel alone.  The launch
// sequence is captured once as a CUDA graph and replayed.
#include <cub/cub.cuh>

#include <algorithm>
#include <mutex>
#include <numeric>
#include <unordered_set>
#include <vector>

#include "gg_loop.cuh"

// Graph i's vertices are vfirst .. vfirst + n - 1 in the arenas: the union's
// ids, or 0 .. n - 1 where the batch is too large for one union graph.
struct BatchDesc {
  uint64_t off_base;  // the offset of the graph's first vertex in the offsets arena
  uint64_t idx_base;  // where the offsets count from in the index arena
  uint64_t lev_base;  // first level slot of the graph
  uint32_t n;
  uint32_t vfirst;
};

struct gg_graph_batch_s {
  int device = 0;
  cudaStream_t stream = nullptr;
  int32_t count = 0;
  uint64_t total_n = 0, total_m = 0;
  uint64_t edges = 0;  // edges in the arena: a graph's from its offsets[0] on
  uint32_t max_n = 0;
  std::vector<uint64_t> firsts;
  bool whole = false;  // union ids in the arenas (else every graph counts from 0)
  bool loop = false;   // the union's in-edges and loop buffers exist: the loop runs first (else one CTA per graph alone)
  int num_sms = 0;
  gg::UnionBfs uni;
  uint32_t *d_ioff = nullptr, *d_iidx = nullptr;
  uint32_t *d_off = nullptr, *d_idx = nullptr, *d_order = nullptr, *d_src = nullptr, *d_scratch = nullptr;
  BatchDesc* d_desc = nullptr;
  int32_t* d_levels = nullptr;
  unsigned long long* d_ctr = nullptr;  // [0] work ticket, [1] edges traversed
  uint32_t* h_src = nullptr;            // pinned
  int32_t* h_levels = nullptr;          // pinned
  unsigned long long* h_ctr = nullptr;  // pinned: the counters, then the union loop's state
  int grid = 0;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
};

namespace gg {

static std::mutex g_batch_mu;
static std::unordered_set<const gg_graph_batch_s*> g_batches;

static bool batch_live(const gg_graph_batch_s* b) {
  std::lock_guard<std::mutex> lk(g_batch_mu);
  return b && g_batches.count(b);
}

constexpr int kBatchThreads = 256;

__global__ void __launch_bounds__(kBatchThreads) k_batch_bfs(const BatchDesc* __restrict__ desc,
                                                              const uint32_t* __restrict__ order, int32_t count,
                                                              const uint32_t* __restrict__ off,
                                                              const uint32_t* __restrict__ idx, int32_t* levels,
                                                              const uint32_t* __restrict__ src,
                                                              unsigned long long* ctr, uint32_t* scratch,
                                                              uint64_t stride, const gg::LoopState* st) {
  __shared__ int32_t s_graph;
  __shared__ uint32_t s_scan[kBatchThreads + 1];
  __shared__ uint32_t s_beg[kBatchThreads];
  __shared__ uint32_t s_warp[32];
  __shared__ uint32_t s_nq;
  // st: the union loop ran first, and either finished or left the vertices of
  // level levels_done as the frontier
  if (st && st->exit_reason != 4) return;
  const int32_t level0 = st ? st->levels_done : 0;
  const int tid = threadIdx.x, lane = tid & 31;
  const uint32_t lanemask_lt = (1u << lane) - 1u;
  uint32_t* qa = scratch + (uint64_t)blockIdx.x * 2 * stride;
  uint32_t* qb = qa + stride;
  unsigned long long trav = 0;
  for (;;) {
    if (tid == 0) {
      const unsigned long long t = atomicAdd(ctr, 1ull);
      s_graph = t < (unsigned long long)count ? (int32_t)order[t] : -1;
    }
    __syncthreads();
    const int32_t gi = s_graph;
    if (gi < 0) break;
    const BatchDesc d = desc[gi];
    const uint32_t* go = off + d.off_base;
    const uint32_t* gx = idx + d.idx_base;
    int32_t* lev = levels + d.lev_base;  // lev, go and the queues: local vertices; gx: arena ids
    uint32_t qn = 1;
    int32_t r = level0;
    if (st) {  // the frontier is what the levels say
      if (tid == 0) s_nq = 0;
      __syncthreads();
      for (uint32_t v0 = tid; v0 - tid < d.n; v0 += 8 * kBatchThreads) {  // 8 loads in flight per thread
        int32_t l[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) l[u] = v0 + u * kBatchThreads < d.n ? __ldcg(lev + v0 + u * kBatchThreads) : -1;
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const bool add = l[u] == level0;
          const uint32_t bal = __ballot_sync(0xffffffffu, add);
          if (bal) {
            const int leader = __ffs(bal) - 1;
            uint32_t base = 0;
            if (lane == leader) base = atomicAdd(&s_nq, (uint32_t)__popc(bal));
            base = __shfl_sync(0xffffffffu, base, leader);
            if (add) qa[base + __popc(bal & lanemask_lt)] = v0 + u * kBatchThreads;
          }
        }
      }
      __syncthreads();
      qn = s_nq;
      __syncthreads();
    } else {
      for (uint32_t v = tid; v < d.n; v += kBatchThreads) lev[v] = -1;
      __syncthreads();
      const uint32_t s = src[gi] - d.vfirst;
      if (tid == 0) {
        lev[s] = 0;
        qa[0] = s;
      }
      __syncthreads();
    }
    while (qn > 0) {
      ++r;
      if (tid == 0) s_nq = 0;
      for (uint32_t c0 = 0; c0 < qn; c0 += kBatchThreads) {
        const uint32_t i = c0 + tid;
        uint32_t beg = 0, deg = 0;
        if (i < qn) {
          const uint32_t v = qa[i];
          beg = go[v];
          deg = go[v + 1] - beg;
        }
        uint32_t total;
        const uint32_t excl = block_excl_scan(deg, s_warp, &total);
        s_scan[tid] = excl;
        s_beg[tid] = beg;
        if (tid == 0) s_scan[kBatchThreads] = total;
        __syncthreads();
        trav += (tid == 0) ? total : 0u;
        for (uint32_t t0 = 0; t0 < total; t0 += kBatchThreads) {
          const uint32_t t = t0 + tid;
          bool add = false;
          uint32_t u = 0;
          if (t < total) {
            // owner: the last slot whose exclusive start is <= t
            int lo = 0, hi = kBatchThreads - 1;
            while (lo < hi) {
              const int mid = (lo + hi + 1) >> 1;
              if (s_scan[mid] <= t)
                lo = mid;
              else
                hi = mid - 1;
            }
            u = gx[s_beg[lo] + (t - s_scan[lo])] - d.vfirst;
            if (__ldcg(lev + u) < 0) add = atomicCAS(lev + u, -1, r) == -1;
          }
          const uint32_t bal = __ballot_sync(0xffffffffu, add);
          if (bal) {
            const int leader = __ffs(bal) - 1;
            uint32_t base = 0;
            if (lane == leader) base = atomicAdd(&s_nq, (uint32_t)__popc(bal));
            base = __shfl_sync(0xffffffffu, base, leader);
            if (add) qb[base + __popc(bal & lanemask_lt)] = u;
          }
        }
        __syncthreads();
      }
      qn = s_nq;
      uint32_t* t = qa;
      qa = qb;
      qb = t;
      __syncthreads();
    }
  }
  if (tid == 0 && trav) atomicAdd(ctr + 1, trav);
}

static void batch_release(gg_graph_batch_s* b) {
  if (!b) return;
  if (b->exec) cudaGraphExecDestroy(b->exec);
  if (b->graph) cudaGraphDestroy(b->graph);
  gg::union_bfs_free(b->uni);
  cudaFree(b->d_off);
  cudaFree(b->d_idx);
  cudaFree(b->d_ioff);
  cudaFree(b->d_iidx);
  cudaFree(b->d_order);
  cudaFree(b->d_src);
  cudaFree(b->d_scratch);
  cudaFree(b->d_desc);
  cudaFree(b->d_levels);
  cudaFree(b->d_ctr);
  if (b->h_src) cudaFreeHost(b->h_src);
  if (b->h_levels) cudaFreeHost(b->h_levels);
  if (b->h_ctr) cudaFreeHost(b->h_ctr);
  if (b->stream) cudaStreamDestroy(b->stream);
  delete b;
}

// Global ids for every edge of the union (CTAs over graphs).
__global__ void k_batch_globalise(const BatchDesc* desc, const uint64_t* edge_first, int32_t count, uint32_t* idx) {
  for (int32_t i = blockIdx.x; i < count; i += gridDim.x) {
    const uint32_t base = desc[i].vfirst;
    for (uint64_t e = edge_first[i] + threadIdx.x; e < edge_first[i + 1]; e += blockDim.x) idx[e] += base;
  }
}

// The source of every out-edge, one warp per vertex.
__global__ void k_batch_src(uint32_t n, const uint32_t* off, uint32_t* src) {
  const uint64_t w0 = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t v = w0; v < n; v += nw)
    for (uint32_t e = off[v] + (threadIdx.x & 31); e < off[v + 1]; e += 32) src[e] = (uint32_t)v;
}

// In-offsets from the edges' destinations in ascending order: each vertex's is
// found by bisection, so that a long run of vertices without in-edges is not
// one thread's work (64M vertices without edges: gg_batch_create 455 ms with a
// thread per edge that fills the run before it, 242 ms now).
__global__ void k_batch_in_off(uint64_t m, uint32_t n, const uint32_t* __restrict__ dst, uint32_t* ioff) {
  for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v <= n; v += (uint64_t)gridDim.x * blockDim.x) {
    uint64_t lo = 0, hi = m;  // the first edge whose destination is >= v
    while (lo < hi) {
      const uint64_t mid = (lo + hi) >> 1;
      if (dst[mid] < v)
        lo = mid + 1;
      else
        hi = mid;
    }
    ioff[v] = (uint32_t)lo;
  }
}

// The union's in-edges, for the bottom-up levels: a stable sort by
// destination, so in-lists stay in source order.
static int batch_in_edges(gg_graph_batch_s* b, uint32_t n) {
  const uint64_t m = b->edges;
  GG_CUDA(cudaMalloc(&b->d_ioff, 4 * ((uint64_t)n + 1)));
  GG_CUDA(cudaMalloc(&b->d_iidx, 4 * (m + 16)));
  GG_CUDA(cudaMemsetAsync(b->d_iidx + m, 0, 64, b->stream));
  struct Hold {
    void* p[3] = {nullptr, nullptr, nullptr};
    ~Hold() {
      for (void* q : p) cudaFree(q);
    }
  } h;
  const uint64_t me = std::max<uint64_t>(m, 1);
  GG_CUDA(cudaMalloc(&h.p[0], 4 * me));
  GG_CUDA(cudaMalloc(&h.p[1], 4 * me));
  uint32_t *src = static_cast<uint32_t*>(h.p[0]), *dst = static_cast<uint32_t*>(h.p[1]);
  const int grid = b->num_sms * 8;
  int bits = 1;
  while (bits < 32 && (n - 1) >> bits) ++bits;
  if (m) {
    k_batch_src<<<grid, 256, 0, b->stream>>>(n, b->d_off, src);
    GG_CUDA(cudaGetLastError());
    size_t temp = 0;
    GG_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, temp, b->d_idx, dst, src, b->d_iidx, m, 0, bits, b->stream));
    GG_CUDA(cudaMalloc(&h.p[2], std::max<size_t>(temp, 1)));
    GG_CUDA(cub::DeviceRadixSort::SortPairs(h.p[2], temp, b->d_idx, dst, src, b->d_iidx, m, 0, bits, b->stream));
  }
  k_batch_in_off<<<grid, 256, 0, b->stream>>>(m, n, dst, b->d_ioff);
  GG_CUDA(cudaGetLastError());
  GG_CUDA(cudaStreamSynchronize(b->stream));
  return GG_OK;
}

// One CTA per graph, and its counters to the host: alone (st null), or from
// where the union loop with state st stopped.
static int batch_per_cta(gg_graph_batch_s* b, const LoopState* st) {
  GG_CUDA(cudaMemsetAsync(b->d_ctr, 0, 16, b->stream));
  k_batch_bfs<<<b->grid, kBatchThreads, 0, b->stream>>>(b->d_desc, b->d_order, b->count, b->d_off, b->d_idx,
                                                          b->d_levels, b->d_src, b->d_ctr, b->d_scratch, b->max_n, st);
  GG_CUDA(cudaGetLastError());
  GG_CUDA(cudaMemcpyAsync(b->h_ctr, b->d_ctr, 16, cudaMemcpyDeviceToHost, b->stream));
  return GG_OK;
}

// Host data to the device in the order of the batch's stream.  That stream does
// not wait for the default stream, in which a plain copy of pageable memory may
// still be under way when the call returns.
template <class T>
static int upload(gg_graph_batch_s* b, T* dst, const T* src, uint64_t count) {
  GG_CUDA(cudaMemcpyAsync(dst, src, sizeof(T) * count, cudaMemcpyHostToDevice, b->stream));
  return GG_OK;
}

// A batch of small graphs that are all resident at once needs no union: the
// loop's three launches and its barriers cost more than the largest graph takes
// in a CTA (64 R-MAT graphs of n + m = 1050 / 4950 / 8170 / 13000, loop against
// one CTA per graph: 75 / 75 / 76 / 78 us against 53 / 72 / 83 / 111; 4000 of
// 2800, more than are resident: 190 against 204).
constexpr uint64_t kSmallGraph = 6144;

static int batch_build(int32_t count, const gg_host_graph* graphs, const gg_batch_opts& opts, gg_graph_batch_s* b) {
  b->count = count;
  std::vector<BatchDesc> desc(count);
  for (int32_t i = 0; i < count; ++i) {
    const gg_host_graph& h = graphs[i];
    if (h.n == 0 || !h.offsets || (h.m && !h.indices) || h.offsets[h.n] != h.m || h.offsets[0] > h.m)
      return fail(GG_ERR_INVALID_ARG, "gg_batch_create: graph %d is malformed", i);
    b->firsts.push_back(b->total_n);
    b->total_m += h.m;
    b->total_n += h.n;
    b->max_n = std::max(b->max_n, h.n);
  }
  // a graph's first edges, where offsets[0] is not 0, belong to no vertex and
  // stay out of the arena
  std::vector<uint64_t> edge_first(count + 1, 0);
  for (int32_t i = 0; i < count; ++i) edge_first[i + 1] = edge_first[i] + graphs[i].m - graphs[i].offsets[0];
  b->edges = edge_first[count];
  uint64_t largest = 0;  // vertices and edges of the largest graph
  for (int32_t i = 0; i < count; ++i)
    largest = std::max(largest, graphs[i].n + (edge_first[i + 1] - edge_first[i]));
  b->whole = opts.form != GG_BATCH_SEPARATE && b->total_n < (1ull << 31) && b->edges < (1ull << 32) - 64;
  for (int32_t i = 0; i < count; ++i) {
    const uint64_t v0 = b->firsts[i];
    desc[i] = b->whole ? BatchDesc{v0, 0, v0, graphs[i].n, (uint32_t)v0}
                       : BatchDesc{v0 + (uint64_t)i, edge_first[i], v0, graphs[i].n, 0};
  }
  const uint64_t offs = b->whole ? b->total_n + 1 : b->total_n + count;
  GG_CUDA(cudaGetDevice(&b->device));
  GG_CUDA(cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking));
  GG_CUDA(cudaDeviceGetAttribute(&b->num_sms, cudaDevAttrMultiProcessorCount, b->device));
  GG_CUDA(cudaMalloc(&b->d_off, 4 * offs));
  GG_CUDA(cudaMalloc(&b->d_idx, 4 * std::max<uint64_t>(b->edges, 1)));
  GG_CUDA(cudaMalloc(&b->d_levels, 4 * b->total_n));
  GG_CUDA(cudaMalloc(&b->d_desc, sizeof(BatchDesc) * count));
  GG_CUDA(cudaMalloc(&b->d_order, 4 * count));
  GG_CUDA(cudaMalloc(&b->d_src, 4 * count));
  GG_CUDA(cudaMalloc(&b->d_ctr, 16));
  // all that one CTA per graph needs comes before the union's buffers, which a
  // batch can do without
  int per_sm = 0;
  GG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_batch_bfs, kBatchThreads, 0));
  b->grid = std::max(1, std::min(count, b->num_sms * std::max(per_sm, 1)));
  GG_CUDA(cudaMalloc(&b->d_scratch, 8ull * b->max_n * b->grid));
  GG_CUDA(cudaMallocHost(&b->h_src, 4 * count));
  GG_CUDA(cudaMallocHost(&b->h_levels, 4 * b->total_n));
  GG_CUDA(cudaMallocHost(&b->h_ctr, 16 + sizeof(LoopState)));
  GG_TRY(upload(b, b->d_desc, desc.data(), count));
  {
    std::vector<uint32_t> off(offs);
#pragma omp parallel for schedule(dynamic, 8)
    for (int32_t i = 0; i < count; ++i) {
      const gg_host_graph& h = graphs[i];
      const uint32_t base = (b->whole ? (uint32_t)edge_first[i] : 0u) - h.offsets[0];
      for (uint64_t v = 0; v < (uint64_t)h.n + (b->whole ? 0 : 1); ++v) off[desc[i].off_base + v] = h.offsets[v] + base;
    }
    if (b->whole) off[b->total_n] = (uint32_t)b->edges;
    GG_TRY(upload(b, b->d_off, off.data(), offs));
    GG_CUDA(cudaStreamSynchronize(b->stream));  // off leaves scope
  }
  for (int32_t i = 0; i < count; ++i)
    if (edge_first[i + 1] > edge_first[i])
      GG_TRY(upload<uint32_t>(b, b->d_idx + edge_first[i], graphs[i].indices + graphs[i].offsets[0],
                              edge_first[i + 1] - edge_first[i]));
  if (b->whole) {
    uint64_t* d_first = nullptr;
    GG_CUDA(cudaMalloc(&d_first, 8 * ((uint64_t)count + 1)));
    struct Hold {
      void* p;
      ~Hold() { cudaFree(p); }
    } hold{d_first};
    GG_TRY(upload(b, d_first, edge_first.data(), (uint64_t)count + 1));
    k_batch_globalise<<<std::min(count, b->num_sms * 8), 256, 0, b->stream>>>(b->d_desc, d_first, count, b->d_idx);
    GG_CUDA(cudaGetLastError());
    b->uni.off = b->d_off;
    b->uni.idx = b->d_idx;
    b->uni.levels = b->d_levels;
    b->uni.n = (uint32_t)b->total_n;
    b->uni.m = b->edges;
    if (opts.wait_budget) b->uni.wait_budget = opts.wait_budget < 0 ? 0u : (unsigned)opts.wait_budget;
    // a batch whose in-edges or loop buffers do not fit beside it keeps one
    // CTA per graph, as on a device without cooperative launches
    int rc = GG_ERR_UNSUPPORTED;
    if (opts.form == GG_BATCH_AUTO && !(largest <= kSmallGraph && count <= b->grid)) {
      rc = batch_in_edges(b, (uint32_t)b->total_n);
      b->uni.ioff = b->d_ioff;
      b->uni.iidx = b->d_iidx;
      if (!rc) rc = union_bfs_prepare(b->uni, b->device, b->num_sms);
      if (rc && cudaGetLastError() != cudaErrorMemoryAllocation && rc != GG_ERR_UNSUPPORTED) return rc;
    }
    b->loop = rc == GG_OK;
    if (!b->loop) {
      union_bfs_free(b->uni);
      cudaFree(b->d_ioff);
      cudaFree(b->d_iidx);
      b->d_ioff = b->d_iidx = nullptr;
    }
  }
  std::vector<uint32_t> order(count);
  std::iota(order.begin(), order.end(), 0u);
  std::stable_sort(order.begin(), order.end(), [&](uint32_t x, uint32_t y) { return graphs[x].m > graphs[y].m; });
  GG_TRY(upload(b, b->d_order, order.data(), count));
  GG_CUDA(cudaStreamSynchronize(b->stream));  // the host arrays are the caller's and this function's
  // the replayed sequence: sources up, counters reset, traversal, counters down
  GG_CUDA(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal));
  cudaMemcpyAsync(b->d_src, b->h_src, 4 * count, cudaMemcpyHostToDevice, b->stream);
  if (b->loop) GG_TRY(union_bfs_enqueue(b->uni, b->stream, b->num_sms, b->d_src, (uint32_t)count));
  GG_TRY(batch_per_cta(b, b->loop ? b->uni.st : nullptr));
  if (b->loop)
    cudaMemcpyAsync(b->h_ctr + 2, b->uni.st, sizeof(LoopState), cudaMemcpyDeviceToHost, b->stream);
  GG_CUDA(cudaStreamEndCapture(b->stream, &b->graph));
  GG_CUDA(cudaGraphInstantiate(&b->exec, b->graph, 0));
  return GG_OK;
}

// Whether bytes [p, p + bytes) are page-locked host memory at both ends (a
// copy from the device then needs no staging).
static bool pinned_range(const void* p, size_t bytes) {
  if (bytes == 0) return false;
  cudaPointerAttributes a{}, z{};
  const bool ok = cudaPointerGetAttributes(&a, p) == cudaSuccess && a.type == cudaMemoryTypeHost &&
                  cudaPointerGetAttributes(&z, static_cast<const char*>(p) + bytes - 1) == cudaSuccess &&
                  z.type == cudaMemoryTypeHost;
  if (!ok) cudaGetLastError();
  return ok;
}

}  // namespace gg

using namespace gg;

extern "C" {

int gg_batch_create(int32_t count, const gg_host_graph* graphs, gg_graph_batch_t* out) {
  return gg_batch_create_opts(count, graphs, nullptr, out);
}

int gg_batch_create_opts(int32_t count, const gg_host_graph* graphs, const gg_batch_opts* opts, gg_graph_batch_t* out) {
  const gg_batch_opts o = opts ? *opts : gg_batch_opts{GG_BATCH_AUTO, 0};
  if (count <= 0 || !graphs || !out || o.form < GG_BATCH_AUTO || o.form > GG_BATCH_SEPARATE)
    return fail(GG_ERR_INVALID_ARG, "gg_batch_create: bad arguments");
  int devs = 0;
  if (cudaGetDeviceCount(&devs) != cudaSuccess || devs == 0) {
    cudaGetLastError();
    return fail(GG_ERR_NO_DEVICE, "no CUDA device is visible");
  }
  gg_graph_batch_s* b = new (std::nothrow) gg_graph_batch_s;
  if (!b) return fail(GG_ERR_OOM, "batch: out of host memory");
  const int rc = batch_build(count, graphs, o, b);
  if (rc) {
    const std::string keep = last_error();
    cudaStreamEndCapture(b->stream, &b->graph);  // leaves no capture open on a failed build
    cudaGetLastError();
    batch_release(b);
    set_error("%s", keep.c_str());
    return rc;
  }
  {
    std::lock_guard<std::mutex> lk(g_batch_mu);
    g_batches.insert(b);
  }
  *out = b;
  return GG_OK;
}

int gg_batch_destroy(gg_graph_batch_t b) {
  {
    std::lock_guard<std::mutex> lk(g_batch_mu);
    if (!b || !g_batches.erase(b)) return fail(GG_ERR_INVALID_ARG, "gg_batch_destroy: unknown batch");
  }
  cudaStreamSynchronize(b->stream);
  batch_release(b);
  return GG_OK;
}

int gg_batch_info(gg_graph_batch_t b, uint64_t* total_vertices, uint64_t* total_edges, uint64_t* firsts) {
  if (!batch_live(b)) return fail(GG_ERR_INVALID_ARG, "gg_batch_info: unknown batch");
  if (total_vertices) *total_vertices = b->total_n;
  if (total_edges) *total_edges = b->total_m;
  if (firsts) std::copy(b->firsts.begin(), b->firsts.end(), firsts);
  return GG_OK;
}

int gg_batch_bfs(gg_graph_batch_t b, const uint32_t* sources, int32_t* levels, gg_run_stats* st) {
  if (!batch_live(b) || !sources) return fail(GG_ERR_INVALID_ARG, "gg_batch_bfs: bad arguments");
  for (int32_t i = 0; i < b->count; ++i) {
    const uint64_t n = (i + 1 < b->count ? b->firsts[i + 1] : b->total_n) - b->firsts[i];
    if (sources[i] >= n) return fail(GG_ERR_INVALID_ARG, "gg_batch_bfs: source %u of graph %d out of range", sources[i], i);
  }
  for (int32_t i = 0; i < b->count; ++i) b->h_src[i] = sources[i] + (b->whole ? (uint32_t)b->firsts[i] : 0u);
  EventTimer tm(b->stream);
  GG_CUDA(cudaGraphLaunch(b->exec, b->stream));
  int32_t* down = levels && pinned_range(levels, 4 * b->total_n) ? levels : b->h_levels;
  cudaError_t copied = cudaMemcpyAsync(down, b->d_levels, 4 * b->total_n, cudaMemcpyDeviceToHost, b->stream);
  if (copied == cudaErrorInvalidValue && down == levels) {  // page-locked at its ends only
    cudaGetLastError();
    down = b->h_levels;
    copied = cudaMemcpyAsync(down, b->d_levels, 4 * b->total_n, cudaMemcpyDeviceToHost, b->stream);
  }
  GG_CUDA(copied);
  double ms = tm.stop();
  GG_CUDA(cudaStreamSynchronize(b->stream));
  const LoopState* loop = b->loop ? reinterpret_cast<const LoopState*>(b->h_ctr + 2) : nullptr;
  int kernels = loop ? 4 : 1;
  uint64_t trav = loop ? loop->trav : 0;
  if (loop && loop->exit_reason != 1 && loop->exit_reason != 4) {
    // a grid barrier's wait ran out: one CTA per graph has none
    GG_TRY(batch_per_cta(b, nullptr));
    GG_CUDA(cudaMemcpyAsync(down, b->d_levels, 4 * b->total_n, cudaMemcpyDeviceToHost, b->stream));
    ms = tm.stop();
    GG_CUDA(cudaStreamSynchronize(b->stream));
    ++kernels;
    trav = 0;
  }
  GG_CUDA(cudaGetLastError());
  if (levels && down != levels) std::copy(b->h_levels, b->h_levels + b->total_n, levels);
  if (st) {
    st->ms = ms;
    st->rounds = 1;
    st->edges_traversed = trav + b->h_ctr[1];
    st->kernels = kernels;
  }
  return GG_OK;
}

}  // extern "C"
