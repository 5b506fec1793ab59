// Device-driven BFS levels: one cooperative launch runs consecutive
// sparse-push levels of app/BFS.C:77-101 (edgeMap's sparse branch,
// graphgrind/ligra-numa.h:868-916, with BFS_F::updateAtomic) without
// returning to the host between levels.  All CTAs are co-resident
// (cooperative launch); a level ends at a grid barrier, after which every CTA
// reads the next frontier's size and out-degree and applies edgeMap's
// direction rule (size + out-degree > threshold means a dense level): the
// launch returns when the frontier is empty, needs a dense level, or a level
// cap is reached, and the host continues with edgeMap.  A level's
// edges go to the CTAs in windows of 512: every queue slot carries its first
// edge's offset, and whoever appends a slot notes it as the first of each
// window whose first edge it holds, so a CTA reaches its window's slots with
// one load.  The barrier wait is bounded: on expiry the kernel records an error
// and returns.
#include "gg_loop.cuh"

namespace gg {

// Threads of a loop CTA, and edges of a window of a sparse level.  A sparse
// level of a high-diameter graph costs its latency: the grid barrier (whose
// arrivals all go to one L2 word) and one window's chain of dependent loads.
// Wider CTAs make fewer arrivals and hold more of the frontier per window, but
// a window's block barriers cost more (2049^2 grid, 125 levels: gg_bfs 1.85 /
// 1.59 / 2.16 ms with 256 / 512 / 1024 threads; R-MAT-22 0.53 / 0.52 / 0.53).
constexpr int kLoopThreads = 512;
constexpr int kLoopWarps = kLoopThreads / 32;

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ unsigned long long ld_relaxed_u64(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ int ld_relaxed_i32(const int32_t* p) {
  int v;
  asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// A slot's counters into shared memory: packed, zeros, dcnt, ddeg, rep.
__device__ __forceinline__ void read_slot(const LoopSlot* sl, unsigned long long* s_rd) {
  s_rd[0] = ld_relaxed_u64(&sl->packed);
  s_rd[1] = ld_relaxed_u64(&sl->zeros);
  s_rd[2] = ld_relaxed_u64(&sl->dcnt);
  s_rd[3] = ld_relaxed_u64(&sl->ddeg);
  s_rd[4] = (unsigned long long)(uint32_t)ld_relaxed_i32(&sl->rep);
}

// All CTAs of the (co-resident) grid arrive; returns false if the wait ran out
// (more than `budget` probes of the arrival count, each followed by a short
// sleep).  The arrival is a release and the wait an acquire by thread 0, so
// with the block barriers around them every write of the grid before the
// barrier is visible to every thread after it.  With `rd`, thread 0 then
// reads that slot's counters into s_rd for the whole CTA.
__device__ __forceinline__ bool grid_barrier(unsigned* bar, unsigned target, unsigned budget, int* s_ok,
                                             const LoopSlot* rd = nullptr, unsigned long long* s_rd = nullptr) {
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
    int ok = 1;
    for (unsigned it = 0; (int)(ld_acquire_u32(bar) - target) < 0; ++it) {
      if (it >= budget) {
        ok = 0;
        break;
      }
      __nanosleep(32);
    }
    if (ok && rd) read_slot(rd, s_rd);
    *s_ok = ok;
  }
  __syncthreads();
  return *s_ok != 0;
}

// A queue slot whose edges start at eoff is noted as the first slot of every
// window whose first edge it holds, so that a CTA finds its window's slots with
// one load.
__device__ __forceinline__ void note_windows(uint32_t* wst, uint32_t slot, uint32_t eoff, uint32_t deg) {
  for (uint64_t w = ((uint64_t)eoff + kLoopThreads - 1) / kLoopThreads; w * kLoopThreads < (uint64_t)eoff + deg; ++w)
    wst[w] = slot;
}
// The same for the lanes of a warp that add a slot (every lane calls it): a
// lane notes the first windows itself, and the warp a hub's others (a star's hub
// of 16M out-edges, 32768 windows: traversal 0.33 ms with one lane's stores, 0.18
// now).
constexpr uint32_t kOwnWindows = 256, kHubEdges = kOwnWindows * kLoopThreads;
__device__ __forceinline__ void note_windows_warp(uint32_t* wst, bool add, uint32_t slot, uint32_t eoff, uint32_t deg) {
  const uint32_t w0 = (uint32_t)(((uint64_t)eoff + kLoopThreads - 1) / kLoopThreads);
  const uint32_t w1 = add ? (uint32_t)(((uint64_t)eoff + deg + kLoopThreads - 1) / kLoopThreads) : w0;
  for (uint32_t w = w0; w < w1 && w - w0 < kOwnWindows; ++w) wst[w] = slot;
  uint32_t hubs = __ballot_sync(0xffffffffu, w1 - w0 > kOwnWindows);
  while (hubs) {
    const int l = __ffs(hubs) - 1;
    hubs &= hubs - 1;
    const uint32_t b = __shfl_sync(0xffffffffu, w0, l) + kOwnWindows, e = __shfl_sync(0xffffffffu, w1, l);
    const uint32_t sl = __shfl_sync(0xffffffffu, slot, l);
    for (uint32_t w = b + (threadIdx.x & 31); w < e; w += 32) wst[w] = sl;
  }
}

// Warp-cooperative append to the next frontier (every lane calls it).  A
// vertex with out-edges gets its queue slot and its first edge offset from one
// 64-bit atomic (slots in the high half, edges in the low half), so slot order
// is edge-offset order; a vertex without out-edges goes to the far end.
__device__ __forceinline__ void loop_append(bool add, uint32_t u, uint32_t deg, uint32_t* nq, uint32_t* neo,
                                            uint32_t* nwst, uint32_t n, unsigned long long* packed,
                                            unsigned long long* zeros) {
  const int lane = threadIdx.x & 31;
  const uint32_t lanemask_lt = (1u << lane) - 1u;
  const bool pos = add && deg > 0, zer = add && deg == 0;
  uint32_t inc = pos ? deg : 0u;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, inc, d);
    if (lane >= d) inc += t;
  }
  const uint32_t wsum = __shfl_sync(0xffffffffu, inc, 31);
  const uint32_t bal = __ballot_sync(0xffffffffu, pos);
  if (bal) {
    const int leader = __ffs(bal) - 1;
    unsigned long long old = 0;
    if (lane == leader) old = atomicAdd(packed, ((unsigned long long)__popc(bal) << 32) | wsum);
    old = __shfl_sync(0xffffffffu, old, leader);
    const uint32_t slot = (uint32_t)(old >> 32) + __popc(bal & lanemask_lt), eoff = (uint32_t)old + inc - deg;
    if (pos) {
      nq[slot] = u;
      neo[slot] = eoff;
    }
    note_windows_warp(nwst, pos, slot, eoff, deg);
  }
  const uint32_t zb = __ballot_sync(0xffffffffu, zer);
  if (zb) {
    const int leader = __ffs(zb) - 1;
    unsigned long long old = 0;
    if (lane == leader) old = atomicAdd(zeros, (unsigned long long)__popc(zb));
    old = __shfl_sync(0xffffffffu, old, leader);
    if (zer) nq[n - 1 - (old + __popc(zb & lanemask_lt))] = u;
  }
}

// block-wide exclusive scan of one 64-bit value (kLoopThreads threads)
__device__ __forceinline__ unsigned long long block_scan(unsigned long long a, unsigned long long* total,
                                                         unsigned long long* s) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned long long x = a;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long u = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += u;
  }
  if (lane == 31) s[warp] = x;
  __syncthreads();
  unsigned long long before = 0, all = 0;
#pragma unroll
  for (int w = 0; w < kLoopWarps; ++w) {
    if (w < warp) before += s[w];
    all += s[w];
  }
  *total = all;
  return before + x - a;
}

// Block-wide append to the next frontier (every thread calls it): one
// 64-bit atomic per CTA for the vertices with out-edges (slots and edge
// offsets, as loop_append) and one for those without.
__device__ __forceinline__ void block_append(bool add, uint32_t u, uint32_t deg, uint32_t* nq, uint32_t* neo,
                                             uint32_t* nwst, uint32_t n, unsigned long long* packed,
                                             unsigned long long* zeros, uint32_t* nbits,
                                             unsigned long long* s_scan, unsigned long long* s_base) {
  if (nbits && add) atomicOr(nbits + (u >> 5), 1u << (u & 31));
  const bool pos = add && deg > 0, zer = add && deg == 0;
  // counts packed as (with out-edges << 48) | (without << 32) | edges; at most kLoopThreads vertices
  unsigned long long total;
  const unsigned long long ex = block_scan((pos ? 1ull << 48 : 0ull) | (zer ? 1ull << 32 : 0ull) | (pos ? deg : 0u),
                                           &total, s_scan);
  const uint32_t np = (uint32_t)(total >> 48), nz = (uint32_t)(total >> 32) & 0xffffu;
  if (threadIdx.x == 0 && np) s_base[0] = atomicAdd(packed, ((unsigned long long)np << 32) | (uint32_t)total);
  if (threadIdx.x == 32 && nz) s_base[1] = atomicAdd(zeros, (unsigned long long)nz);
  __syncthreads();
  uint32_t slot = 0, eoff = 0;
  if (pos) {
    const unsigned long long old = s_base[0];
    slot = (uint32_t)(old >> 32) + (uint32_t)(ex >> 48);
    eoff = (uint32_t)old + (uint32_t)ex;
    nq[slot] = u;
    neo[slot] = eoff;
  } else if (zer) {
    nq[n - 1 - (s_base[1] + ((uint32_t)(ex >> 32) & 0xffffu))] = u;
  }
  note_windows_warp(nwst, pos, slot, eoff, deg);
}

// The shared memory of a sparse level's window.
struct PushShared {
  uint32_t eo[kLoopThreads];
  uint32_t v[kLoopThreads];
  uint32_t beg[kLoopThreads];
  unsigned long long scan[kLoopWarps];
  unsigned long long base[2];
};

// One sparse (top-down) level, this CTA's windows of its E edges: queue q with
// slot edge offsets eo (k slots, each with >= 1 edge) and window starts wst;
// vertices reached for the first time go to nq/neo/nwst (and nbits when given).
// mark: the value written to `parents` is the level r instead of the parent.
__device__ __noinline__ void push_level(const uint32_t* __restrict__ off, const uint32_t* __restrict__ idx,
                                        int32_t* parents, int32_t* levels, const uint32_t* q, const uint32_t* eo,
                                        const uint32_t* wst, uint32_t* nq, uint32_t* neo, uint32_t* nwst, uint64_t k,
                                        uint64_t E, uint32_t n, int32_t r, int mark, unsigned long long* packed,
                                        unsigned long long* zeros, uint32_t* nbits, PushShared* s) {
  const int tid = threadIdx.x;
  const uint64_t windows = (E + kLoopThreads - 1) / kLoopThreads;
  for (uint64_t w = blockIdx.x; w < windows; w += gridDim.x) {
    const uint64_t base = w * kLoopThreads, last = base + kLoopThreads < E ? base + kLoopThreads - 1 : E - 1;
    // Stage the slots this window touches: the one holding its first edge,
    // then (every slot has >= 1 edge) at most kLoopThreads - 1 more.
    const uint64_t sl = (uint64_t)wst[w] + tid;
    const bool have = sl < k;
    const uint32_t e = have ? eo[sl] : 0xffffffffu;
    const uint32_t v = have ? q[sl] : 0u;
    const bool mine = have && e <= last;
    s->eo[tid] = e;
    if (mine) {
      s->v[tid] = v;
      s->beg[tid] = off[v];
    }
    const int ns = __syncthreads_count(mine);
    const uint64_t t = base + tid;
    bool add = false;
    uint32_t u = 0, deg = 0;
    if (t <= last) {
      int a = 0, b = ns - 1;  // the last staged slot whose offset is <= t
      while (a < b) {
        const int mid = (a + b + 1) >> 1;
        if (s->eo[mid] <= t)
          a = mid;
        else
          b = mid - 1;
      }
      u = idx[s->beg[a] + (uint32_t)(t - s->eo[a])];
      if (__ldcg(parents + u) == -1) {
        // the degree is loaded beside the claim, not after it
        const uint32_t d0 = __ldg(off + u), d1 = __ldg(off + u + 1);
        if (atomicCAS(parents + u, -1, mark ? r : (int32_t)s->v[a]) == -1) {
          add = true;
          if (levels) levels[u] = r;
          deg = d1 - d0;
        }
      }
    }
    block_append(add, u, deg, nq, neo, nwst, n, packed, zeros, nbits, s->scan, s->base);
    __syncthreads();
  }
}

// Level 0's queue: the input frontier's vertices with out-edges, with offsets.
__global__ void k_loop_seed(const uint32_t* in_q, uint64_t k, const uint32_t* off, uint32_t* q0, uint32_t* eo0,
                            uint32_t* wst0, uint32_t n, LoopState* st) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i0 = (uint64_t)blockIdx.x * blockDim.x; i0 < k; i0 += stride) {  // warp-uniform trip count
    const uint64_t i = i0 + threadIdx.x;
    uint32_t v = 0, deg = 0;
    if (i < k) {
      v = in_q[i];
      deg = off[v + 1] - off[v];
    }
    loop_append(i < k && deg > 0, v, deg, q0, eo0, wst0, n, &st->slot[0].packed, &st->slot[0].zeros);
  }
}

__global__ void __launch_bounds__(kLoopThreads) k_bfs_push_loop(const uint32_t* __restrict__ off,
                                                                const uint32_t* __restrict__ idx, int32_t* parents,
                                                                int32_t* levels, uint32_t* q0, uint32_t* q1,
                                                                uint32_t* eo0, uint32_t* eo1, uint32_t* wst0,
                                                                uint32_t* wst1, uint32_t n, LoopState* st,
                                                                int32_t round0, unsigned long long threshold,
                                                                int32_t max_levels, unsigned wait_budget) {
  __shared__ PushShared s_push;
  __shared__ unsigned long long s_rd[5];
  __shared__ int s_ok;
  const int tid = threadIdx.x;
  if (tid == 0) read_slot(&st->slot[0], s_rd);
  __syncthreads();
  unsigned long long pk = s_rd[0];
  unsigned target = 0;
  for (int32_t i = 0; i < max_levels; ++i) {
    const int nxt = (i + 1) % 3, old = (i + 2) % 3;
    const uint32_t* q = (i & 1) ? q1 : q0;
    const uint32_t* eo = (i & 1) ? eo1 : eo0;
    uint32_t* nq = (i & 1) ? q0 : q1;
    uint32_t* neo = (i & 1) ? eo0 : eo1;
    const uint64_t k = pk >> 32;
    const uint64_t E = pk & 0xffffffffull;
    if (blockIdx.x == 0 && tid == 0) {  // counters of level i+2's frontier; nobody touches them in level i
      st->slot[old].packed = 0;
      st->slot[old].zeros = 0;
      st->trav += E;
    }
    const int32_t r = round0 + i;
    push_level(off, idx, parents, levels, q, eo, (i & 1) ? wst1 : wst0, nq, neo, (i & 1) ? wst0 : wst1, k, E, n, r, 0,
               &st->slot[nxt].packed, &st->slot[nxt].zeros, nullptr, &s_push);
    target += gridDim.x;
    if (!grid_barrier(&st->bar, target, wait_budget, &s_ok, &st->slot[nxt], s_rd)) {
      if (tid == 0) atomicExch(&st->exit_reason, -1);
      return;
    }
    pk = s_rd[0];
    const unsigned long long nk = (pk >> 32) + s_rd[1];
    const unsigned long long nE = pk & 0xffffffffull;
    const int reason = nk == 0 ? 1 : (nk + nE > threshold ? 2 : 0);
    if (reason) {
      if (blockIdx.x == 0 && tid == 0) {
        st->levels_done = i + 1;
        atomicCAS(&st->exit_reason, 0, reason);  // a timeout (-1) recorded by any CTA stays
      }
      return;
    }
  }
  if (blockIdx.x == 0 && tid == 0) {
    st->levels_done = max_levels;
    atomicCAS(&st->exit_reason, 0, 3);
  }
}

// Runs sparse BFS levels from frontier *F (its size plus out-degree at most
// `threshold`) on the device.  On return *F holds the next frontier (queue
// form, every vertex of it), *rounds the levels run and *trav their out-degree
// sum.
int bfs_device_levels(gg_graph_s* g, gg_frontier_s** F, int32_t* parents, int32_t* levels, int32_t round0,
                      uint64_t threshold, int32_t* rounds, uint64_t* trav) {
  gg_frontier_s* in = *F;
  const uint32_t n = g->n;
  if (!in->has_sparse) GG_TRY(frontier_to_sparse(in));
  static DeviceOnce occ;
  const int per_sm = occ.get(g->device, [dev = g->device]() {
    int coop = 0, b = 0;
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    if (!coop || cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_bfs_push_loop, kLoopThreads, 0) != cudaSuccess || b < 1)
      return -1;
    return b;
  });
  if (per_sm < 1) return fail(GG_ERR_UNSUPPORTED, "no cooperative launch of the BFS level loop on this device");
  gg_frontier_s *fa = nullptr, *fb = nullptr;
  GG_TRY(frontier_new(g, &fa));
  int rc = frontier_new(g, &fb);
  if (!rc) rc = frontier_ensure_queue(fa);
  if (!rc) rc = frontier_ensure_queue(fb);
  DevBuf<uint32_t> eo0, eo1, wst;
  const uint64_t windows = g->m / kLoopThreads + 2;
  if (!rc) rc = eo0.alloc(g, n);
  if (!rc) rc = eo1.alloc(g, n);
  if (!rc) rc = wst.alloc(g, 2 * windows);
  if (rc) {
    frontier_free(fa);
    frontier_free(fb);
    return rc;
  }
  LoopState* d_st = reinterpret_cast<LoopState*>(g->ws.d_loop);
  LoopState h{};
  cudaError_t e = cudaMemsetAsync(d_st, 0, sizeof(LoopState), g->stream);
  if (e == cudaSuccess) {
    k_loop_seed<<<generic_grid(g, in->dm), kGenericThreads, 0, g->stream>>>(in->d_queue, in->dm, g->out_off(),
                                                                            fa->d_queue, eo0.p, wst.p, n, d_st);
    e = cudaGetLastError();
  }
  // a few CTAs per SM (2 unless set): sparse levels are small, and every CTA joins each barrier
  const int grid = g->num_sms * std::min(per_sm, g->loop_ctas_per_sm > 0 ? g->loop_ctas_per_sm : 2);
  const uint32_t* off = g->out_off();
  const uint32_t* idx = g->out_idx();
  uint32_t* q0 = fa->d_queue;
  uint32_t* q1 = fb->d_queue;
  uint32_t* e0 = eo0.p;
  uint32_t* e1 = eo1.p;
  uint32_t* w0 = wst.p;
  uint32_t* w1 = wst.p + windows;
  uint32_t nn = n;
  unsigned long long thr = threshold;
  int32_t cap = 1 << 20;
  unsigned budget = g->loop_wait_budget;
  void* args[] = {(void*)&off, (void*)&idx, (void*)&parents, (void*)&levels, (void*)&q0, (void*)&q1, (void*)&e0,
                  (void*)&e1, (void*)&w0, (void*)&w1, (void*)&nn, (void*)&d_st, (void*)&round0, (void*)&thr,
                  (void*)&cap, (void*)&budget};
  if (e == cudaSuccess)
    e = cudaLaunchCooperativeKernel((const void*)k_bfs_push_loop, grid, kLoopThreads, args, 0, g->stream);
  int rr = GG_OK;
  if (e == cudaSuccess) rr = read_small(g, &h, d_st);
  g->kernels += 2;
  if (e != cudaSuccess || rr != GG_OK || h.exit_reason < 0) {
    frontier_free(fa);
    frontier_free(fb);
    if (e != cudaSuccess) return fail(GG_ERR_CUDA, "BFS level loop: %s", cudaGetErrorString(e));
    if (rr != GG_OK) return rr;
    return fail(GG_ERR_TIMEOUT, "BFS level loop: a grid barrier wait ran out");
  }
  const int32_t L = h.levels_done;
  // level L-1 appended into queue (L & 1): fb when L is odd, fa when even
  gg_frontier_s* res = (L & 1) ? fb : fa;
  gg_frontier_s* dead = res == fa ? fb : fa;
  const LoopSlot& last = h.slot[L % 3];
  const uint64_t K = last.packed >> 32, Z = last.zeros;
  if (Z) {  // the vertices without out-edges move from the far end next to the others
    e = cudaMemcpyAsync(res->d_queue + K, res->d_queue + (n - Z), 4 * Z, cudaMemcpyDeviceToDevice, g->stream);
    if (e != cudaSuccess) {
      frontier_free(fa);
      frontier_free(fb);
      return fail(GG_ERR_CUDA, "BFS level loop: %s", cudaGetErrorString(e));
    }
  }
  res->has_sparse = true;
  res->has_dense = false;
  res->bit = false;
  res->dm = K + Z;
  res->out_edges = last.packed & 0xffffffffull;
  frontier_free(dead);
  frontier_free(in);
  *F = res;
  *rounds = L;
  *trav = h.trav;
  return GG_OK;
}

// ===================================================== every level on device
// The whole BFS (app/BFS.C:77-101) in one cooperative launch: after each
// level's grid barrier every CTA reads the next frontier's size and
// out-degree and applies edgeMap's direction rule itself
// (graphgrind/ligra-numa.h:953: size + out-degree > threshold is dense).
// A dense level runs bottom-up over the in-edges with early exit
// (edgeMapDenseCSC with BFS_F, :608-626: a destination takes its first
// frontier in-neighbour), a sparse level runs top-down over the queue
// (push_level).  Every frontier keeps a bitmap (the dense step's input);
// a sparse level also builds its successor's queue, and a dense level whose
// successor is sparse builds that queue from its bitmap in two more grid
// phases (per-CTA counts, then each CTA writes its vertices at the prefix of
// the counts before it, in id order).  Three bitmaps rotate: the one of the
// level before the current is cleared while the current level runs.
// One bottom-up level, this CTA's share (warps over 32-vertex groups, grid
// stride): a vertex without a parent takes its first in-neighbour that is in
// the frontier bitmap bcur and joins bnxt.  *cnt / *deg: this thread's new
// vertices and their out-degree sum.  Not inlined: the loop then keeps its
// registers whatever the rest of the level-loop kernel holds.
// vec: the in-list is read in 16-byte aligned groups of 4 edges (the edge
// arrays are 16-byte aligned and padded past their end), the group's 4
// frontier tests issued together; the first hit in list order still wins.
__device__ __noinline__ void bottom_up_level(const uint32_t* __restrict__ off, const uint32_t* __restrict__ ioff,
                                             const uint32_t* __restrict__ iidx, int32_t* parents, int32_t* levels,
                                             const uint32_t* bcur, uint32_t* bnxt, uint32_t n, int32_t r,
                                             int mark, uint32_t* cnt, uint32_t* deg, int vec) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t stride = gridDim.x * blockDim.x;  // <= 2^31 threads
  uint32_t c = 0, dg = 0;
  uint32_t b = blockIdx.x * blockDim.x + (threadIdx.x & ~31u);
  // Loads run ahead of the walk: a lane's parent word and in-list bounds two
  // groups ahead, its first in-neighbour one group ahead, so that they arrive
  // while the current group walks its in-lists (a vertex is this lane's alone
  // during a bottom-up level: nobody else writes its parent).
  auto load = [&](uint32_t bb, int32_t& pv, uint32_t& j0, uint32_t& e1) {
    const uint32_t v = bb + lane;
    pv = 0;
    j0 = e1 = 0;
    if (v < n) {
      pv = __ldcg(parents + v);
      j0 = ioff[v];
      e1 = ioff[v + 1];
    }
  };
  auto first = [&](int32_t pv, uint32_t j0, uint32_t e1) -> uint32_t {
    return (pv == -1 && j0 < e1) ? iidx[j0] : 0u;
  };
  // groups b (pv, j0, e1, s0) and b + stride (pv1, j1, e11)
  int32_t pv = 0, pv1 = 0;
  uint32_t j0 = 0, e1 = 0, j1 = 0, e11 = 0, s0 = 0;
  if (b < n) load(b, pv, j0, e1);
  if ((uint64_t)b + stride < n) load(b + stride, pv1, j1, e11);
  if (b < n) s0 = first(pv, j0, e1);
  for (; b < n; b += stride) {
    const bool last = (uint64_t)b + stride >= n;  // no group after this one
    int32_t pv2 = 0;
    uint32_t j2 = 0, e2 = 0, s1 = 0;
    if ((uint64_t)b + 2ull * stride < n) load(b + 2 * stride, pv2, j2, e2);
    if (!last) s1 = first(pv1, j1, e11);
    const uint32_t v = b + lane;
    bool act = false;
    if (v < n && pv == -1 && j0 < e1) {
      if ((bcur[s0 >> 5] >> (s0 & 31)) & 1u) {
        parents[v] = mark ? r : (int32_t)s0;
        if (levels) levels[v] = r;
        act = true;
      } else if (vec) {
        for (uint32_t a = (j0 + 1) & ~3u; a < e1; a += 4) {
          const uint4 q = __ldg(reinterpret_cast<const uint4*>(iidx + a));
          const uint32_t ss[4] = {q.x, q.y, q.z, q.w};
          int hit = -1;
#pragma unroll
          for (int t = 3; t >= 0; --t) {
            const uint32_t e = a + (uint32_t)t;
            if (e > j0 && e < e1 && ((bcur[ss[t] >> 5] >> (ss[t] & 31)) & 1u)) hit = t;
          }
          if (hit >= 0) {
            parents[v] = mark ? r : (int32_t)ss[hit];
            if (levels) levels[v] = r;
            act = true;
            break;
          }
        }
      } else {
        for (uint32_t j = j0 + 1; j < e1; ++j) {
          const uint32_t s = iidx[j];
          if ((bcur[s >> 5] >> (s & 31)) & 1u) {
            parents[v] = mark ? r : (int32_t)s;
            if (levels) levels[v] = r;
            act = true;
            break;
          }
        }
      }
    }
    const uint32_t word = __ballot_sync(0xffffffffu, act);
    if (act) dg += off[v + 1] - off[v];
    if (lane == 0 && word) {
      atomicOr(bnxt + (b >> 5), word);
      c += __popc(word);
    }
    if (last) break;
    pv = pv1;
    j0 = j1;
    e1 = e11;
    s0 = s1;
    pv1 = pv2;
    j1 = j2;
    e11 = e2;
  }
  *cnt = c;
  *deg = dg;
}

// The start of a BFS in one pass: parents (and levels) unreached but for the
// source, the bitmaps and the loop state clear, level 0's queue.
__global__ void k_bfs_full_init(uint32_t n, uint32_t start, const uint32_t* off, int32_t* parents, int32_t* levels,
                                uint32_t* q0, uint32_t* eo0, uint32_t* wst0, uint32_t* bits, uint32_t bit_words,
                                LoopState* st) {
  const uint64_t t0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = t0; i < n; i += stride) {
    parents[i] = i == start ? (int32_t)start : -1;
    if (levels) levels[i] = i == start ? 0 : -1;
  }
  for (uint64_t w = t0; w < bit_words; w += stride) bits[w] = w == (start >> 5) ? 1u << (start & 31) : 0u;
  const uint32_t d = off[start + 1] - off[start];
  for (uint64_t w = t0; w * kLoopThreads < d; w += stride) wst0[w] = 0;
  if (t0 == 0) {
    *st = LoopState{};
    q0[0] = start;
    eo0[0] = 0;
    if (d > 0)
      st->slot[0].packed = (1ull << 32) | d;
    else
      st->slot[0].zeros = 1;
  }
}

// Sums of five values over the CTA, returned to every thread.
__device__ __forceinline__ void block_sum5(unsigned long long* v, unsigned long long (*s_red)[kLoopWarps]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int j = 0; j < 5; ++j) v[j] = warp_sum(v[j]);
  __syncthreads();
  if (lane == 0)
#pragma unroll
    for (int j = 0; j < 5; ++j) s_red[j][warp] = v[j];
  __syncthreads();
#pragma unroll
  for (int j = 0; j < 5; ++j) {
    unsigned long long t = 0;
    for (int w = 0; w < kLoopWarps; ++w) t += s_red[j][w];
    v[j] = t;
  }
}

__global__ void __launch_bounds__(kLoopThreads, 2048 / kLoopThreads)
    k_bfs_full(const uint32_t* __restrict__ off, const uint32_t* __restrict__ idx, const uint32_t* __restrict__ ioff,
               const uint32_t* __restrict__ iidx, int32_t* parents, int32_t* levels, uint32_t* q0, uint32_t* q1,
               uint32_t* eo0, uint32_t* eo1, uint32_t* wst0, uint32_t* wst1, uint32_t* bits, uint32_t wstride,
               unsigned long long* cta, uint32_t n, LoopState* st, int32_t round0, unsigned long long threshold,
               int32_t max_levels, unsigned wait_budget, int bu_vec, int mark, unsigned long long handover) {
  __shared__ PushShared s_push;
  __shared__ unsigned long long s_red[5][kLoopWarps];
  __shared__ unsigned long long s_rd[5];
  __shared__ int s_ok;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t nw = (n + 31) / 32;
  const uint32_t wper = (nw + gridDim.x - 1) / gridDim.x;
  const uint32_t w0 = min(nw, blockIdx.x * wper), w1 = min(nw, w0 + wper);
  // s_rd holds the current frontier's counters (slot layout), from one level to the next
  if (tid == 0) read_slot(&st->slot[0], s_rd);
  __syncthreads();
  unsigned target = 0;
  for (int32_t i = 0; i < max_levels; ++i) {
    const int cur = i % 3, nxt = (i + 1) % 3, old = (i + 2) % 3;
    const int rep = (int)s_rd[4];
    const unsigned long long pk = s_rd[0];
    const uint32_t* q = (i & 1) ? q1 : q0;
    const uint32_t* eo = (i & 1) ? eo1 : eo0;
    uint32_t* nq = (i & 1) ? q0 : q1;
    uint32_t* neo = (i & 1) ? eo0 : eo1;
    uint32_t* nwst = (i & 1) ? wst0 : wst1;
    const uint32_t* bcur = bits + (size_t)cur * wstride;
    uint32_t* bnxt = bits + (size_t)nxt * wstride;
    uint32_t* bold = bits + (size_t)old * wstride;
    const uint64_t k = rep == 0 ? pk >> 32 : 0;
    const uint64_t E = rep == 0 ? pk & 0xffffffffull : s_rd[3];
    const uint64_t nk = rep == 0 ? k + s_rd[1] : s_rd[2];
    if (blockIdx.x == 0 && tid == 0) {  // counters of level i+2's frontier; nobody touches them in level i
      LoopSlot& o = st->slot[old];
      o.packed = 0;
      o.zeros = 0;
      o.dcnt = 0;
      o.ddeg = 0;
      st->trav += E;
    }
    for (uint32_t w = w0 + tid; w < w1; w += blockDim.x) bold[w] = 0u;  // level i-1's frontier, done with
    const int32_t r = round0 + i;
    if (nk + E > threshold) {
      // bottom-up: one lane per destination, the first frontier in-neighbour wins
      uint32_t c32 = 0, dg32 = 0;
      bottom_up_level(off, ioff, iidx, parents, levels, bcur, bnxt, n, r, mark, &c32, &dg32, bu_vec);
      unsigned long long c = warp_sum((unsigned long long)c32), dg = warp_sum((unsigned long long)dg32);
      if (lane == 0) {
        s_red[0][warp] = c;
        s_red[1][warp] = dg;
      }
      __syncthreads();
      if (tid == 0) {
        unsigned long long tc = 0, td = 0;
        for (int w = 0; w < kLoopWarps; ++w) {
          tc += s_red[0][w];
          td += s_red[1][w];
        }
        if (tc) atomicAdd(&st->slot[nxt].dcnt, tc);
        if (td) atomicAdd(&st->slot[nxt].ddeg, td);
        if (blockIdx.x == 0) st->slot[nxt].rep = 1;
      }
    } else {
      push_level(off, idx, parents, levels, q, eo, (i & 1) ? wst1 : wst0, nq, neo, nwst, k, E, n, r, mark,
                 &st->slot[nxt].packed, &st->slot[nxt].zeros, bnxt, &s_push);
      if (blockIdx.x == 0 && tid == 0) st->slot[nxt].rep = 0;
    }
    target += gridDim.x;
    if (!grid_barrier(&st->bar, target, wait_budget, &s_ok, &st->slot[nxt], s_rd)) {
      if (tid == 0) atomicExch(&st->exit_reason, -1);
      return;
    }
    const int nrep = (int)s_rd[4];
    const unsigned long long npk = s_rd[0];
    const unsigned long long nk2 = nrep == 0 ? (npk >> 32) + s_rd[1] : s_rd[2];
    const unsigned long long nE = nrep == 0 ? npk & 0xffffffffull : s_rd[3];
    // a frontier this small that grows by less than four times goes back to the caller, for good
    const bool give = nk2 + nE < handover && nE < 4 * E;
    if (nk2 == 0 || give) {
      if (blockIdx.x == 0 && tid == 0) {
        st->levels_done = i + 1;
        atomicCAS(&st->exit_reason, 0, nk2 == 0 ? 1 : 4);  // a timeout (-1) recorded by any CTA stays
      }
      return;
    }
    if (nrep == 1 && nk2 + nE <= threshold) {
      // the next level pushes: its queue from the bitmap, vertices with
      // out-edges in id order (phase A: this CTA's counts of its words)
      unsigned long long v5[5] = {0, 0, 0, 0, 0};
      for (uint32_t w = w0 + tid; w < w1; w += blockDim.x) {
        uint32_t x = bnxt[w];
        while (x) {
          const uint32_t v = w * 32 + (__ffs(x) - 1);
          x &= x - 1;
          const uint32_t d = off[v + 1] - off[v];
          if (d) {
            ++v5[0];
            v5[1] += d;
          } else {
            ++v5[2];
          }
        }
      }
      block_sum5(v5, s_red);
      if (tid < 3) cta[(size_t)blockIdx.x * 3 + tid] = v5[tid];
      target += gridDim.x;
      if (!grid_barrier(&st->bar, target, wait_budget, &s_ok)) {
        if (tid == 0) atomicExch(&st->exit_reason, -1);
        return;
      }
      // phase B: the counts of the CTAs before this one and of all, then the writes
      unsigned long long t5[5] = {0, 0, 0, 0, 0};  // before: slots, edges; all: slots, edges, zeros
      for (uint32_t c2 = tid; c2 < gridDim.x; c2 += blockDim.x) {
        const unsigned long long x0 = cta[(size_t)c2 * 3], x1 = cta[(size_t)c2 * 3 + 1],
                                 x2 = cta[(size_t)c2 * 3 + 2];
        if (c2 < blockIdx.x) {
          t5[0] += x0;
          t5[1] += x1;
        }
        t5[2] += x0;
        t5[3] += x1;
        t5[4] += x2;
      }
      block_sum5(t5, s_red);
      unsigned long long base_p = t5[0], base_d = t5[1];
      // words in chunks of a CTA's threads, one per thread, in order
      for (uint32_t c0 = w0; c0 < w1; c0 += blockDim.x) {
        const uint32_t w = c0 + tid;
        const uint32_t x = w < w1 ? bnxt[w] : 0u;
        uint32_t mp = 0, md = 0;
        bool hub = false;
        uint32_t y = x;
        while (y) {
          const uint32_t v = w * 32 + (__ffs(y) - 1);
          y &= y - 1;
          const uint32_t d = off[v + 1] - off[v];
          if (d) {
            ++mp;
            md += d;
            hub |= d > kHubEdges;
          }
        }
        // slots and edges of the words before (at most 32 kLoopThreads slots)
        unsigned long long tot;
        const unsigned long long ex = block_scan(((unsigned long long)mp << 32) | md, &tot, s_push.scan);
        __syncthreads();
        uint32_t slot = (uint32_t)base_p + (uint32_t)(ex >> 32), eoff = (uint32_t)base_d + (uint32_t)ex;
        y = x;
        if (!__any_sync(0xffffffffu, hub)) {
          while (y) {
            const uint32_t v = w * 32 + (__ffs(y) - 1);
            y &= y - 1;
            const uint32_t d = off[v + 1] - off[v];
            if (d) {
              nq[slot] = v;
              neo[slot] = eoff;
              note_windows(nwst, slot, eoff, d);
              ++slot;
              eoff += d;
            }
          }
        } else {
          while (__any_sync(0xffffffffu, y != 0)) {
            uint32_t d = 0;
            if (y) {
              const uint32_t v = w * 32 + (__ffs(y) - 1);
              y &= y - 1;
              d = off[v + 1] - off[v];
              if (d) {
                nq[slot] = v;
                neo[slot] = eoff;
              }
            }
            note_windows_warp(nwst, d != 0, slot, eoff, d);
            slot += d != 0;
            eoff += d;
          }
        }
        base_p += tot >> 32;
        base_d += (uint32_t)tot;
      }
      // every CTA holds the totals (the next level's counters); the slot records them as well
      if (tid == 0) {
        s_rd[0] = (t5[2] << 32) | t5[3];
        s_rd[1] = t5[4];
        s_rd[4] = 0;
        if (blockIdx.x == 0) {
          st->slot[nxt].packed = s_rd[0];
          st->slot[nxt].zeros = s_rd[1];
          st->slot[nxt].rep = 0;
        }
      }
      target += gridDim.x;
      if (!grid_barrier(&st->bar, target, wait_budget, &s_ok)) {
        if (tid == 0) atomicExch(&st->exit_reason, -1);
        return;
      }
    }
  }
  if (blockIdx.x == 0 && tid == 0) {
    st->levels_done = max_levels;
    atomicCAS(&st->exit_reason, 0, 3);
  }
}

// CTAs of the all-levels loop: every warp slot unless set (the bottom-up
// levels are latency-bound), but no more than the graph has work for: a CTA
// that only joins the barriers delays them (R-MAT-10: 53 us with every slot).
static int full_grid(int num_sms, int ctas_per_sm, uint64_t n, uint64_t m) {
  return (int)std::min<uint64_t>((uint64_t)num_sms * ctas_per_sm,
                                 std::max<uint64_t>(1, (n + m / 8) / (2 * kLoopThreads)));
}

// CTAs per SM that k_bfs_full can have resident in a cooperative launch; -1 if none.
static int full_occupancy(int device) {
  static DeviceOnce occ;
  return occ.get(device, [device]() {
    int coop = 0, b = 0;
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device);
    if (!coop || cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_bfs_full, kLoopThreads, 0) != cudaSuccess || b < 1)
      return -1;
    return b;
  });
}

// The buffers of one BFS inside its arena: *parents and, when want_levels,
// *levels (n entries each), then the loop's own.
struct FullBufs {
  unsigned long long* cta;
  int32_t *par, *lev;
  uint32_t *q0, *q1, *eo0, *eo1, *wst0, *wst1, *bits;
  uint32_t wstride;
  int grid;
  uint64_t words;  // of the whole arena
};

static int full_bufs(const gg_graph_s* g, bool want_levels, uint32_t* arena, FullBufs* out) {
  const int per_sm = full_occupancy(g->device);
  if (per_sm < 1) return fail(GG_ERR_UNSUPPORTED, "no cooperative launch of the BFS loop on this device");
  const int ctas = std::min(per_sm, g->loop_ctas_per_sm > 0 ? g->loop_ctas_per_sm : 2048 / kLoopThreads);
  FullBufs b{};
  b.grid = full_grid(g->num_sms, ctas, g->n, g->m);
  b.wstride = (g->words() + 31) & ~31u;  // 128-byte aligned bitmaps
  const uint64_t na = ((uint64_t)g->n + 63) & ~63ull, wa = (g->m / kLoopThreads + 2 + 63) & ~63ull;
  auto take = [&](uint64_t count) {
    uint32_t* r = arena ? arena + b.words : nullptr;
    b.words += count;
    return r;
  };
  b.cta = reinterpret_cast<unsigned long long*>(take(((uint64_t)b.grid * 6 + 63) & ~63ull));
  b.par = reinterpret_cast<int32_t*>(take(na));
  if (want_levels) b.lev = reinterpret_cast<int32_t*>(take(na));
  b.q0 = take(na);
  b.q1 = take(na);
  b.eo0 = take(na);
  b.eo1 = take(na);
  b.wst0 = take(wa);
  b.wst1 = take(wa);
  b.bits = take(3ull * b.wstride);
  *out = b;
  return GG_OK;
}

int bfs_device_full_prepare(gg_graph_s* g, bool want_levels, DevBuf<uint32_t>& arena) {
  FullBufs b;
  GG_TRY(full_bufs(g, want_levels, nullptr, &b));
  GG_TRY(arena.alloc(g, b.words));
  // the bottom-up levels walk the in-lists hub sources first (same edges,
  // other order: a vertex then meets a frontier in-neighbour sooner), where the
  // caller has asked for that copy (graphs it cannot be built for, past 2^31
  // edges or without the memory, walk the CSC's own in-lists).  It is not built
  // unasked: it costs a segmented sort of all edges and its temporaries, which
  // takes thousands of traversals to earn back (17 ms on R-MAT-22 against a
  // loop of 172 instead of 176 us, on R-MAT-24 433 instead of 447 us; on
  // Erdos-Renyi graphs the loop is slower with it, 281 against 275 us).
  if (g->bu_wanted && !g->d_bu_idx && build_bu_index(g) != GG_OK) cudaGetLastError();
  g->bu_wanted = false;
  return GG_OK;
}

// Enqueues every level of the BFS from `start` as one cooperative launch
// (k_bfs_full) on the graph's stream and returns without waiting; `arena` comes
// from bfs_device_full_prepare.  bfs_device_full_begin_result queues the
// read-back of the outcome, which bfs_device_full_result takes once the stream
// has passed it.
int bfs_device_full(gg_graph_s* g, uint32_t start, bool want_levels, DevBuf<uint32_t>& arena, int32_t** parents,
                    int32_t** levels, uint64_t threshold) {
  const uint32_t n = g->n;
  FullBufs b;
  GG_TRY(full_bufs(g, want_levels, arena.p, &b));
  LoopState* d_st = reinterpret_cast<LoopState*>(g->ws.d_loop);
  k_bfs_full_init<<<generic_grid(g, n), kGenericThreads, 0, g->stream>>>(n, start, g->out_off(), b.par, b.lev, b.q0,
                                                                         b.eo0, b.wst0, b.bits, 3 * b.wstride, d_st);
  GG_CUDA(cudaGetLastError());
  const uint32_t* off = g->out_off();
  const uint32_t* idx = g->out_idx();
  const uint32_t* ioff = g->in_off();
  const uint32_t* iidx = g->early_kernel == 3 && g->d_bu_idx ? g->d_bu_idx : g->in_idx();
  uint32_t nn = n;
  int32_t round0 = 1;
  unsigned long long thr = threshold;
  int32_t cap = n < (uint32_t)INT32_MAX ? (int32_t)n + 1 : INT32_MAX;
  unsigned budget = g->loop_wait_budget;
  int vec = g->early_kernel >= 2 ? 1 : 0, mark = 0;
  unsigned long long handover = 0;
  void* args[] = {(void*)&off,    (void*)&idx,    (void*)&ioff,   (void*)&iidx,   (void*)&b.par,  (void*)&b.lev,
                  (void*)&b.q0,   (void*)&b.q1,   (void*)&b.eo0,  (void*)&b.eo1,  (void*)&b.wst0, (void*)&b.wst1,
                  (void*)&b.bits, (void*)&b.wstride, (void*)&b.cta, (void*)&nn,   (void*)&d_st,   (void*)&round0,
                  (void*)&thr,    (void*)&cap,    (void*)&budget, (void*)&vec,    (void*)&mark,   (void*)&handover};
  GG_CUDA(cudaLaunchCooperativeKernel((const void*)k_bfs_full, b.grid, kLoopThreads, args, 0, g->stream));
  g->kernels += 2;
  *parents = b.par;
  *levels = b.lev;
  return GG_OK;
}

int bfs_device_full_begin_result(gg_graph_s* g) {
  return read_small_begin(g, reinterpret_cast<const LoopState*>(g->ws.d_loop));
}

// The outcome of the BFS bfs_device_full enqueued, after the stream has passed
// bfs_device_full_begin_result: *rounds, the number of edgeMap rounds (the last
// one finds nothing), *trav, the out-degree sum of the frontiers processed.
int bfs_device_full_result(gg_graph_s* g, int32_t* rounds, uint64_t* trav) {
  LoopState h{};
  read_small_end(g, &h);
  if (h.exit_reason < 0) return fail(GG_ERR_TIMEOUT, "BFS loop: a grid barrier wait ran out");
  if (h.exit_reason != 1)
    return fail(GG_ERR_CUDA, "BFS loop: stopped without an empty frontier (reason %d)", h.exit_reason);
  *rounds = h.levels_done;
  *trav = h.trav;
  return GG_OK;
}

// ================================================== many graphs side by side
// The loop's buffers inside a union's arena.
struct UnionBufs {
  unsigned long long* cta;
  LoopState* st;
  uint32_t *q0, *q1, *eo0, *eo1, *wst0, *wst1, *bits;
  uint32_t wstride;
  uint64_t words;  // of the whole arena
};

static UnionBufs union_bufs(const UnionBfs& u) {
  UnionBufs b{};
  const uint64_t na = ((uint64_t)u.n + 63) & ~63ull, wa = (u.m / kLoopThreads + 2 + 63) & ~63ull;
  b.wstride = ((u.n + 31) / 32 + 31) & ~31u;
  uint32_t* at = u.arena;
  auto take = [&](uint64_t count) {
    uint32_t* r = at ? at + b.words : nullptr;
    b.words += count;
    return r;
  };
  b.st = reinterpret_cast<LoopState*>(take(128));
  b.cta = reinterpret_cast<unsigned long long*>(take(((uint64_t)u.grid * 6 + 63) & ~63ull));
  b.q0 = take(na);
  b.q1 = take(na);
  b.eo0 = take(na);
  b.eo1 = take(na);
  b.wst0 = take(wa);
  b.wst1 = take(wa);
  b.bits = take(3ull * b.wstride);
  return b;
}

int union_bfs_prepare(UnionBfs& u, int device, int num_sms) {
  const int per_sm = full_occupancy(device);
  if (per_sm < 1) return fail(GG_ERR_UNSUPPORTED, "no cooperative launch of the BFS loop on this device");
  u.grid = full_grid(num_sms, std::min(per_sm, 2048 / kLoopThreads), u.n, u.m);
  GG_CUDA(cudaMalloc(&u.arena, 4 * union_bufs(u).words));
  u.st = union_bufs(u).st;
  return GG_OK;
}

void union_bfs_free(UnionBfs& u) {
  cudaFree(u.arena);
  u.arena = nullptr;
}

__global__ void k_union_init(uint32_t n, int32_t* levels, uint32_t* bits, uint32_t bit_words, LoopState* st) {
  const uint64_t t0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = t0; i < n; i += stride) levels[i] = -1;
  for (uint64_t w = t0; w < bit_words; w += stride) bits[w] = 0;
  if (t0 == 0) *st = LoopState{};
}

__global__ void k_union_seed(const uint32_t* seeds, uint32_t count, const uint32_t* off, int32_t* levels, uint32_t n,
                             uint32_t* q0, uint32_t* eo0, uint32_t* wst0, uint32_t* bits, LoopState* st) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t v = 0, deg = 0;
  if (i < count) {
    v = seeds[i];
    deg = off[v + 1] - off[v];
    levels[v] = 0;
    atomicOr(bits + (v >> 5), 1u << (v & 31));
  }
  loop_append(i < count, v, deg, q0, eo0, wst0, n, &st->slot[0].packed, &st->slot[0].zeros);
}

int union_bfs_enqueue(const UnionBfs& u, cudaStream_t s, int num_sms, const uint32_t* seeds, uint32_t count) {
  const UnionBufs b = union_bufs(u);
  k_union_init<<<num_sms * 8, kGenericThreads, 0, s>>>(u.n, u.levels, b.bits, 3 * b.wstride, b.st);
  k_union_seed<<<(count + 255) / 256, 256, 0, s>>>(seeds, count, u.off, u.levels, u.n, b.q0, b.eo0, b.wst0, b.bits,
                                                   b.st);
  GG_CUDA(cudaGetLastError());
  int32_t* lev = u.levels;
  int32_t* none = nullptr;
  uint32_t ws = b.wstride, nn = u.n;
  int32_t round0 = 1, cap = u.n < (uint32_t)INT32_MAX ? (int32_t)u.n + 1 : INT32_MAX;
  unsigned long long thr = u.m / 20;  // edgeMap's m/20, over the union
  unsigned budget = u.wait_budget;
  int vec = 1, mark = 1;
  // A level of the whole GPU costs about 10 us, a level inside one CTA per
  // graph about 2.5 us a window: below a window of edges per graph the second
  // is the faster one (256 R-MAT graphs: 0.62 ms with 2048 edges per graph, 0.56 with
  // 512 and with 128).
  unsigned long long handover = (unsigned long long)kLoopThreads * count;
  void* args[] = {(void*)&u.off,  (void*)&u.idx,  (void*)&u.ioff,   (void*)&u.iidx, (void*)&lev,  (void*)&none,
                  (void*)&b.q0,   (void*)&b.q1,   (void*)&b.eo0,    (void*)&b.eo1,  (void*)&b.wst0, (void*)&b.wst1,
                  (void*)&b.bits, (void*)&ws,     (void*)&b.cta,    (void*)&nn,     (void*)&b.st, (void*)&round0,
                  (void*)&thr,    (void*)&cap,    (void*)&budget,   (void*)&vec,    (void*)&mark, (void*)&handover};
  GG_CUDA(cudaLaunchCooperativeKernel((const void*)k_bfs_full, u.grid, kLoopThreads, args, 0, s));
  return GG_OK;
}

}  // namespace gg
