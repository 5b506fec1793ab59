// The all-levels BFS loop (gg_loop.cu) as other files use it: its state, and
// the form that traverses many graphs side by side as one union graph.
#pragma once
#include "gg_runtime.cuh"

namespace gg {

// One frontier's counters; the loops keep three, by level mod 3.
struct LoopSlot {
  // queue form: (slots << 32) | out-edges; vertices with out-edges fill the
  // queue from the front in edge-offset order
  unsigned long long packed;
  unsigned long long zeros;  // queue form: members without out-edges (not among the slots)
  unsigned long long dcnt;   // bitmap form: members
  unsigned long long ddeg;   // bitmap form: their out-degree sum
  int32_t rep;               // 0 queue (and bitmap), 1 bitmap only
  int32_t pad;
};

// State of a device level loop.  The counters are read after each grid
// barrier by one thread per CTA (into shared memory); the barrier's arrival
// word sits on a cache line of its own.
struct LoopState {
  LoopSlot slot[3];
  unsigned long long trav;  // out-edges of the frontiers processed
  alignas(128) unsigned int bar;  // barrier arrivals
  int32_t levels_done;
  int32_t exit_reason;  // 1 empty, 2 next level is dense (sparse loop), 3 level cap, 4 handed over, -1 barrier timeout
};
static_assert(sizeof(LoopState) <= 64 * sizeof(unsigned long long), "loop state exceeds its workspace");

// A union graph (disjoint graphs numbered consecutively) on the device and the
// loop's buffers; the arrays belong to the caller, the buffers are one
// allocation (arena).
struct UnionBfs {
  const uint32_t *off = nullptr, *idx = nullptr;    // out-edges
  const uint32_t *ioff = nullptr, *iidx = nullptr;  // in-edges, 16-byte aligned, padded past their end
  int32_t* levels = nullptr;
  uint32_t n = 0;
  uint64_t m = 0;
  uint32_t* arena = nullptr;
  LoopState* st = nullptr;
  int grid = 0;
  unsigned wait_budget = kWaitBudget;  // probes of a grid barrier's wait
};
// Allocates u's buffers for its n and m; union_bfs_free releases them.
int union_bfs_prepare(UnionBfs& u, int device, int num_sms);
void union_bfs_free(UnionBfs& u);
// Enqueues the BFS of all graphs from seeds[count] (one vertex of each graph,
// device memory) on stream s: every level of all graphs in one cooperative
// launch, until the frontier is empty (exit_reason 1) or has become too small
// for whole-GPU levels (exit_reason 4; `levels` then holds levels_done as the
// largest level).
int union_bfs_enqueue(const UnionBfs& u, cudaStream_t s, int num_sms, const uint32_t* seeds, uint32_t count);

}  // namespace gg
