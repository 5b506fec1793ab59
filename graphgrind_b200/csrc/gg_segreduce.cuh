// Row reductions over a segmented edge stream (CSC in-edges or CSR
// out-edges of the current orientation), eight edges per lane.
#pragma once
#include "gg_runtime.cuh"

namespace gg {

struct SegStream {
  const uint32_t* idx;
  const uint32_t* head;
  const uint32_t* blk;
  const uint32_t* rows;
  uint64_t nblocks, m;
};

__device__ __forceinline__ float seg_shfl_up(float v, int d) { return __shfl_up_sync(0xffffffffu, v, d); }
__device__ __forceinline__ float2 seg_shfl_up(float2 v, int d) {
  return make_float2(__shfl_up_sync(0xffffffffu, v.x, d), __shfl_up_sync(0xffffffffu, v.y, d));
}
__device__ __forceinline__ float seg_shfl(float v, int l) { return __shfl_sync(0xffffffffu, v, l); }
__device__ __forceinline__ float2 seg_shfl(float2 v, int l) {
  return make_float2(__shfl_sync(0xffffffffu, v.x, l), __shfl_sync(0xffffffffu, v.y, l));
}

// For every row: op.flush(row, combine over the row's edges e of
// op.val(op.load(e, y, row), e), complete) with y the edge's other end (if
// Op::kNeedsIdx) and row its own (if Op::kNeedsRow).  One warp per 256-edge
// block.  The pass is bound by the latency of its gathers and by instruction
// issue, so a lane loads four of its 8 edges (edge 32 i + lane: consecutive
// lanes gather for consecutive edges, whose sources share cache lines) before
// it uses any, the edge stream bypasses L1, and a block without a ragged end
// tests no bounds.  The values then change hands through shared memory: lane l
// reduces edges 8 l .. 8 l + 7 in order, and one segmented scan over the lanes
// joins the rows that cross them, instead of a scan per 32 edges.  Four CTAs
// per SM: more of them evict each other's gathered lines (12.6M edges, R-MAT-20,
// forward / backward step: 63 / 77 us with a scan per 32 edges, 54 / 63 us with
// this, 60 / 90 us with five CTAs).  A row that lies inside the block is flushed
// once with complete = true; a row split across blocks is flushed once per
// block with complete = false (the op combines those atomically).
template <class Op>
__global__ void __launch_bounds__(256, 4) k_seg_reduce(SegStream p, Op op) {
  using T = typename Op::T;
  __shared__ uint32_t s_row[8][kSegBlock + 1];
  __shared__ __align__(16) T s_val[8][kSegBlock];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t lanemask_le = 0xffffffffu >> (31 - lane);
  const uint64_t warps = (uint64_t)gridDim.x * (blockDim.x >> 5);
  for (uint64_t b = (uint64_t)blockIdx.x * (blockDim.x >> 5) + warp; b < p.nblocks; b += warps) {
    const uint64_t e0 = b * kSegBlock;
    const uint4 ha = __ldg(reinterpret_cast<const uint4*>(p.head + b * 8));
    const uint4 hb = __ldg(reinterpret_cast<const uint4*>(p.head + b * 8) + 1);
    const uint32_t hw[8] = {ha.x, ha.y, ha.z, ha.w, hb.x, hb.y, hb.z, hb.w};
    const uint32_t h0 = __ldg(p.blk + b), nr = __ldg(p.blk + b + 1) - h0 + 1;
    // the block's values in edge order; FULL: every slot holds an edge
    auto values = [&](auto full) {
      constexpr bool FULL = decltype(full)::value;
      const uint64_t e1 = e0 + lane;
      uint32_t y[8];
#pragma unroll
      for (int i = 0; i < 8; ++i)
        y[i] = Op::kNeedsIdx && (FULL || e1 + 32 * i < p.m) ? ld_stream_u32(p.idx + e1 + 32 * i) : 0u;
      // row of each slot: slot 0 continues from the previous block, one slot per head
      for (uint32_t i = lane; i < nr; i += 32) s_row[warp][i] = (i > 0 || h0 > 0) ? __ldg(p.rows + h0 - 1 + i) : 0u;
      __syncwarp();
      uint32_t running = 0;
#pragma unroll
      for (int i0 = 0; i0 < 8; i0 += 4) {
        typename Op::In in[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint32_t row = Op::kNeedsRow ? s_row[warp][running + __popc(hw[i0 + i] & lanemask_le)] : 0u;
          if (FULL || e1 + 32 * (i0 + i) < p.m) in[i] = op.load(e1 + 32 * (i0 + i), y[i0 + i], row);
          if (Op::kNeedsRow) running += __popc(hw[i0 + i]);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
          s_val[warp][32 * (i0 + i) + lane] =
              FULL || e1 + 32 * (i0 + i) < p.m ? op.val(in[i], e1 + 32 * (i0 + i)) : Op::identity();
      }
    };
    if (e0 + kSegBlock <= p.m)
      values(std::true_type{});
    else
      values(std::false_type{});
    __syncwarp();
    // this lane's 8 consecutive edges: their head bits, and the heads before them
    const int w = lane >> 2, sh = (lane & 3) * 8;
    uint32_t mine = 0, before = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (i < w) before += __popc(hw[i]);
      if (i == w) mine = hw[i];
    }
    before += __popc(mine & ((1u << sh) - 1u));
    const uint32_t bits = (mine >> sh) & 0xffu;
    T v[8];
    const uint4* sv = reinterpret_cast<const uint4*>(&s_val[warp][8 * lane]);
#pragma unroll
    for (int k = 0; k < (int)(8 * sizeof(T) / 16); ++k) reinterpret_cast<uint4*>(v)[k] = sv[k];
    // acc: the run in progress; lead: the one that continues from the lanes before
    T acc = Op::identity(), lead = Op::identity();
    uint32_t rel = before;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if ((bits >> k) & 1u) {
        if (rel == before)
          lead = acc;
        else
          op.flush(s_row[warp][rel], acc, true);
        ++rel;
        acc = v[k];
      } else {
        acc = Op::combine(acc, v[k]);
      }
    }
    // carry: the run in progress at the lane's end, over all its lanes
    const uint32_t hl = __ballot_sync(0xffffffffu, bits != 0) & lanemask_le;
    const int seg0 = hl ? 31 - __clz(hl) : 0;
    T carry = acc;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const T t = seg_shfl_up(carry, d);
      if (lane >= seg0 + d) carry = Op::combine(t, carry);
    }
    const T prev = seg_shfl_up(carry, 1);
    // the run that a lane's first head ends
    if (bits != 0 && (lane > 0 || !(bits & 1u)) && (before > 0 || h0 > 0))
      op.flush(s_row[warp][before], lane > 0 ? Op::combine(prev, lead) : lead, before > 0);
    // the block's last run
    if (lane == 31 && (rel > 0 || h0 > 0)) {
      const uint64_t nb = e0 + kSegBlock;
      const bool ends_block = nb >= p.m || (__ldg(p.head + (nb >> 5)) & 1u);
      op.flush(s_row[warp][rel], carry, rel > 0 && ends_block);
    }
    __syncwarp();
  }
}

// The same with one edge per lane and step: lane l takes edge 32 i + l, and a
// segmented scan per 32 edges combines each row's lanes.  It needs half the
// registers, so twice as many warps hide its latencies.
template <class Op>
__global__ void __launch_bounds__(256) k_seg_scan(SegStream p, Op op) {
  using T = typename Op::T;
  __shared__ uint32_t s_row[8][kSegBlock + 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t lanemask_le = 0xffffffffu >> (31 - lane);
  const uint64_t warps = (uint64_t)gridDim.x * (blockDim.x >> 5);
  for (uint64_t b = (uint64_t)blockIdx.x * (blockDim.x >> 5) + warp; b < p.nblocks; b += warps) {
    const uint64_t e0 = b * kSegBlock;
    // row of each slot: slot 0 continues from the previous block, one slot per head
    const uint32_t h0 = __ldg(p.blk + b), nr = __ldg(p.blk + b + 1) - h0 + 1;
    for (uint32_t i = lane; i < nr; i += 32) s_row[warp][i] = (i > 0 || h0 > 0) ? __ldg(p.rows + h0 - 1 + i) : 0u;
    __syncwarp();
    const uint64_t nb = e0 + kSegBlock;
    const bool ends_block = nb >= p.m || (__ldg(p.head + (nb >> 5)) & 1u);
    uint32_t running = 0;
    T carry = Op::identity();
    uint32_t hw = __ldg(p.head + b * 8);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint32_t hw_next = i < 7 ? __ldg(p.head + b * 8 + i + 1) : 0u;
      const uint64_t e = e0 + 32 * i + lane;
      const uint32_t rel = running + __popc(hw & lanemask_le);
      T v = Op::identity();
      if (e < p.m) v = op.val(op.load(e, Op::kNeedsIdx ? __ldg(p.idx + e) : 0u, s_row[warp][rel]), e);
      const uint32_t hb = hw & lanemask_le;
      const int seg0 = hb ? 31 - __clz(hb) : 0;
      if (lane == 0 && !(hw & 1u)) v = Op::combine(carry, v);
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const T t = seg_shfl_up(v, d);
        if (lane >= seg0 + d) v = Op::combine(t, v);
      }
      const bool ends = lane < 31 ? ((hw >> (lane + 1)) & 1u) : (i < 7 ? (hw_next & 1u) : ends_block);
      if ((ends || (lane == 31 && i == 7)) && (rel > 0 || h0 > 0)) op.flush(s_row[warp][rel], v, rel > 0 && ends);
      const T v31 = seg_shfl(v, 31);
      carry = (i < 7 && !(hw_next & 1u)) ? v31 : Op::identity();
      running += __popc(hw);
      hw = hw_next;
    }
    __syncwarp();
  }
}

// CTAs per SM that a reduction kernel can have resident.
template <class K>
int seg_resident(DeviceOnce& once, int device, K kernel) {
  return once.get(device, [kernel]() {
    int b = 0;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kernel, 256, 0) == cudaSuccess && b > 0 ? b : 1;
  });
}

// One resident wave of CTAs; the warps take blocks in a grid stride.  An op
// without gathers (Op::kMayScan) takes k_seg_scan where k_seg_reduce's warps
// need several blocks each and either k_seg_scan's need one only or no row is
// longer than a block (gg_bp, k_seg_reduce / k_seg_scan: Erdos-Renyi 1M of
// degree 8, 31K blocks, 324 / 274 us; 700^2 grid, 7.7K blocks, 113 / 101; R-MAT-18
// with 4 edges per vertex, 4.0K blocks, 89 / 92; R-MAT-20 with 16, 63K, 528 / 847).
template <class Op>
inline int seg_reduce(gg_graph_s* g, bool in_edges, Op op) {
  if (g->m == 0) return GG_OK;
  const int seg = g->symmetric ? 0 : ((in_edges != g->transposed) ? 0 : 1);
  const SegIndex& si = g->seg[seg];
  SegStream p{in_edges ? g->in_idx() : g->out_idx(), si.d_head, si.d_blk, si.d_rows,
              (g->m + kSegBlock - 1) / kSegBlock, g->m};
  static DeviceOnce occ;
  const uint64_t ctas = (p.nblocks + 7) / 8;
  const uint64_t wave = (uint64_t)g->num_sms * seg_resident(occ, g->device, k_seg_reduce<Op>);
  bool scan = false;
  if constexpr (Op::kMayScan) {
    static DeviceOnce occ_scan;
    const uint64_t wide = (uint64_t)g->num_sms * seg_resident(occ_scan, g->device, k_seg_scan<Op>);
    scan = ctas > wave && (ctas <= wide || si.longest <= kSegBlock);
    if (scan) k_seg_scan<Op><<<(int)std::min(ctas, wide), 256, 0, g->stream>>>(p, op);
  }
  if (!scan) k_seg_reduce<Op><<<(int)std::min(ctas, wave), 256, 0, g->stream>>>(p, op);
  g->kernels++;
  GG_CUDA(cudaGetLastError());
  return GG_OK;
}

}  // namespace gg
