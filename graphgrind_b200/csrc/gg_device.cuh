// Device-side building blocks for sm_100a: bitmap helpers, warp reductions,
// mbarrier + bulk-copy (TMA) primitives with bounded waits.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace gg {

// Error word bits written by kernels (read back by the host after a step).
enum : uint32_t { DEV_ERR_TIMEOUT = 1u, DEV_ERR_BOUNDS = 2u };

// Bounded spin budget of every device-side wait.  One try_wait probe may
// suspend for up to the hardware time limit; 1<<22 probes is seconds at most.
constexpr uint32_t kWaitBudget = 1u << 22;

__device__ __forceinline__ bool test_bit(const uint32_t* bm, uint32_t v) {
  return (__ldg(bm + (v >> 5)) >> (v & 31)) & 1u;
}

// What a functor's commit reads of its destination (raw 32-bit words):
// commit(d, acc) is commit_apply(d, commit_load(d), acc), split so that a
// caller can issue the loads of several destinations before it needs any.
struct CommitIn {
  uint32_t a, b;
};

template <class T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// ------------------------------------------------------------ cache hints
// L2 eviction policies (createpolicy, sm_80+) for loads that carry a
// .L2::cache_hint operand: evict_first for data read once (a COO edge
// stream), evict_last for data gathered again and again (source values).
__device__ __forceinline__ uint64_t l2_policy_evict_first() {
  uint64_t pol;
  asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
  return pol;
}
__device__ __forceinline__ uint64_t l2_policy_evict_last() {
  uint64_t pol;
  asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol));
  return pol;
}
// 16-byte read-only load that bypasses L1 (streamed data), with an L2 policy.
__device__ __forceinline__ uint4 ld_stream_v4(const void* ptr, uint64_t pol) {
  uint4 r;
  asm("ld.global.nc.L1::no_allocate.L2::cache_hint.v4.u32 {%0, %1, %2, %3}, [%4], %5;"
      : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
      : "l"(ptr), "l"(pol));
  return r;
}
// 4-byte read-only load that bypasses L1 (streamed data).
__device__ __forceinline__ uint32_t ld_stream_u32(const uint32_t* ptr) {
  uint32_t r;
  asm("ld.global.nc.L1::no_allocate.u32 %0, [%1];" : "=r"(r) : "l"(ptr));
  return r;
}
__device__ __forceinline__ float ld_stream_f32(const float* ptr) {
  float r;
  asm("ld.global.nc.L1::no_allocate.f32 %0, [%1];" : "=f"(r) : "l"(ptr));
  return r;
}
// 4-byte read-only gather kept in L1 and L2 ahead of streamed lines.
__device__ __forceinline__ float ld_keep_f32(const float* ptr, uint64_t pol) {
  float r;
  asm("ld.global.nc.L1::evict_last.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(r) : "l"(ptr), "l"(pol));
  return r;
}

// ------------------------------------------------------------ mbarrier
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// Orders this thread's generic-proxy shared-memory accesses before later
// async-proxy (bulk copy) writes to the same buffers.
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Wait for phase `parity` of `bar` to complete; false if the budget ran out.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity) {
  for (uint32_t it = 0; it < kWaitBudget; ++it)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}

// Bulk global->shared copy completed on `bar` (cp.async.bulk, no multicast).
// dst, src 16-byte aligned; bytes a multiple of 16.
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

}  // namespace gg
