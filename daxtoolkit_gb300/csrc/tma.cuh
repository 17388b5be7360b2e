// Bulk TMA copies, mbarriers, acquire / release accesses and bounded waits
// shared by the kernels that stage global data in shared memory or wait on
// other blocks.
#pragma once
#include <cstdint>
#include "common.cuh"

namespace daxgb {

constexpr unsigned long long kSpinNs = 200000000ull;  // 0.2 s

__device__ __forceinline__ unsigned smem_addr(const void* p) {
  return (unsigned)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ unsigned long long now_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ unsigned ld_acquire(const uint32_t* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(uint32_t* p, unsigned v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned ld_relaxed(const uint32_t* p) {
  unsigned v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive_tx(uint64_t* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_test(uint64_t* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n"
      " mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_addr(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Field bytes [src, src + bytes) into shared memory, completion counted on
// bar; the field is streamed once, so it is marked evict-first in L2 (the
// bit stream and offsets stay resident for the emit).
__device__ __forceinline__ void bulk_load(void* dst, const void* src, unsigned bytes, uint64_t* bar,
                                          unsigned long long policy) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
      " [%0], [%1], %2, [%3], %4;" ::"r"(smem_addr(dst)),
      "l"(src), "r"(bytes), "r"(smem_addr(bar)), "l"(policy)
      : "memory");
}
__device__ __forceinline__ void fence_proxy_async() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
// Shared-memory bytes [src, src + bytes) to global memory as one bulk copy
// (both addresses and the size multiples of 16), then wait until the copy has
// read all of its source, after which the shared memory may be reused.
// The threads that wrote src must run fence_proxy_async() and meet the
// issuing thread at a barrier first.
__device__ __forceinline__ void bulk_store_and_wait_read(void* dst, const void* src,
                                                         unsigned bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst),
               "r"(smem_addr(src)), "r"(bytes)
               : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
  asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}

// Bounded waiting: more() is false once `polls` polls or kSpinNs have passed
// since the first poll.  A wait that runs out with a copy into the block's
// shared memory in flight waits once more, with the default limit, before the
// block leaves: the copy would land in memory that is another block's by then.
struct Spin {
  unsigned n = 0, polls;
  unsigned long long t0 = 0;
  __device__ __forceinline__ explicit Spin(unsigned polls = kSpinIters) : polls(polls) {}
  __device__ __forceinline__ bool more() {
    if (n == 0) t0 = now_ns();
    ++n;
    if (n >= polls) return false;
    if ((n & 63u) == 0u && now_ns() - t0 > kSpinNs) return false;
    return true;
  }
};

}  // namespace daxgb
