// mbarriers and set-up of bulk tensor copies (TMA).  Loads only, no cluster
// multicast.
//
// Every wait on an mbarrier is bounded by the global timer, so a broken
// pipeline never hangs the GPU: the waiting kernel records
// EFWI_STATUS_TIMEOUT, waits (again bounded) for its copies in flight and
// leaves.
#pragma once
#include <cuda.h>
#include <stdint.h>

#include <atomic>

namespace efwi {

constexpr unsigned long long TMA_WAIT_NS = 2000000000ULL;  // 2 s

enum { EFWI_STATUS_OK = 0, EFWI_STATUS_TIMEOUT = 1 };

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// Orders this thread's earlier generic-proxy shared-memory accesses before
// later async-proxy (bulk copy) writes to the same slots.
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}

// One try: the thread may be suspended up to TMA_SUSPEND_NS while the
// phase is incomplete, instead of spinning and taking issue slots.
constexpr uint32_t TMA_SUSPEND_NS = 2000;
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity), "r"(TMA_SUSPEND_NS)
      : "memory");
  return ok != 0;
}

// Bounded wait: true when the phase completed, false after TMA_WAIT_NS.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, uint32_t parity) {
  if (mbar_try_wait(bar, parity)) return true;
  const unsigned long long t0 = global_ns();
  while (!mbar_try_wait(bar, parity)) {
    if (global_ns() - t0 > TMA_WAIT_NS) return false;
  }
  return true;
}

// Raises a kernel's dynamic shared-memory limit once per device: the
// attribute belongs to the device's context, so a process that drives
// several GPUs sets it on each (bit d of `done` stands for device d).  The
// bit is set only when the call succeeded; a failure stays pending as the
// runtime's last error, which the launch wrapper's check reports for the
// launch that needed the attribute.
template <class K>
inline void set_smem_once(K kernel, int bytes, std::atomic<unsigned long long> &done) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return;
  const unsigned long long bit = 1ull << (dev & 63);
  if (done.load(std::memory_order_acquire) & bit) return;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) ==
      cudaSuccess)
    done.fetch_or(bit, std::memory_order_acq_rel);
}

}  // namespace efwi
