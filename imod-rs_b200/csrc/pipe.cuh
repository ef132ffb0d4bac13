// pipe.cuh -- the bulk-copy and mbarrier primitives of the back-projectors'
// pipelines, with bounded waits.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace tg {

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void *src, uint32_t bytes,
                                         uint32_t bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
      "l"(src), "r"(bytes), "r"(bar)
      : "memory");
}
// TMA box of a 3-D tensor map: x counts elements of the innermost dimension, its byte offset
// a multiple of 16.  The map is a kernel parameter, or in global memory and acquired first.
__device__ __forceinline__ void tma_box3(uint32_t dst, const void *map, int x, int y, int z, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst),
      "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar)
      : "memory");
}
// Before a CTA's first use of a tensor map that the host copied to global memory: copies read
// their map through a cache of its own, which may still hold what was at this address before.
__device__ __forceinline__ void tensormap_acquire(const void *map) {
  asm volatile("fence.proxy.tensormap::generic.acquire.sys [%0], 128;" ::"l"(map) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// try_wait that lets the hardware suspend the thread (up to hint_ns) until the
// phase completes, instead of returning at once
__device__ __forceinline__ bool mbar_try_wait_sleep(uint32_t bar, uint32_t parity, uint32_t hint_ns) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity), "r"(hint_ns)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ uint64_t globaltimer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// Bounded wait on an mbarrier phase: sleeps in try_wait, gives up after limit_ns
// of wall time (BpArgs::wait_limit_ns, 2 s by default: a stage never
// legitimately takes that long) or, when abort is given, as soon as another warp
// of the CTA has given up.
__device__ __forceinline__ bool wait_phase(uint32_t bar, uint32_t parity, volatile int *abort, uint64_t limit_ns) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = globaltimer_ns();
  for (;;) {
    if (mbar_try_wait_sleep(bar, parity, 20000u)) return true;
    if ((abort && *abort) || globaltimer_ns() - t0 > limit_ns) return false;
  }
}

// The same for a pipeline whose steps are no longer than reading the timer: ordinary
// waits end in the polls before it.  (Stages of bp_fast_kernel are longer; with the
// polls its back-projection of 2048x2048x800 x 121 took 56.64 ms, without 56.28.)
__device__ __forceinline__ bool poll_phase(uint32_t bar, uint32_t parity, volatile int *abort, uint64_t limit_ns) {
#pragma unroll 1
  for (int i = 0; i < 64; ++i)
    if (mbar_try_wait(bar, parity)) return true;
  return wait_phase(bar, parity, abort, limit_ns);
}

constexpr float MAGIC = 12582912.0f;      // 1.5 * 2^23
constexpr uint32_t MAGIC_BITS = 0x4B400000u;

}  // namespace tg
