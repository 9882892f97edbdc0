// bulk_pipeline.cuh — mbarriers and bulk copies into shared memory, for the
// sweeps that prepare one item while another is swept.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace tos {
namespace {

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void bar_init(unsigned long long* b, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_arrive(unsigned long long* b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(b)) : "memory");
}
__device__ __forceinline__ void bar_arrive_tx(unsigned long long* b, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(b)), "r"(bytes) : "memory");
}
// Wait for the phase of the given parity; false when `limit_ms` of the global
// timer have gone by.  A limit in time, not in tries, whose length the hardware
// sets: a warp may wait while another looks through a long list of items.
// limit_ms 0: one look.
__device__ __forceinline__ bool bar_try(unsigned long long* b, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
               : "=r"(ok)
               : "r"(smem_addr(b)), "r"(parity)
               : "memory");
  return ok != 0u;
}
__device__ __forceinline__ bool bar_test(unsigned long long* b, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n.reg .pred p;\nmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
               : "=r"(ok)
               : "r"(smem_addr(b)), "r"(parity)
               : "memory");
  return ok != 0u;
}
__device__ __forceinline__ uint32_t global_ms() {  // (of 2^20 ns)
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return (uint32_t)(t >> 20);
}
__device__ __forceinline__ bool bar_wait(unsigned long long* b, uint32_t parity, uint32_t limit_ms) {
  if (limit_ms == 0u) return bar_test(b, parity);
  if (bar_try(b, parity)) return true;
  const uint32_t t0 = global_ms();
  while (!bar_try(b, parity))
    if (global_ms() - t0 > limit_ms) return false;
  return true;
}
// The longest a sweep waits by default, and for its own copies before it gives up.
constexpr uint32_t kWaitMs = 10000;
// Bulk copy of `bytes` (a multiple of 16; both addresses 16-byte aligned)
// into shared memory, counted on barrier b.
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, unsigned long long* b) {
  asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_addr(dst)),
               "l"(src), "r"(bytes), "r"(smem_addr(b))
               : "memory");
}

}  // namespace
}  // namespace tos
