// Shared-memory barriers and bulk copies (PTX mbarrier, cp.async.bulk).
//
// Every wait is bounded: a role that waits longer than kWaitNs gets false, and
// its kernel sets ST_WAIT_TIMEOUT and ends.
#pragma once
#include <cstdint>

namespace mgc {

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t* b, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(b)), "r"(count)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* b) {
  asm volatile(
      "{\n\t.reg .b64 st;\n\tmbarrier.arrive.release.cta.shared::cta.b64 st, [%0];\n\t}" ::"r"(
          smem_addr(b))
      : "memory");
}
// one test of the phase, the thread suspended until it completes or for at
// most kSuspendNs
constexpr uint32_t kSuspendNs = 200000;
__device__ __forceinline__ bool mbar_try(uint32_t addr, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cta.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(addr), "r"(parity), "n"(kSuspendNs)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// a waiting role gives up after this long (the whole kernel normally takes
// milliseconds)
constexpr uint64_t kWaitNs = 2000000000ull;
// Bounded wait for the completion of phase *parity* of barrier *b*; false
// when the time limit ran out or another role raised *abort* (if given).
__device__ __forceinline__ bool mbar_wait(uint64_t* b, uint32_t parity,
                                          const volatile int* abort) {
  const uint32_t a = smem_addr(b);
  if (mbar_try(a, parity)) return true;
  const uint64_t t0 = global_ns();
  for (;;) {
    if (mbar_try(a, parity)) return true;
    if (abort && *abort) return false;
    if (global_ns() - t0 > kWaitNs) return false;
  }
}
// arrive and announce *bytes* of bulk copies
__device__ __forceinline__ void mbar_expect(uint64_t* b, uint32_t bytes) {
  asm volatile(
      "{\n\t.reg .b64 st;\n\t"
      "mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 st, [%0], %1;\n\t}" ::"r"(smem_addr(b)),
      "r"(bytes)
      : "memory");
}
// copy *bytes* (a multiple of 16, both addresses 16-byte aligned) from global
// to shared memory, counted on *b*
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* b) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_addr(dst)),
      "l"(src), "r"(bytes), "r"(smem_addr(b))
      : "memory");
}

}  // namespace mgc
