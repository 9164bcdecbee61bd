// mbarrier and bulk-copy helpers of the product sketch and FWHT-of-rows kernels.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace cmm {
namespace {

constexpr int kPSkip = -0x7fffffff;  // row pair with a zero row: contributes nothing

__device__ __forceinline__ double pow2(int e) { return __longlong_as_double((long long)(1023 + e) << 52); }

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void bar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_expect(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool bar_test(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred P1;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, P1;\n\t}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait, by the device's clock (a count of polls would not do, try_wait
// itself may suspend the thread for as long as it likes).  state: [0] a role of
// the CTA has given up, upon which the others do at once; [1] limit in us.
constexpr int kWaitUs = 2000000;
__device__ __forceinline__ uint64_t clock_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ bool bar_wait(uint64_t* bar, uint32_t parity, volatile int* state) {
  for (int it = 0; it < 64; ++it)
    if (bar_test(bar, parity)) return true;
  const uint64_t t0 = clock_ns(), limit = 1000ull * (unsigned)state[1];
  do {
    if (bar_test(bar, parity)) return true;
    if (state[0]) return false;
    __nanosleep(20);
  } while (clock_ns() - t0 < limit);
  state[0] = 1;
  return false;
}
// the same for what is in flight when a CTA gives up
__device__ __forceinline__ void bar_drain(uint64_t* bar, uint32_t parity, volatile int* state) {
  const uint64_t t0 = clock_ns(), limit = 1000ull * (unsigned)state[1];
  while (!bar_test(bar, parity) && clock_ns() - t0 < limit) __nanosleep(20);
}
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void bar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

}  // namespace
}  // namespace cmm
