// ptx.cuh -- small inline-PTX helpers shared by the GEMM kernels: shared-memory
// addresses, mbarriers with bounded waits, acquire loads.
#pragma once
#include <cstdint>

namespace sadmrg {

constexpr unsigned long long kWaitNs = 2000000000ull;   // 2 s per wait
constexpr long long kWaitIters = 1ll << 26;

__device__ __forceinline__ uint32_t saddr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ unsigned long long gtime() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
// one arrival on the barrier once every cp.async this thread has issued so far has
// landed (counted in the barrier's expected arrivals)
__device__ __forceinline__ void mbar_arrive_cp_async(uint32_t bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];\n" ::"r"(bar) : "memory");
}

// Bounded wait for the phase with the given parity.  Gives up (false) after
// limit_ns, or as soon as *abort is set when abort is non-null.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, const volatile int* abort,
                                          unsigned long long limit_ns = kWaitNs) {
  unsigned long long t0 = 0;
  for (long long i = 0; i < kWaitIters; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok) return true;
    if ((i & 63) == 63) {
      if (abort && *abort) return false;
      if (t0 == 0) t0 = gtime();
      else if (gtime() - t0 > limit_ns) return false;
    }
  }
  return false;
}

__device__ __forceinline__ int ld_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

}  // namespace sadmrg
