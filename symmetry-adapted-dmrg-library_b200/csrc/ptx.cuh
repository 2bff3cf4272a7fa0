// ptx.cuh -- small inline-PTX helpers shared by the GEMM kernels: shared-memory
// addresses, mbarriers with bounded waits, acquire loads, and chained launches.
#pragma once
#include <cuda_runtime.h>
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

// First statement of every kernel that launch_chained starts, in every thread: the next
// such kernel of the stream may be set up now, and everything the kernels before have
// written is visible from here on.  (A block that left without it would let the next
// kernel pass its own wait while kernels before this one still run.)
__device__ __forceinline__ void chain_begin() {
  asm volatile("griddepcontrol.launch_dependents;\n\tgriddepcontrol.wait;" ::: "memory");
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
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

// Launch on a stream whose blocks are set up while the kernel before it still runs
// (programmatic dependent launch): its grid, parameters and first instructions are in place
// when chain_begin lets it go on.  A Krylov step is 6 kernels of 3 to 10 us at small bond
// dimensions: U(1) D = 64 bond solve (288 launches) 2.70 -> 2.11 ms, SU(2) D = 512 8.5 -> 8.1,
// 64 problems at once 15.1 -> 14.2.
template <class... P, class... A>
inline void launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);   // an error is seen by the callers' next check
}

}  // namespace sadmrg
