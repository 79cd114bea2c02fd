// Device-side flags of the fused solve sweeps: bounded waits, acquire / release.
#pragma once
#include <cuda_runtime.h>

#include <climits>
#include <cstdint>

namespace mfd {

constexpr long long kSolveWaitLimit = 1ll << 31;    // cycles, about a second
constexpr long long kSolveProbeLimit = 1ll << 21;   // the test request's wait (~1 ms)

__device__ __forceinline__ int ld_acquire_i32(const int32_t* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_i32(int32_t* p, int v) {
  asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// thread 0 waits for *flag >= need (bounded; gives up at once when another
// CTA's wait expired); the result is the CTA's.  probe (a test request): the
// wait is for a value no producer writes, with a ~1 ms limit, so it expires.
__device__ __forceinline__ bool cta_wait_flag(const int32_t* flag, int32_t* expired, int* sh_ok, bool probe,
                                              int need = 1) {
  if (threadIdx.x == 0) {
    int ok = 1;
    if (probe) need = INT_MAX;
    const long long limit = probe ? kSolveProbeLimit : kSolveWaitLimit;
    if (ld_acquire_i32(flag) < need) {
      const long long t0 = clock64();
      while (ld_acquire_i32(flag) < need) {
        if (clock64() - t0 > limit || ld_acquire_i32(expired) != 0) {
          ok = 0;
          atomicExch(expired, 1);
          break;
        }
        __nanosleep(32);
      }
    }
    *sh_ok = ok;
  }
  __syncthreads();
  return *sh_ok != 0;
}

}  // namespace mfd
