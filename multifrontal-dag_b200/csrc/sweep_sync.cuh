// Shared by the fused solve sweeps: device-side flags (bounded waits, acquire /
// release) and the forward gather.
#pragma once
#include <cuda_runtime.h>

#include <climits>
#include <cstdint>

#include "plan.hpp"

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

// Entry i of front f's vector before its panel steps: its own right-hand side
// (Xf: the front's first column) plus the children's update vectors in child
// order (V: nrhs columns per front, column r), two children's loads in flight;
// with many children (`many`, said by the task) the sum is in G already (launch_gather_many).
// kMany: the level has such fronts; the others' sweeps are compiled without (37 x 41 x 43 solve
// 801 us, 805 with the branch).
template <bool kMany, typename T>
__device__ __forceinline__ T gather_row(const DevFronts& F, int f, bool many, int i, int nf, int nc, const T* Xf, const T* V,
                                        const double* G, int nrhs, int r) {
  if (kMany && many) return (T)G[F.g_off[f] * nrhs + (int64_t)r * nf + i];
  T v = i < nc ? Xf[i] : T(0);
  const int ce = F.child_ptr[f + 1];
  for (int t = F.child_ptr[f]; t < ce; t += 2) {
    T x[2];
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      x[s] = T(0);
      if (t + s < ce) {
        const ChildRec c = F.crec[t + s];
        const int ci = F.inv[c.inv_off + i];
        if (ci >= 0) x[s] = V[c.v_off * nrhs + (int64_t)r * (c.nc + c.nr) + c.nc + ci];
      }
    }
    v += x[0];
    v += x[1];
  }
  return v;
}

}  // namespace mfd
