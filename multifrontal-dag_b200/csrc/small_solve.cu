// Triangular solves of small fronts (nf <= 160): nf <= 32 one warp per front,
// four per CTA; above, one CTA of two to five warps per front.
//
// The panel goes to shared memory with cp.async, every copy in flight at once
// and next to the front's vectors and its children's, with an odd leading
// dimension: lanes over rows (forward) and lanes over columns (backward) both
// read it without bank conflicts.  One warp then runs the substitution from
// there: 45 cycles of dependent latency per column (product, shuffle,
// multiply-add).  The other warps of a front copy, gather and, backward, take
// their share of the rows below.
//
// Latency bounds these kernels.  A warp per front reading the panel from
// global memory eight columns at a time paid a memory round trip per group (and
// backward per row block too), after a chain of six dependent loads to its
// first operand; now there are three round trips in all (record, then panel,
// vectors and children's records, then the children's vectors).  Solve of a batch
// of 200 2D systems 1177 -> 770 us (0.9 TB/s over panels and vectors).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "kernels.cuh"

namespace mfd {

namespace {

template <int R>
__host__ __device__ constexpr int warps_per_front() { return R == 1 ? 1 : R == 2 ? 2 : R <= 4 ? 4 : 5; }
template <int R>
__host__ __device__ constexpr int fronts_per_cta() { return R == 1 ? 4 : 1; }
template <int R>
__host__ __device__ constexpr int solve_threads() { return 32 * warps_per_front<R>() * fronts_per_cta<R>(); }
// per front: the staged panel (at most panel_elems = (nf | 1) nc), the vector, the backward partial sums
template <int R>
__host__ __device__ int front_elems(int panel_elems) {
  return panel_elems + 32 * R + (R == 1 ? 0 : 32 * R * warps_per_front<R>());
}

template <int R>
__device__ __forceinline__ void front_sync() {
  if constexpr (warps_per_front<R>() == 1) __syncwarp();
  else __syncthreads();
}

template <typename T>
__device__ __forceinline__ void copy_async(T* dst, const T* src) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(dst);
  if constexpr (sizeof(T) == 8) asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(src));
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(sa), "l"(src));
}

// the lower part of the nf x nc panel, column stride ld
template <typename T, int R>
__device__ __forceinline__ void stage_panel(T* L, int ld, const T* P, int nf, int nc, int lane, int wl) {
  constexpr int W = warps_per_front<R>();
  for (int j = wl; j < nc; j += W)
    for (int i = j + lane; i < nf; i += 32) copy_async(L + j * ld + i, P + (size_t)j * nf + i);
  asm volatile("cp.async.commit_group;\n" ::);
}
__device__ __forceinline__ void staged() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// grid y: right-hand sides
template <typename T, int R>
__global__ void __launch_bounds__(solve_threads<R>()) k_fwd_small(DevFronts F, const FrontRec* __restrict__ recs, int count,
                                                                  int panel_elems, const T* __restrict__ panel, T* X,
                                                                  int64_t ldx, T* V, int nrhs) {
  constexpr int W = warps_per_front<R>(), FPC = fronts_per_cta<R>();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, tl = threadIdx.x % (32 * W), wl = tl >> 5, fg = threadIdx.x / (32 * W);
  const int slot = blockIdx.x * FPC + fg, r = blockIdx.y;
  if (slot >= count) return;                             // a whole warp (R == 1), else never
  T* L = reinterpret_cast<T*>(smem_raw) + (size_t)fg * front_elems<R>(panel_elems);
  T* vs = L + panel_elems;
  const FrontRec rec = recs[slot];
  const int nc = rec.nc, nf = nc + rec.nr, ld = nf | 1;
  stage_panel<T, R>(L, ld, panel + rec.panel_off, nf, nc, lane, wl);
  // children's records one per lane of every warp, broadcast by shuffles
  const int nch = rec.child_end - rec.child_beg;
  int cnc = 0, cnr = 0, clo = 0;
  long long cvo = 0;
  auto records = [&](int t0) {
    cnc = cnr = clo = 0;
    cvo = 0;
    if (t0 + lane < nch) {
      const ChildRec c = F.crec[rec.child_beg + t0 + lane];
      cnc = c.nc; cnr = c.nr; clo = c.lrow_off; cvo = c.v_off;
    }
  };
  records(0);
  T* Xr = X + rec.first + r * ldx;
#pragma unroll
  for (int q = 0; q < (R + W - 1) / W; ++q) {
    const int i = tl + 32 * W * q;
    if (i < 32 * R) vs[i] = i < nc ? Xr[i] : T(0);
  }
  // child t's update vector: one entry per thread (nr < 32 R <= 32 W), the next child's loads ahead
  int li = -1;
  T vv = T(0);
  auto fetch = [&](int t, int& l, T& v) {
    const int q = t & 31, n = __shfl_sync(0xffffffffu, cnr, q), c = __shfl_sync(0xffffffffu, cnc, q);
    const int lo = __shfl_sync(0xffffffffu, clo, q);
    const long long vo = __shfl_sync(0xffffffffu, cvo, q);
    l = -1;
    if (tl < n) {
      l = F.local[lo + tl] - 1;
      v = V[vo * nrhs + (int64_t)r * (c + n) + c + tl];
    }
  };
  if (nch > 0) fetch(0, li, vv);
  front_sync<R>();
  for (int t = 0; t < nch; ++t) {
    int ln = -1;
    T vn = T(0);
    if (t + 1 < nch) {
      if (((t + 1) & 31) == 0) records(t + 1);
      fetch(t + 1, ln, vn);
    }
    if (li >= 0) vs[li] += vv;
    front_sync<R>();
    li = ln;
    vv = vn;
  }
  staged();
  front_sync<R>();
  if (wl > 0) return;
  T v[R], dinv[R];
#pragma unroll
  for (int q = 0; q < R; ++q) {
    const int i = lane + 32 * q;
    v[q] = vs[i];
    dinv[q] = i < nc ? T(1) / L[i * ld + i] : T(1);
  }
#pragma unroll
  for (int b = 0; b < R; ++b) {
    const int k0 = 32 * b, kn = min(32, nc - k0);
#pragma unroll 8
    for (int kk = 0; kk < kn; ++kk) {
      const T* Lk = L + (k0 + kk) * ld + lane;
      const T y = __shfl_sync(0xffffffffu, v[b] * dinv[b], kk);
#pragma unroll
      for (int q = b; q < R; ++q) {
        const bool below = (q > b || lane > kk) && lane + 32 * q < nf;
        const T l = below ? Lk[32 * q] : T(0);
        v[q] -= l * y;
      }
      if (lane == kk) v[b] = y;
    }
  }
  T* Vf = V + rec.v_off * nrhs + (int64_t)r * nf;
#pragma unroll
  for (int q = 0; q < R; ++q) {
    const int i = lane + 32 * q;
    if (i < nc) Xr[i] = v[q];
    else if (i < nf) Vf[i] = v[q];
  }
}

template <typename T, int R>
__global__ void __launch_bounds__(solve_threads<R>()) k_bwd_small(DevFronts F, const FrontRec* __restrict__ recs, int count,
                                                                  int panel_elems, const T* __restrict__ panel, T* X,
                                                                  int64_t ldx) {
  constexpr int W = warps_per_front<R>(), FPC = fronts_per_cta<R>();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, tl = threadIdx.x % (32 * W), wl = tl >> 5, fg = threadIdx.x / (32 * W);
  const int slot = blockIdx.x * FPC + fg;
  if (slot >= count) return;
  T* L = reinterpret_cast<T*>(smem_raw) + (size_t)fg * front_elems<R>(panel_elems);
  T* xs = L + panel_elems;
  T* part = xs + 32 * R;                                 // W x 32 R, R > 1
  const FrontRec rec = recs[slot];
  const int nc = rec.nc, nf = nc + rec.nr, ld = nf | 1;
  T* Xr = X + blockIdx.y * ldx;
  stage_panel<T, R>(L, ld, panel + rec.panel_off, nf, nc, lane, wl);
#pragma unroll
  for (int q = 0; q < (R + W - 1) / W; ++q) {
    const int i = tl + 32 * W * q;
    if (i < nf) xs[i] = Xr[i < nc ? rec.first + i : F.lrow[rec.lrow_off + i - nc]];
  }
  staged();
  front_sync<R>();
  // rows below the triangle: lanes over columns, rows i = nc + wl, nc + wl + W, ...
  T t[R], s[R];
#pragma unroll
  for (int q = 0; q < R; ++q) {
    s[q] = T(0);
    const int c = lane + 32 * q;
    if (c < nc) {
      T s4[4] = {T(0), T(0), T(0), T(0)};
      int i = nc + wl;
      for (; i + 3 * W < nf; i += 4 * W)
#pragma unroll
        for (int u = 0; u < 4; ++u) s4[u] += L[c * ld + i + u * W] * xs[i + u * W];
      for (; i < nf; i += W) s4[0] += L[c * ld + i] * xs[i];
      s[q] = (s4[0] + s4[1]) + (s4[2] + s4[3]);
    }
  }
  if constexpr (W > 1) {
#pragma unroll
    for (int q = 0; q < R; ++q) part[wl * 32 * R + lane + 32 * q] = s[q];
    __syncthreads();
    if (wl > 0) return;
#pragma unroll
    for (int q = 0; q < R; ++q)
#pragma unroll
      for (int w = 1; w < W; ++w) s[q] += part[w * 32 * R + lane + 32 * q];
  }
  T dinv[R];
#pragma unroll
  for (int q = 0; q < R; ++q) {
    const int c = lane + 32 * q;
    t[q] = c < nc ? xs[c] - s[q] : T(0);
    dinv[q] = c < nc ? T(1) / L[c * ld + c] : T(1);
  }
#pragma unroll
  for (int b = R - 1; b >= 0; --b) {
    const int k0 = 32 * b, kn = min(32, nc - k0);
#pragma unroll 8
    for (int kk = kn - 1; kk >= 0; --kk) {
      const T* Lk = L + k0 + kk;                         // row k0 + kk: column c at Lk[c ld]
      const T x = __shfl_sync(0xffffffffu, t[b] * dinv[b], kk);
#pragma unroll
      for (int q = 0; q <= b; ++q) {
        const T l = q < b || lane < kk ? Lk[(lane + 32 * q) * ld] : T(0);
        t[q] -= l * x;
      }
      if (lane == kk) t[b] = x;
    }
  }
#pragma unroll
  for (int q = 0; q < R; ++q)
    if (lane + 32 * q < nc) Xr[rec.first + lane + 32 * q] = t[q];
}

}  // namespace

template <typename T>
size_t small_solve_smem(int nf_max, int panel_elems) {
  switch ((nf_max + 31) / 32) {
    case 1: return sizeof(T) * fronts_per_cta<1>() * (size_t)front_elems<1>(panel_elems);
    case 2: return sizeof(T) * (size_t)front_elems<2>(panel_elems);
    case 3: return sizeof(T) * (size_t)front_elems<3>(panel_elems);
    case 4: return sizeof(T) * (size_t)front_elems<4>(panel_elems);
    default: return sizeof(T) * (size_t)front_elems<5>(panel_elems);
  }
}

cudaError_t prepare_small_solve() {
  cudaError_t e = cudaSuccess;
  auto chk = [&](auto k, size_t bytes) {
    cudaError_t r = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (r != cudaSuccess && e == cudaSuccess) e = r;
  };
  auto both = [&](auto one, int nf) {                    // the largest panel: (nf | 1) nf
    using T = decltype(one);
    const size_t bytes = small_solve_smem<T>(nf, (nf | 1) * nf);
    switch (nf / 32) {
      case 1: chk(k_fwd_small<T, 1>, bytes); chk(k_bwd_small<T, 1>, bytes); break;
      case 2: chk(k_fwd_small<T, 2>, bytes); chk(k_bwd_small<T, 2>, bytes); break;
      case 3: chk(k_fwd_small<T, 3>, bytes); chk(k_bwd_small<T, 3>, bytes); break;
      case 4: chk(k_fwd_small<T, 4>, bytes); chk(k_bwd_small<T, 4>, bytes); break;
      default: chk(k_fwd_small<T, 5>, bytes); chk(k_bwd_small<T, 5>, bytes); break;
    }
  };
  for (int nf = 32; nf <= kSmallFrontMax; nf += 32) {
    both(0.0, nf);
    both(0.0f, nf);
  }
  return e;
}

template <typename T>
void launch_fwd_small(const DevFronts& F, const FrontRec* rec, int count, int nf_max, int panel_elems, const T* panel,
                      T* X, int64_t ldx, T* V, int nrhs, cudaStream_t st) {
  if (count <= 0) return;
  const size_t sm = small_solve_smem<T>(nf_max, panel_elems);
  auto go = [&](auto k, int fpc, int nt) {
    k<<<dim3((count + fpc - 1) / fpc, nrhs), nt, sm, st>>>(F, rec, count, panel_elems, panel, X, ldx, V, nrhs);
  };
  switch ((nf_max + 31) / 32) {
    case 1: go(k_fwd_small<T, 1>, fronts_per_cta<1>(), solve_threads<1>()); break;
    case 2: go(k_fwd_small<T, 2>, 1, solve_threads<2>()); break;
    case 3: go(k_fwd_small<T, 3>, 1, solve_threads<3>()); break;
    case 4: go(k_fwd_small<T, 4>, 1, solve_threads<4>()); break;
    default: go(k_fwd_small<T, 5>, 1, solve_threads<5>()); break;
  }
}
template <typename T>
void launch_bwd_small(const DevFronts& F, const FrontRec* rec, int count, int nf_max, int panel_elems, const T* panel,
                      T* X, int64_t ldx, int nrhs, cudaStream_t st) {
  if (count <= 0) return;
  const size_t sm = small_solve_smem<T>(nf_max, panel_elems);
  auto go = [&](auto k, int fpc, int nt) {
    k<<<dim3((count + fpc - 1) / fpc, nrhs), nt, sm, st>>>(F, rec, count, panel_elems, panel, X, ldx);
  };
  switch ((nf_max + 31) / 32) {
    case 1: go(k_bwd_small<T, 1>, fronts_per_cta<1>(), solve_threads<1>()); break;
    case 2: go(k_bwd_small<T, 2>, 1, solve_threads<2>()); break;
    case 3: go(k_bwd_small<T, 3>, 1, solve_threads<3>()); break;
    case 4: go(k_bwd_small<T, 4>, 1, solve_threads<4>()); break;
    default: go(k_bwd_small<T, 5>, 1, solve_threads<5>()); break;
  }
}

#define MFD_INSTANTIATE_SMALL_SOLVE(T)                                                                              \
  template void launch_fwd_small<T>(const DevFronts&, const FrontRec*, int, int, int, const T*, T*, int64_t, T*,   \
                                    int, cudaStream_t);                                                             \
  template void launch_bwd_small<T>(const DevFronts&, const FrontRec*, int, int, int, const T*, T*, int64_t, int,  \
                                    cudaStream_t);
MFD_INSTANTIATE_SMALL_SOLVE(double)
MFD_INSTANTIATE_SMALL_SOLVE(float)

}  // namespace mfd
