// Large-front solves with several right-hand sides: each level's forward and
// backward sweep as one launch over the single-RHS sweep's task list
// (launch_large_fused), every task split into tiles of R right-hand sides, 8
// up to eight of them and 16 beyond.
//
// A task multiplies 128 x 128 blocks of the factor by 128 x R blocks of the
// vectors on m8n8k4 DMMA, in FP64 whatever the storage type.  The factor goes
// from global memory straight into operand fragments (the contraction index
// taken in the order 0 2 4 6, 1 3 5 7 of each eight, as in chol_smem.cuh), half
// a block at a time, 32 values per thread in flight, the first half before the
// wait on the vectors it meets; only the vectors pass through shared memory.
//
// Half blocks keep a thread under 128 registers, so that two CTAs share an SM:
// the levels of many fronts are bound by each task's chain of loads (ticket,
// front, factor, vectors), 5 us per task with one CTA per SM and whole blocks
// in registers, the top levels by the chain of steps.  Sixteen columns halve
// the tasks of many right-hand sides.  Whole steps against one launch per panel
// step (2-7 columns) or four GEMM-shaped ones (8 and more): 5 columns on 30x33x35
// 4.48 -> 3.5 ms, 16 columns of 21^3 elasticity in FP32 + refinement 10.45 -> 6.30,
// 64 columns of 30^3 elasticity 20.3 -> 16.8.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "chol_smem.cuh"
#include "kernels.cuh"
#include "sweep_sync.cuh"

namespace mfd {

namespace {

constexpr int kHalf = 8;          // blocks of eight columns per register half

// The 128 x (8 NB) block of the vectors (column stride ld, `rows` rows, `cols`
// columns valid) as B fragments: element (k, n) at Y[(n / 8) 1024 + (k / 8) 64 +
// 8 (n % 8) + k % 8], zero outside.  Read past L1: other CTAs wrote it.
// idx (may be null): row k is row idx[k] of v.
template <int NB, typename T>
__device__ __forceinline__ void stage_vectors(double* Y, const T* v, int64_t ld, int rows, int cols,
                                              const int32_t* idx = nullptr) {
  const int k = threadIdx.x & 127, kr = k < rows ? (idx ? idx[k] : k) : 0;
#pragma unroll
  for (int u = 0; u < 4 * NB; ++u) {
    const int n = (threadIdx.x >> 7) + 2 * u;
    Y[(n >> 3) * 1024 + (k >> 3) * 64 + (n & 7) * 8 + (k & 7)] = k < rows && n < cols ? (double)__ldcg(v + n * ld + kr) : 0.0;
  }
}

// acc[m][n] += A[m] B[n] over blocks [b0, min(b0 + kHalf, kb)) of eight, A in registers
template <int NB, typename T>
__device__ __forceinline__ void mul_half(double2 (&acc)[2][NB], const T (&a)[2][kHalf][2], const double* Y, int b0,
                                         int kb, int lane) {
  const double2* Yf = reinterpret_cast<const double2*>(Y) + lane;
#pragma unroll
  for (int b = 0; b < kHalf; ++b)
    if (b0 + b < kb) {
#pragma unroll
      for (int n = 0; n < NB; ++n) {
        const double2 y = Yf[n * 512 + (b0 + b) * 32];
#pragma unroll
        for (int m = 0; m < 2; ++m) dmma8(acc[m][n], make_double2((double)a[m][b][0], (double)a[m][b][1]), y);
      }
    }
}

// half h of rows (row0, row0 + 8) x 128 columns: entry (row, c) at p[row + c ld], zero outside
template <typename T>
__device__ __forceinline__ void load_rows(T (&a)[2][kHalf][2], const T* p, size_t ld, int row0, int row1, int w, int h,
                                          int q2) {
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    const bool ok = row0 + 8 * m < row1;
    const T* pr = p + (ok ? row0 + 8 * m : 0) + (size_t)(64 * h + q2) * ld;
#pragma unroll
    for (int b = 0; b < kHalf; ++b)
#pragma unroll
      for (int e = 0; e < 2; ++e) a[m][b][e] = ok && 64 * h + 8 * b + q2 + e < w ? pr[(size_t)(8 * b + e) * ld] : T(0);
  }
}
// half h of the transposed operand: columns (col0, col0 + 8) x 128 rows, entry (r, col) at p[r + col ld]
template <typename T>
__device__ __forceinline__ void load_cols(T (&a)[2][kHalf][2], const T* p, size_t ld, int col0, int w, int rows, int h,
                                          int q2) {
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    const bool ok = col0 + 8 * m < w;
    const T* pc = p + 64 * h + q2 + (size_t)(ok ? col0 + 8 * m : 0) * ld;
#pragma unroll
    for (int b = 0; b < kHalf; ++b)
#pragma unroll
      for (int e = 0; e < 2; ++e) a[m][b][e] = ok && 64 * h + 8 * b + q2 + e < rows ? pc[8 * b + e] : T(0);
  }
}
// this lane's accumulator entries into the B fragment layout
template <int NB>
__device__ __forceinline__ void put_vectors(double* Y, const double2 (&v)[2][NB], int warp, int g, int q2) {
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int n = 0; n < NB; ++n) {
      Y[n * 1024 + (2 * warp + m) * 64 + q2 * 8 + g] = v[m][n].x;
      Y[n * 1024 + (2 * warp + m) * 64 + (q2 + 1) * 8 + g] = v[m][n].y;
    }
}
template <int NB>
__device__ __forceinline__ void zero(double2 (&v)[2][NB]) {
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int n = 0; n < NB; ++n) v[m][n] = make_double2(0.0, 0.0);
}

// gather_row (sweep_sync.cuh) for right-hand sides rc + 8 n and rc + 8 n + 1, n < NB, below re; row i < 0: zeros
template <int NB, bool kMany, typename T>
__device__ __forceinline__ void gather_rows(double2 (&v)[NB], const DevFronts& F, int f, bool many, int i, int nf, int nc, const T* Xf,
                                            int64_t ldx, const T* V, const double* G, int nrhs, int rc, int re) {
  if (kMany && many) {
    const double* g = G + F.g_off[f] * nrhs + i;
#pragma unroll
    for (int n = 0; n < NB; ++n) {
      const int r = rc + 8 * n;
      v[n].x = i >= 0 && r < re ? g[(int64_t)r * nf] : 0.0;
      v[n].y = i >= 0 && r + 1 < re ? g[(int64_t)(r + 1) * nf] : 0.0;
    }
    return;
  }
#pragma unroll
  for (int n = 0; n < NB; ++n) {
    const int r = rc + 8 * n;
    v[n].x = i >= 0 && i < nc && r < re ? (double)Xf[i + (int64_t)r * ldx] : 0.0;
    v[n].y = i >= 0 && i < nc && r + 1 < re ? (double)Xf[i + (int64_t)(r + 1) * ldx] : 0.0;
  }
  if (i < 0) return;
  for (int t = F.child_ptr[f], ce = F.child_ptr[f + 1]; t < ce; ++t) {
    const ChildRec c = F.crec[t];
    const int ci = F.inv[c.inv_off + i];
    if (ci < 0) continue;
    const int ld = c.nc + c.nr;
    const T* p = V + c.v_off * nrhs + (int64_t)rc * ld + c.nc + ci;
#pragma unroll
    for (int n = 0; n < NB; ++n) {
      if (rc + 8 * n < re) v[n].x += (double)p[(int64_t)(8 * n) * ld];
      if (rc + 8 * n + 1 < re) v[n].y += (double)p[(int64_t)(8 * n + 1) * ld];
    }
  }
}

// Forward: task (f, s, tile): y_s = Li (v_s - sum_{t<s} L_st y_t); rest tasks
// (128 rows below the columns): v -= sum_t L_rest,t y_t.  Warp w has rows
// 16 w .. 16 w + 15 of the task.
template <typename T, int NB, bool kMany>
__global__ void __launch_bounds__(256, 2)
    k_fwd_multi(DevFronts F, const int4* __restrict__ tasks, int ntask, int tiles, int stride, int32_t* ticket, int32_t* flags,
                int32_t* expired, const T* __restrict__ panel, const T* __restrict__ dinv, T* X, int64_t ldx, T* V,
                const double* __restrict__ G, int nrhs, const int32_t* test_req) {
  __shared__ int sh_t, sh_ok;
  __shared__ __align__(16) double Y[NB * 1024];
  if (threadIdx.x == 0) sh_t = atomicAdd(ticket, 1);
  __syncthreads();
  const int t = sh_t;
  if (t >= ntask * tiles) return;
  const int4 tk = tasks[t / tiles];
  const int tile = t % tiles, f = tk.x, code = tk.y;
  int32_t* fl = flags + (int64_t)tk.z * stride + tile;     // step s at fl[s stride]
  const bool probe = *test_req != 0;
  const int nc = F.nc[f], nf = nc + F.nr[f];
  const int r0 = code >= 0 ? code * kSolveB : nc + (-1 - code) * kSolveB;
  const int r1 = min(code >= 0 ? nc : nf, r0 + kSolveB);
  const int nsteps = code >= 0 ? code : (nc + kSolveB - 1) / kSolveB;   // steps whose y this task consumes
  const int c0r = tile * 8 * NB, cols = min(8 * NB, nrhs - c0r);
  const T* P = panel + F.panel_off[f];
  T* Vf = V + F.v_off[f] * nrhs + (int64_t)c0r * nf;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, q2 = 2 * (lane & 3);
  const int ri = 16 * warp + g;                            // rows r0 + ri and r0 + ri + 8
  double2 acc[2][NB];
  zero(acc);
  // the task's own rows of the vectors, gathered here (each row once), off the chain of steps
  double2 v[2][NB];
  const int first = F.first[f];
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    const int r = r0 + ri + 8 * m;
    gather_rows<NB, kMany>(v[m], F, f, tk.w != 0, r < r1 ? r : -1, nf, nc, X + first, ldx, V, G, nrhs, c0r + q2, c0r + cols);
  }
  T a[2][kHalf][2];
  for (int s = 0; s < nsteps; ++s) {
    const int c0 = s * kSolveB, w = min(kSolveB, nc - c0), kb = (w + 7) >> 3;
    const T* Pc = P + (size_t)c0 * nf;
    load_rows(a, Pc, nf, r0 + ri, r1, w, 0, q2);
    if (!cta_wait_flag(fl + (int64_t)s * stride, expired, &sh_ok, probe)) return;   // also: Y is free again
    stage_vectors<NB>(Y, Vf + c0, nf, w, cols);
    __syncthreads();
    mul_half(acc, a, Y, 0, kb, lane);
    if (kb > kHalf) {
      load_rows(a, Pc, nf, r0 + ri, r1, w, 1, q2);
      mul_half(acc, a, Y, kHalf, kb, lane);
    }
  }
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int n = 0; n < NB; ++n) {
      v[m][n].x -= acc[m][n].x;
      v[m][n].y -= acc[m][n].y;
    }
  if (code >= 0) {                                         // y = Li v (Li lower, zero outside its w x w part)
    const T* Li = dinv + F.d_off[f] + (size_t)code * kSolveB * kSolveB;
    const int kb = 2 * warp + 2;                           // the warp's rows end there
    load_rows(a, Li, kSolveB, ri, kSolveB, 8 * kb, 0, q2);
    __syncthreads();                                       // the last step's reads of Y
    put_vectors(Y, v, warp, g, q2);
    __syncthreads();
    zero(v);
    mul_half(v, a, Y, 0, kb, lane);
    if (kb > kHalf) {
      load_rows(a, Li, kSolveB, ri, kSolveB, 8 * kb, 1, q2);
      mul_half(v, a, Y, kHalf, kb, lane);
    }
  }
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    const int r = r0 + ri + 8 * m;
    if (r >= r1) continue;
#pragma unroll
    for (int n = 0; n < NB; ++n)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int c = 8 * n + q2 + e;
        if (c >= cols) continue;
        const T y = (T)(e ? v[m][n].y : v[m][n].x);
        Vf[(int64_t)c * nf + r] = y;
        if (code >= 0) X[first + r + (int64_t)(c0r + c) * ldx] = y;
      }
  }
  if (code < 0) return;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    st_release_i32(fl + (int64_t)code * stride, 1);
  }
}

// Backward: first the partial sums over the update rows (chunks of
// kBwdRestRows, their x known from the ancestors), then the column blocks from the last down: x_s =
// Li^T (v_s - L_below,s^T x_below), the chunks' partials added in chunk order.
// part: [front's step and chunk][tile][128 columns][8 NB].
template <typename T, int NB>
__global__ void __launch_bounds__(256, 2)
    k_bwd_multi(DevFronts F, const int4* __restrict__ tasks, int ntask, int tiles, int stride, int32_t* ticket, int32_t* flags,
                int32_t* expired, const T* __restrict__ panel, const T* __restrict__ dinv, T* X, int64_t ldx,
                int nrhs, T* part, int32_t* counters, const int32_t* test_req) {
  __shared__ int sh_t, sh_ok;
  __shared__ __align__(16) double Y[NB * 1024];
  if (threadIdx.x == 0) sh_t = atomicAdd(ticket, 1);
  __syncthreads();
  const int t = sh_t;
  if (t >= ntask * tiles) return;
  const int4 tk = tasks[t / tiles];
  const int tile = t % tiles, f = tk.x;
  int32_t* fl = flags + (int64_t)tk.z * stride + tile;
  int32_t* ctr = counters + (int64_t)tk.z * stride + tile;
  const bool probe = *test_req != 0;
  const int nc = F.nc[f], nr = F.nr[f], nf = nc + nr;
  const int nsteps = (nc + kSolveB - 1) / kSolveB, nch = (nr + kBwdRestRows - 1) / kBwdRestRows;
  const int c0r = tile * 8 * NB, cols = min(8 * NB, nrhs - c0r);
  const T* P = panel + F.panel_off[f];
  const int first = F.first[f];
  T* Xt = X + (int64_t)c0r * ldx;                          // the tile's right-hand sides
  const int32_t* lr = F.lrow + F.lrow_off[f] - nc;         // row r >= nc of the front is row lr[r] of X
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, q2 = 2 * (lane & 3);
  const int ci = 16 * warp + g;                            // columns c0 + ci and c0 + ci + 8
  // this lane's first entry of partial (s, j)
  auto partial = [&](int s, int j) {
    return part + (((int64_t)tk.w / kSolveB + (int64_t)s * nch + j) * tiles + tile) * (kSolveB * 8 * NB) + ci * (8 * NB) + q2;
  };
  double2 acc[2][NB];
  zero(acc);
  T a[2][kHalf][2];
  // acc += (rows [ra, rb) of column block Pc)^T x, the first half of the rows loaded
  auto finish_rows = [&](const T* Pc, int w, int ra, int rb) {
    const int kb = (rb - ra + 7) >> 3;
    if (ra < nc) stage_vectors<NB>(Y, Xt + first + ra, ldx, rb - ra, cols);
    else stage_vectors<NB>(Y, Xt, ldx, rb - ra, cols, lr + ra);
    __syncthreads();
    mul_half(acc, a, Y, 0, kb, lane);
    if (kb > kHalf) {
      load_cols(a, Pc + ra, nf, ci, w, rb - ra, 1, q2);
      mul_half(acc, a, Y, kHalf, kb, lane);
    }
  };
  if (tk.y < 0) {
    const int code = -1 - tk.y, s = code >> 16, j = code & 0xffff;
    const int c0 = s * kSolveB, w = min(kSolveB, nc - c0);
    const T* Pc = P + (size_t)c0 * nf;
    const int re = min(nf, nc + (j + 1) * kBwdRestRows);
    for (int ra = nc + j * kBwdRestRows; ra < re; ra += kSolveB) {
      const int rb = min(re, ra + kSolveB);
      load_cols(a, Pc + ra, nf, ci, w, rb - ra, 0, q2);
      __syncthreads();
      finish_rows(Pc, w, ra, rb);
    }
    T* pt = partial(s, j);
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int n = 0; n < NB; ++n) {
        pt[m * 64 * NB + 8 * n] = (T)acc[m][n].x;
        pt[m * 64 * NB + 8 * n + 1] = (T)acc[m][n].y;
      }
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      atomicAdd(ctr + (int64_t)s * stride, 1);
    }
    return;
  }
  const int s = tk.y, c0 = s * kSolveB, w = min(kSolveB, nc - c0);
  const T* Pc = P + (size_t)c0 * nf;
  double2 v[2][NB];                                        // the task's own rows, off the chain of steps
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int n = 0; n < NB; ++n) {
      const int i = ci + 8 * m, c = 8 * n + q2;
      const T* p = Xt + (int64_t)c * ldx + first + c0 + i;
      v[m][n].x = i < w && c < cols ? (double)p[0] : 0.0;
      v[m][n].y = i < w && c + 1 < cols ? (double)p[ldx] : 0.0;
    }
  for (int b = nsteps - 1; b > s; --b) {                   // later diagonal blocks
    const int ra = b * kSolveB, rb = min(nc, ra + kSolveB);
    load_cols(a, Pc + ra, nf, ci, w, rb - ra, 0, q2);
    if (!cta_wait_flag(fl + (int64_t)b * stride, expired, &sh_ok, probe)) return;
    finish_rows(Pc, w, ra, rb);
  }
  // x = Li^T t: row ci needs k >= ci; Li is zero outside its w x w part
  const T* Li = dinv + F.d_off[f] + (size_t)s * kSolveB * kSolveB;
  load_cols(a, Li, kSolveB, ci, kSolveB, w, 0, q2);
  if (nch > 0) {
    if (!cta_wait_flag(ctr + (int64_t)s * stride, expired, &sh_ok, probe, nch)) return;
  } else {
    __syncthreads();                                       // the last block's reads of Y
  }
  double2 rs[2][NB];
  zero(rs);
  for (int j = 0; j < nch; ++j) {
    const T* pt = partial(s, j);
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int n = 0; n < NB; ++n) {
        rs[m][n].x += (double)__ldcg(pt + m * 64 * NB + 8 * n);
        rs[m][n].y += (double)__ldcg(pt + m * 64 * NB + 8 * n + 1);
      }
  }
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int n = 0; n < NB; ++n) {
      rs[m][n].x = v[m][n].x - (rs[m][n].x + acc[m][n].x);   // zero past the block's columns and right-hand sides
      rs[m][n].y = v[m][n].y - (rs[m][n].y + acc[m][n].y);
    }
  put_vectors(Y, rs, warp, g, q2);
  __syncthreads();
  zero(acc);
  const int kb = (w + 7) >> 3;
  mul_half(acc, a, Y, 0, kb, lane);
  if (kb > kHalf) {
    load_cols(a, Li, kSolveB, ci, kSolveB, w, 1, q2);
    mul_half(acc, a, Y, kHalf, kb, lane);
  }
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    const int i = ci + 8 * m;
    if (i >= w) continue;
#pragma unroll
    for (int n = 0; n < NB; ++n)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int c = 8 * n + q2 + e;
        if (c >= cols) continue;
        Xt[first + c0 + i + (int64_t)c * ldx] = (T)(e ? acc[m][n].y : acc[m][n].x);
      }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    st_release_i32(fl + (int64_t)s * stride, 1);
  }
}

}  // namespace

template <typename T>
void launch_large_multi(const DevFronts& F, const int4* tasks, int ntask, bool backward, int32_t* ticket, int32_t* flags,
                        int32_t* expired, const T* panel, const T* dinv, T* X, int64_t ldx, T* V, const double* G, int nrhs,
                        cudaStream_t st, const int32_t* test_req, T* part, int32_t* counters) {
  if (ntask <= 0) return;
  const int stride = multi_tiles(nrhs);
  auto go = [&](auto fwd, auto bwd, int width) {
    const int tiles = (nrhs + width - 1) / width;
    if (backward)
      bwd<<<ntask * tiles, 256, 0, st>>>(F, tasks, ntask, tiles, stride, ticket, flags, expired, panel, dinv, X, ldx,
                                         nrhs, part, counters, test_req);
    else
      fwd<<<ntask * tiles, 256, 0, st>>>(F, tasks, ntask, tiles, stride, ticket, flags, expired, panel, dinv, X, ldx, V,
                                         G, nrhs, test_req);
  };
  // Sixteen columns per task where the level has more tasks than the chip holds: there the tasks'
  // number counts.  Where all run at once the chain of steps counts, and eight columns have half
  // its MMAs (elasticity 30^3, 64 right-hand sides, root front of 2,883 columns: forward sweep
  // 207 us with 8, 360 us with 16; its level of 928 fronts: 268 us with 16, 716 us with 8 and
  // whole blocks in registers).
  if (nrhs <= 8 || (int64_t)ntask * stride <= 4 * kNumSms) {
    if (G) go(k_fwd_multi<T, 1, true>, k_bwd_multi<T, 1>, 8);
    else go(k_fwd_multi<T, 1, false>, k_bwd_multi<T, 1>, 8);
  } else {
    if (G) go(k_fwd_multi<T, 2, true>, k_bwd_multi<T, 2>, 16);
    else go(k_fwd_multi<T, 2, false>, k_bwd_multi<T, 2>, 16);
  }
}

#define MFD_INSTANTIATE_MULTI(T)                                                                                     \
  template void launch_large_multi<T>(const DevFronts&, const int4*, int, bool, int32_t*, int32_t*, int32_t*,        \
                                      const T*, const T*, T*, int64_t, T*, const double*, int, cudaStream_t,         \
                                      const int32_t*, T*, int32_t*);
MFD_INSTANTIATE_MULTI(double)
MFD_INSTANTIATE_MULTI(float)

}  // namespace mfd
