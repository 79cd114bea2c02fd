// sm_100a kernels of the multifrontal numeric phase.
//
// Index maps (built once):      local_index, supernodal_index + assembly map,
//                               block_local_index (reference tiling, export only)
// Factorization, per tree level: large fronts in global memory (gather of the
//                               children, assembly, trailing SYRK/GEMM on the FP64
//                               tensor pipe (DMMA) or FFMA tiles; small fronts are
//                               in small_front.cu, the panel steps' POTRF / TRSM in
//                               panel.cu, the updates from packed operands in
//                               update_dp.cu and update_tc.cu)
// Solves:                       permutations and the large fronts' per-step form
//                               (small_solve.cu, solve_single.cu and solve_multi.cu
//                               hold the rest)
// Residual / norms:             FP64 CSR SpMV for iterative refinement.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstdint>
#include <type_traits>

#include "chol_smem.cuh"
#include "kernels.cuh"

namespace mfd {

namespace {

__device__ __forceinline__ int lower_bound_dev(const int32_t* a, int n, int32_t key) {
  int lo = 0, hi = n;
  while (lo < hi) {
    int mid = (lo + hi) >> 1;
    if (a[mid] < key) lo = mid + 1; else hi = mid;
  }
  return lo;
}


inline int ceil_div(int64_t a, int64_t b) { return (int)((a + b - 1) / b); }

__device__ __forceinline__ void cp_async8(void* smem_dst, const void* gsrc, bool valid) {

  unsigned sa = (unsigned)__cvta_generic_to_shared(smem_dst);
  int sz = valid ? 8 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(sa), "l"(gsrc), "r"(sz));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

// Strided element loop (e = threadIdx.x, += blockDim.x, e < total) whose
// global loads are issued kBatch at a time before the matching stores, so a
// thread keeps kBatch independent loads in flight instead of one.
constexpr int kBatch = 16;
template <typename Load, typename Store>
__device__ __forceinline__ void batched_loop(int total, Load&& load, Store&& store) {
  using V = decltype(load(0));
  for (int e0 = threadIdx.x; e0 < total; e0 += blockDim.x * kBatch) {
    V v[kBatch];
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int e = e0 + u * (int)blockDim.x;
      v[u] = e < total ? load(e) : V(0);
    }
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int e = e0 + u * (int)blockDim.x;
      if (e < total) store(e, v[u]);
    }
  }
}
inline int clamp_grid(int64_t g, int64_t cap = 65535) { return (int)std::max<int64_t>(1, std::min<int64_t>(g, cap)); }

// ============================================================================
// index maps
// ============================================================================

// local_index (create_local_index_m.f90:10-45): for every L row r of child c,
// its 1-based position in the parent front: the parent's own column r-first+1,
// or nc_p + (position of r in the parent's sorted L rows).
__global__ void k_local_index(DevFronts F, int32_t* local, int num_front) {
  int c = blockIdx.x;
  if (c >= num_front) return;
  int p = F.parent[c];
  if (p < 0) return;
  int nrc = F.nr[c], off = F.lrow_off[c];
  int fp = F.first[p], ncp = F.nc[p], nrp = F.nr[p];
  const int32_t* lp = F.lrow + F.lrow_off[p];
  for (int i = threadIdx.x; i < nrc; i += blockDim.x) {
    int r = F.lrow[off + i];
    int pos;
    if (r < fp + ncp) {
      pos = r - fp;
    } else {
      int q = lower_bound_dev(lp, nrp, r);
      pos = (q < nrp && lp[q] == r) ? ncp + q : -1;      // -1: structure violation -> 0
    }
    local[off + i] = pos + 1;
  }
}

// supernodal_index (create_supernodal_index_m.f90:10-40) and the assembly map:
// one thread per permuted column; every A entry gets its front position
// (1-based, the reference's value), the source index of its value and its
// offset row + col*nf inside the front's panel.
__global__ void k_assembly_map(DevFronts F, const int32_t* col_front, const int32_t* acol_ptr, const int32_t* arow,
                               const int32_t* ccs_src, int32_t* sidx, int32_t* a_src, int32_t* a_pos, int n_total) {
  int col = blockIdx.x * blockDim.x + threadIdx.x;
  if (col >= n_total) return;
  int f = col_front[col];
  int first = F.first[f], nc = F.nc[f], nr = F.nr[f], nf = nc + nr;
  const int32_t* lr = F.lrow + F.lrow_off[f];
  int jloc = col - first;
  for (int k = acol_ptr[col]; k < acol_ptr[col + 1]; k++) {
    int r = arow[k];
    int pos;
    if (r < first + nc) {
      pos = r - first;
    } else {
      int q = lower_bound_dev(lr, nr, r);
      pos = (q < nr && lr[q] == r) ? nc + q : -1;
    }
    sidx[k] = pos + 1;
    a_src[k] = ccs_src[k];
    a_pos[k] = pos < 0 ? 0 : pos + jloc * nf;
  }
}

// What a small-front kernel needs of a front, one record per entry of the
// launch lists, and of a child, one per entry of the children lists: two loads
// deep where the tables above are six (list entry, front, child id, child).
__global__ void k_front_records(DevFronts F, const int32_t* lists, int n, FrontRec* rec) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const int f = lists[k];
  FrontRec r;
  r.nc = F.nc[f]; r.nr = F.nr[f]; r.first = F.first[f]; r.lrow_off = F.lrow_off[f];
  r.a_beg = F.a_beg[f]; r.a_end = F.a_beg[f + 1];
  r.child_beg = F.child_ptr[f]; r.child_end = F.child_ptr[f + 1];
  r.panel_off = F.panel_off[f]; r.u_off = F.u_off[f]; r.v_off = F.v_off[f];
  r.pad = 0;
  rec[k] = r;
}
__global__ void k_child_records(DevFronts F, int n, ChildRec* rec) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const int c = F.child[k];
  ChildRec r;
  r.nc = F.nc[c]; r.nr = F.nr[c]; r.lrow_off = F.lrow_off[c]; r.pad = 0;
  r.u_off = F.u_off[c]; r.v_off = F.v_off[c]; r.inv_off = F.inv_off ? F.inv_off[c] : 0; r.pad2 = 0;
  rec[k] = r;
}

// block_local_index (block_local_index_creator_m.f90:13-122): a group is a
// maximal run of a child's local index with constant (parent tile, child tile).
__device__ __forceinline__ void bli_key(int loc, int i, int ncc, int nb, int& pt, int& ct) {
  pt = (loc - 1) / nb + 1;            // get_matrix_num(local(i))
  ct = (ncc + i) / nb + 1;            // get_work_num(i+1, node) = get_matrix_num(nc + i + 1)
}

__global__ void k_bli_count(DevFronts F, const int32_t* fronts, int count, int nb, int32_t* groups) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= count) return;
  int c = fronts[t];
  int g = 0;
  if (F.parent[c] >= 0) {
    int nrc = F.nr[c], ncc = F.nc[c], pp = 0, pc = 0;
    const int32_t* loc = F.local + F.lrow_off[c];
    for (int i = 0; i < nrc; i++) {
      int pt, ct;
      bli_key(loc[i], i, ncc, nb, pt, ct);
      if (pt != pp || ct != pc) { pp = pt; pc = ct; g++; }
    }
  }
  groups[t] = g;
}

__global__ void k_bli_fill(DevFronts F, const int32_t* fronts, int count, int nb, const int32_t* group_base,
                           const int32_t* index_base, int32_t* block_ptr, int32_t* pnum, int32_t* cnum,
                           int32_t* offset, int32_t* rebuilt) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= count) return;
  int c = fronts[t];
  int nrc = F.nr[c], ncc = F.nc[c];
  const int32_t* loc = F.local + F.lrow_off[c];
  int ibase = index_base[t];
  for (int i = 0; i < nrc; i++) rebuilt[ibase + i] = (loc[i] - 1) % nb + 1;        // rebuild_val: mod2(local, nb)
  if (F.parent[c] < 0) return;
  int ss = ncc % nb;                                                                // border_supernode_size
  int ws = min(nb - ss, nrc);                                                       // border_work_size
  int g = group_base[t] - 2, pp = 0, pc = 0;                                       // 0-based, before the first group
  for (int i = 0; i < nrc; i++) {
    int pt, ct;
    bli_key(loc[i], i, ncc, nb, pt, ct);
    if (pt != pp || ct != pc) {
      pp = pt; pc = ct; g++;
      pnum[g] = pt;
      cnum[g] = ct;
      block_ptr[g] = ibase + i + 1;                                                 // 1-based start of the group
      int s = i + 1;                                                                // get_start_row_num
      offset[g] = s <= ws ? s - 1 : (ss + s - 1) % nb;                              // get_block_offset
    }
  }
}

// ============================================================================
// factorization
// ============================================================================

// Inverse of a child's local index: for every position of the parent front the
// child's row there, or -1 (children of large fronts, at F.inv_off).
__global__ void k_inverse_index(DevFronts F, const int32_t* kids, int32_t* inv) {
  const int c = kids[blockIdx.x], p = F.parent[c];
  const int nfp = F.nc[p] + F.nr[p], nrc = F.nr[c];
  int32_t* v = inv + F.inv_off[c];
  for (int i = threadIdx.x; i < nfp; i += blockDim.x) v[i] = -1;
  __syncthreads();
  const int32_t* loc = F.local + F.lrow_off[c];
  for (int i = threadIdx.x; i < nrc; i += blockDim.x) v[loc[i] - 1] = i;
}

// Extend-add of a level's large fronts, gathered: every lower entry of a
// front's panel and update matrix is written once, as the sum of its children's
// entries there in child order (zero where no child has one; more than two
// children are taken two at a time).  A warp takes the column pair (j, nf-1-j),
// nf + 1 entries whatever j, lanes over rows, four rows of two children in
// flight; a child without column j costs nothing.
// What bounds it is HBM: per entry two reads and one write, where zeroing and
// one scatter launch per child rank moved seven (64^3 Laplacian, FP64: 6.5 ms
// a factorization in 78 launches).
template <typename T>
__global__ void __launch_bounds__(256) k_gather_children(DevFronts F, const int32_t* list, T* panel, T* upool) {
  constexpr int U = 4;
  const int f = list[blockIdx.y];
  const int nc = F.nc[f], nr = F.nr[f], nf = nc + nr;
  T* P = panel + F.panel_off[f];
  T* Uf = upool + F.u_off[f];
  const int cb = F.child_ptr[f], nch = F.child_ptr[f + 1] - cb;
  const int ce = nch > kManyChildren ? cb : cb + nch;    // many: zero only
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int pairs = (nf + 1) / 2;
  for (int q = blockIdx.x * nw + warp; q < pairs; q += gridDim.x * nw) {
#pragma unroll 1
    for (int hh = 0; hh < 2; ++hh) {
      const int j = hh ? nf - 1 - q : q;
      if (hh && j == q) break;
      T* dst = j < nc ? P + (size_t)j * nf : Uf + (size_t)(j - nc) * nr - nc;   // entry (i, j) at dst[i]
#pragma unroll 1
      for (int t0 = cb; t0 == cb || t0 < ce; t0 += 2) {
        const int32_t* iv[2] = {nullptr, nullptr};
        const T* col[2] = {nullptr, nullptr};
#pragma unroll
        for (int s = 0; s < 2; ++s)
          if (t0 + s < ce) {
            const int c = F.child[t0 + s];
            const int32_t* v = F.inv + F.inv_off[c];
            const int cj = v[j];
            if (cj >= 0) {
              iv[s] = v;
              col[s] = upool + F.u_off[c] + (size_t)cj * F.nr[c];
            }
          }
        const bool first = t0 == cb;
        if (!first && iv[0] == nullptr && iv[1] == nullptr) continue;
        for (int i0 = j + lane; i0 < nf; i0 += 32 * U) {
          int ci[2][U];
          T x[2][U], d[U];
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int i = i0 + 32 * u;
#pragma unroll
            for (int s = 0; s < 2; ++s) ci[s][u] = iv[s] != nullptr && i < nf ? __ldg(iv[s] + i) : -1;
            d[u] = !first && i < nf ? dst[i] : T(0);
          }
#pragma unroll
          for (int u = 0; u < U; ++u)
#pragma unroll
            for (int s = 0; s < 2; ++s) x[s][u] = ci[s][u] >= 0 ? col[s][ci[s][u]] : T(0);
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int i = i0 + 32 * u;
            if (i < nf) dst[i] = (d[u] + x[0][u]) + x[1][u];
          }
        }
      }
    }
  }
}

// A's entries of the large fronts, each with its children's contributions on
// top (A first, then the children in order): written over what the gather put
// there, so that an entry of A is set, not added.
template <typename T>
__global__ void k_assemble_large(DevFronts F, const int32_t* list, const double* __restrict__ a, T* panel,
                                 const T* __restrict__ upool) {
  const int f = list[blockIdx.y];
  const int nf = F.nc[f] + F.nr[f], cb = F.child_ptr[f], nch = F.child_ptr[f + 1] - cb;
  const int ce = nch > kManyChildren ? cb : cb + nch;    // many: added afterwards (k_add_children)
  T* P = panel + F.panel_off[f];
  for (int k = F.a_beg[f] + blockIdx.x * blockDim.x + threadIdx.x; k < F.a_beg[f + 1]; k += gridDim.x * blockDim.x) {
    const int pos = F.a_pos[k], j = pos / nf, i = pos - j * nf;
    T v = T(a[F.a_src[k]]);
    for (int t = cb; t < ce; ++t) {
      const int c = F.child[t];
      const int32_t* iv = F.inv + F.inv_off[c];
      const int cj = iv[j], ci = iv[i];
      if (cj >= 0 && ci >= 0) v += upool[F.u_off[c] + ci + (size_t)cj * F.nr[c]];
    }
    P[pos] = v;
  }
}

// The children of a front with many of them, added in child order to what A's
// entries and zeros left there: the same sums in the same order as above.  A warp
// takes the columns j and nf - 1 - j; its lanes look column j up in 32 children at
// a time and those that have it are added one after another, lanes over their rows.
// Both sides are at kManyChildren.
template <typename T>
__global__ void __launch_bounds__(256) k_add_children(DevFronts F, const int32_t* list, T* panel, T* upool) {
  const int f = list[blockIdx.y];
  const int nc = F.nc[f], nr = F.nr[f], nf = nc + nr;
  T* P = panel + F.panel_off[f];
  T* Uf = upool + F.u_off[f];
  const int cb = F.child_ptr[f], ce = F.child_ptr[f + 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int pairs = (nf + 1) / 2;
  for (int q = blockIdx.x * nw + warp; q < pairs; q += gridDim.x * nw)
#pragma unroll 1
    for (int hh = 0; hh < 2; ++hh) {
      const int j = hh ? nf - 1 - q : q;
      if (hh && j == q) break;
      T* dst = j < nc ? P + (size_t)j * nf : Uf + (size_t)(j - nc) * nr - nc;   // entry (i, j) at dst[i]
      for (int t0 = cb; t0 < ce; t0 += 32) {
        int cnr = 0, clo = 0, cj = 0;
        long long cuo = 0;
        bool has = false;
        if (t0 + lane < ce) {
          const ChildRec c = F.crec[t0 + lane];
          cnr = c.nr; clo = c.lrow_off; cuo = c.u_off;
          cj = lower_bound_dev(F.local + clo, cnr, j + 1);
          has = cj < cnr && F.local[clo + cj] == j + 1;
        }
        for (unsigned m = __ballot_sync(0xffffffffu, has); m; m &= m - 1) {
          const int s = __ffs(m) - 1;
          const int n = __shfl_sync(0xffffffffu, cnr, s), c = __shfl_sync(0xffffffffu, cj, s);
          const int32_t* loc = F.local + __shfl_sync(0xffffffffu, clo, s);
          const T* col = upool + __shfl_sync(0xffffffffu, cuo, s) + (size_t)c * n;
          for (int r = c + lane; r < n; r += 32) dst[loc[r] - 1] += col[r];
          __syncwarp();                                  // the next child's rows may be other lanes'
        }
      }
    }
}

// Inverted diagonal block of panel step `step` of front f (k_invert writes them).
template <typename T>
__device__ __forceinline__ T* inv_block(const DevFronts& F, T* linv, int f, int step) {
  return linv + F.d_off[f] + (size_t)step * kFactB * kFactB;
}

template <typename T>
__device__ __forceinline__ T* trailing_addr(T* P, T* U, int nc, int nr, int nf, int gi, int gj) {
  return gj < nc ? P + gi + (size_t)gj * nf : U + (gi - nc) + (size_t)(gj - nc) * nr;
}

// Trailing update on the FP64 tensor pipe: one 128x128 tile of the trailing
// lower triangle per CTA, C -= P_i P_j^T over the K range of the step's
// deferred group (update_k_range: up to defer x 128 panel columns) in chunks
// of 32, double-buffered with cp.async.  16 warps as 4 (rows) x 4 (columns) of 32x32,
// each 2 x 4 mma.m16n8k16.f64 per K step of 16.  Shared-memory operands are
// k-major with a row stride of 132 doubles (= 4 mod 16): every fragment load of
// a half-warp hits 16 distinct 8-byte bank pairs.  The accumulators are loaded
// with C itself (8 rows x 4 column pairs per warp access: full 32-byte
// sectors) while the first operand chunk is in flight, the A fragments enter
// negated, and the epilogue only stores.
constexpr int kUT = 128, kUK = 32, kULD = 132;
constexpr int kUThreads = 512;              // 16 warps: 4 (rows) x 4 (columns) of 32 x 32
constexpr int kUMF = kUT / (kUThreads / 32 / 4) / 16;   // m16 fragments per warp (2)

__device__ __forceinline__ void dmma16(double (&d)[4], const double (&a)[8], const double (&b)[4]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7,%8,%9,%10,%11}, "
      "{%12,%13,%14,%15}, {%0,%1,%2,%3};\n"
      : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(a[4]), "d"(a[5]), "d"(a[6]), "d"(a[7]), "d"(b[0]),
        "d"(b[1]), "d"(b[2]), "d"(b[3]));
}

__global__ void __launch_bounds__(kUThreads, 1) k_update_dmma(DevFronts F, const int32_t* list, int step, double* panel,
                                                        double* upool, int blo, int bhi, int defer) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* sm = reinterpret_cast<double*>(smem_raw);     // [stage][operand][k][row]
  const int f = list[blockIdx.y];
  const int nc = F.nc[f], nr = F.nr[f], nf = nc + nr;
  const int c0 = step * kFactB;
  if (c0 >= nc) return;
  const int w = min(kFactB, nc - c0);
  const int base = c0 + w;
  const int nrem = nf - base;
  if (nrem <= 0) return;
  const int T = (nrem + kUT - 1) / kUT;
  int ti, tj, kbeg, kend;
  if (!select_tile(T, kUT, blo, bhi, blockIdx.x, ti, tj)) return;
  if (!update_k_range(nc, step, defer, tj, kUT, kbeg, kend)) return;
  const int K = kend - kbeg;                            // panel columns [kbeg, kend) of the front
  const int i0 = base + ti * kUT, j0 = base + tj * kUT;
  double* P = panel + F.panel_off[f];
  double* U = upool + F.u_off[f];
  const int nchunks = (K + kUK - 1) / kUK;
  const bool diag = ti == tj;
  auto load = [&](int stage, int kc) {
    double* dst = sm + stage * (2 * kUK * kULD);
    const int ops = diag ? 1 : 2;                       // a diagonal tile's B is its A
    for (int e = threadIdx.x; e < ops * kUK * kUT; e += blockDim.x) {
      const int op = e / (kUK * kUT), rem = e - op * (kUK * kUT);
      const int k = rem / kUT, r = rem - k * kUT;
      const int row = (op == 0 ? i0 : j0) + r, col = kc * kUK + k;
      const bool valid = row < nf && col < K;
      const double* src = valid ? P + row + (size_t)(kbeg + col) * nf : P;
      cp_async8(dst + op * (kUK * kULD) + k * kULD + r, src, valid);
    }
    cp_async_commit();
  };
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wm = warp >> 2, wn = warp & 3;
  const int g = lane >> 2, q = lane & 3;
  // the accumulators start as C (loads in flight with the first operand chunk) and the
  // A fragments enter negated, so the tile ends as C - P_i P_j^T and the epilogue only stores
  const int rbase = i0 + wm * (16 * kUMF) + g, cbase = j0 + wn * 32 + 2 * q;
  // C may be written by a kernel this one waits on through an event (the
  // lookahead's side stream): everything is read after the wait
  pdl_wait();
  pdl_trigger();
  double acc[kUMF][4][4];
#pragma unroll
  for (int mi = 0; mi < kUMF; ++mi)
#pragma unroll
    for (int ni = 0; ni < 4; ++ni)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int gi = rbase + mi * 16 + 8 * (e >> 1), gj = cbase + ni * 8 + (e & 1);
        acc[mi][ni][e] = (gi < nf && gj < nf && gi >= gj) ? *trailing_addr(P, U, nc, nr, nf, gi, gj) : 0.0;
      }
  load(0, 0);
  for (int kc = 0; kc < nchunks; ++kc) {
    if (kc + 1 < nchunks) {
      load((kc + 1) & 1, kc + 1);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    const double* As = sm + (kc & 1) * (2 * kUK * kULD);
    const double* Bs = diag ? As : As + kUK * kULD;
#pragma unroll
    for (int kk = 0; kk < kUK; kk += 16) {
      double bv[4][4];
#pragma unroll
      for (int ni = 0; ni < 4; ++ni)
#pragma unroll
        for (int i = 0; i < 4; ++i) bv[ni][i] = Bs[(kk + q + 4 * i) * kULD + wn * 32 + ni * 8 + g];
#pragma unroll
      for (int mi = 0; mi < kUMF; ++mi) {
        double av[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) av[i] = -As[(kk + q + 4 * (i >> 1)) * kULD + wm * (16 * kUMF) + mi * 16 + g + 8 * (i & 1)];
#pragma unroll
        for (int ni = 0; ni < 4; ++ni) dmma16(acc[mi][ni], av, bv[ni]);
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int mi = 0; mi < kUMF; ++mi)
#pragma unroll
    for (int ni = 0; ni < 4; ++ni)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int gi = rbase + mi * 16 + 8 * (e >> 1), gj = cbase + ni * 8 + (e & 1);
        if (gi < nf && gj < nf && gi >= gj) *trailing_addr(P, U, nc, nr, nf, gi, gj) = acc[mi][ni][e];
      }
}

// FP64 trailing update in WM x WN warps of 32 x 32 outputs: a CTA computes one
// (32 WM) x (32 WN) piece of a square tile of the band (the same tiles, bands
// and K ranges as k_update_dmma), 2 x 4 mma.m16n8k16.f64 per warp and K step
// of 16.  Two shapes:
//   <4, 2>, 128 x 64: 128 registers and 102 KB of shared memory, two CTAs per
//     SM: one CTA's C loads and stores overlap the other's MMAs;
//   <2, 1>, 64 x 32: 54 KB, four CTAs per SM, for launches whose 128 x 64
//     pieces would leave SMs idle (launch_update).
// Operands come in K chunks of 32 by cp.async (16-byte row pairs where
// aligned), double-buffered; a 128-row diagonal tile's B is in its A.  C is
// loaded into the accumulators (the A fragments enter negated) and stored
// back; pieces wholly inside the trailing matrix, below the diagonal and
// inside the panel or the update matrix take an unchecked path.  Warps whose
// 32 rows all lie above the diagonal skip the MMAs.  Every element sees the
// same K sequence in either shape: the results are bitwise the same.
template <int WM, int WN>
struct UpdShape {
  static constexpr int kThreads = 32 * WM * WN, kM = 32 * WM, kN = 32 * WN;
  static constexpr int kLdA = kM + 4, kLdB = kN + 4;          // = 4 mod 16 doubles: conflict-free fragments
  static constexpr int kStage = kUK * (kLdA + kLdB);          // doubles per pipeline stage
  static constexpr size_t kSmem = 2 * (size_t)kStage * sizeof(double);
  static constexpr int kPerTile = (kUT / kM) * (kUT / kN);    // pieces of a 128 x 128 tile
};

template <int WM, int WN>
__global__ void __launch_bounds__(32 * WM * WN, WM * WN == 8 ? 2 : 4) k_update_dmma2(DevFronts F, const int32_t* list, int step,
                                                              double* panel, double* upool, int blo, int bhi,
                                                              int defer) {
  using Sh = UpdShape<WM, WN>;
  constexpr int kM = Sh::kM, kN = Sh::kN;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* sm = reinterpret_cast<double*>(smem_raw);     // per stage: A [k][kLdA] (kM rows), B [k][kLdB] (kN rows)
  const int f = list[blockIdx.y];
  const int nc = F.nc[f], nr = F.nr[f], nf = nc + nr;
  const int c0 = step * kFactB;
  if (c0 >= nc) return;
  const int w = min(kFactB, nc - c0);
  const int base = c0 + w;
  const int nrem = nf - base;
  if (nrem <= 0) return;
  const int T = (nrem + kUT - 1) / kUT;
  const int piece = blockIdx.x % Sh::kPerTile, hf = piece % (kUT / kN), rf = piece / (kUT / kN);
  int ti, tj, kbeg, kend;
  if (!select_tile(T, kUT, blo, bhi, blockIdx.x / Sh::kPerTile, ti, tj)) return;
  if (!update_k_range(nc, step, defer, tj, kUT, kbeg, kend)) return;
  const int i0 = base + ti * kUT + rf * kM, j0 = base + tj * kUT + hf * kN;
  if (i0 >= nf || j0 >= nf || i0 + kM <= j0) return;    // beyond the matrix, or above the diagonal
  const int K = kend - kbeg;                            // panel columns [kbeg, kend) of the front
  const bool diag = kM == kUT && ti == tj;
  double* P = panel + F.panel_off[f];
  double* U = upool + F.u_off[f];
  const int nchunks = (K + kUK - 1) / kUK;
  // Copies: thread t moves row pairs -- A rows i0 + 2 (t % (kM / 2)) (+1) at
  // columns t / (kM / 2) + kStepA v; B rows and columns likewise -- 16 bytes
  // per copy when the pair's source is 16-byte aligned.  A thread's copies are
  // an even number of columns apart, so the alignment is the same for all of
  // them; otherwise two 8-byte copies.  Rows past the matrix and columns past
  // K are zero-filled.
  constexpr int kStepA = Sh::kThreads / (kM / 2), kStepB = Sh::kThreads / (kN / 2);
  static_assert(kStepA % 2 == 0 && kStepB % 2 == 0, "alignment per thread");
  auto copy = [&](double* d, const double* src, int bytes, bool al) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(d);
    if (al) {
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(sa), "l"(bytes ? src : P), "r"(bytes));
    } else {
      const int b0 = bytes >= 8 ? 8 : 0, b1 = bytes >= 16 ? 8 : 0;
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(sa), "l"(b0 ? src : P), "r"(b0));
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(sa + 8), "l"(b1 ? src + 1 : P), "r"(b1));
    }
  };
  auto load = [&](int stage, int kc) {
    // the per-thread quantities are recomputed here (kept live they would spill)
    const int pa = threadIdx.x % (kM / 2), ka = threadIdx.x / (kM / 2);
    const int ra = i0 + 2 * pa;
    const int na = ra < nf ? (ra + 1 < nf ? 16 : 8) : 0;          // bytes of the A pair inside the matrix
    const bool ala = ((ra + (long long)(kbeg + ka) * nf) & 1) == 0; // panel offsets are multiples of 32 elements
    double* dst = sm + stage * Sh::kStage;
    const int k0 = kc * kUK;
    const double* sa = P + ra + (size_t)(kbeg + k0 + ka) * nf;
    double* da = dst + ka * Sh::kLdA + 2 * pa;
#pragma unroll 1
    for (int v = 0; v < kUK / kStepA; ++v) {        // rolled: unrolled, the copies' addresses would be kept live
      const int k = k0 + ka + kStepA * v;
      copy(da + v * kStepA * Sh::kLdA, sa + (size_t)(kStepA * v) * nf, k < K ? na : 0, ala);
    }
    if (diag) return;
    const int pb = threadIdx.x % (kN / 2), kb = threadIdx.x / (kN / 2);
    const int rb = j0 + 2 * pb;
    const int nbb = rb < nf ? (rb + 1 < nf ? 16 : 8) : 0;
    const bool alb = ((rb + (long long)(kbeg + kb) * nf) & 1) == 0;
    const double* sb = P + rb + (size_t)(kbeg + k0 + kb) * nf;
    double* db = dst + kUK * Sh::kLdA + kb * Sh::kLdB + 2 * pb;
#pragma unroll 1
    for (int v = 0; v < kUK / kStepB; ++v) {
      const int k = k0 + kb + kStepB * v;
      copy(db + v * kStepB * Sh::kLdB, sb + (size_t)(kStepB * v) * nf, k < K ? nbb : 0, alb);
    }
  };
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wm = warp / WN, wn = warp % WN;
  const int g = lane >> 2, q = lane & 3;
  const int rbase = i0 + wm * 32 + g, cbase = j0 + wn * 32 + 2 * q;
  // warps of a diagonal tile whose rows all lie above the diagonal
  const bool idle = i0 + wm * 32 + 31 < j0 + wn * 32;
  // unchecked path: the tile is inside the trailing matrix, wholly below the
  // diagonal and wholly in the panel or wholly in the update matrix (formed
  // again for the epilogue rather than kept live through the K loop)
  auto full_tile = [&]() { return i0 + kM <= nf && j0 + kN <= nf && i0 >= j0 + kN && (j0 + kN <= nc || j0 >= nc); };
  auto c_base = [&]() { return j0 < nc ? P + (size_t)j0 * nf : U + (size_t)(j0 - nc) * nr - nc; };   // C(gi, gj) = Cb[gi + (gj - j0) ldc]
  pdl_wait();
  pdl_trigger();
  load(0, 0);
  cp_async_commit();
  double acc[2][4][4];
  {
  const bool full = full_tile();
  const int ldc = j0 < nc ? nf : nr;
  double* Cb = c_base();
#pragma unroll
  for (int mi = 0; mi < 2; ++mi)
#pragma unroll
    for (int ni = 0; ni < 4; ++ni)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int gi = rbase + mi * 16 + 8 * (e >> 1), gj = cbase + ni * 8 + (e & 1);
        if (full)
          acc[mi][ni][e] = Cb[gi + (size_t)(gj - j0) * ldc];
        else
          acc[mi][ni][e] = (!idle && gi < nf && gj < nf && gi >= gj) ? *trailing_addr(P, U, nc, nr, nf, gi, gj) : 0.0;
      }
  }
  for (int kc = 0; kc < nchunks; ++kc) {
    if (kc + 1 < nchunks) {
      load((kc + 1) & 1, kc + 1);
      cp_async_commit();
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    if (!idle) {
      const double* As = sm + (kc & 1) * Sh::kStage;
      const double* Bs = diag ? As + hf * kN : As + kUK * Sh::kLdA;
      const int ldb = diag ? Sh::kLdA : Sh::kLdB;
#pragma unroll
      for (int kk = 0; kk < kUK; kk += 16) {
        double bv[4][4];
#pragma unroll
        for (int ni = 0; ni < 4; ++ni)
#pragma unroll
          for (int i = 0; i < 4; ++i) bv[ni][i] = Bs[(kk + q + 4 * i) * ldb + wn * 32 + ni * 8 + g];
#pragma unroll
        for (int mi = 0; mi < 2; ++mi) {
          double av[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) av[i] = -As[(kk + q + 4 * (i >> 1)) * Sh::kLdA + wm * 32 + mi * 16 + g + 8 * (i & 1)];
#pragma unroll
          for (int ni = 0; ni < 4; ++ni) dmma16(acc[mi][ni], av, bv[ni]);
        }
      }
    }
    __syncthreads();
  }
  if (idle) return;
  const bool full = full_tile();
  const int ldc = j0 < nc ? nf : nr;
  double* Cb = c_base();
#pragma unroll
  for (int mi = 0; mi < 2; ++mi)
#pragma unroll
    for (int ni = 0; ni < 4; ++ni)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int gi = rbase + mi * 16 + 8 * (e >> 1), gj = cbase + ni * 8 + (e & 1);
        if (full)
          Cb[gi + (size_t)(gj - j0) * ldc] = acc[mi][ni][e];
        else if (gi < nf && gj < nf && gi >= gj)
          *trailing_addr(P, U, nc, nr, nf, gi, gj) = acc[mi][ni][e];
      }
}

// Trailing update on the FMA pipes (any T): 64x64 tiles, K in chunks of 64,
// 256 threads each 4x4 outputs (rows ty+16m, columns tx+16n).
constexpr int kSimtTile = 64, kSimtK = 64;
template <typename T>
__global__ void __launch_bounds__(256) k_update_simt(DevFronts F, const int32_t* list, int step, T* panel, T* upool,
                                                     int blo, int bhi, int defer) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int LDK = kSimtTile + 4;
  T* As = reinterpret_cast<T*>(smem_raw);
  T* Bs = As + kSimtK * LDK;
  const int f = list[blockIdx.y];
  const int nc = F.nc[f], nr = F.nr[f], nf = nc + nr;
  const int c0 = step * kFactB;
  if (c0 >= nc) return;
  const int w = min(kFactB, nc - c0);
  const int base = c0 + w;
  const int nrem = nf - base;
  if (nrem <= 0) return;
  const int Tn = (nrem + kSimtTile - 1) / kSimtTile;
  int ti, tj, kbeg, kend;
  if (!select_tile(Tn, kSimtTile, blo, bhi, blockIdx.x, ti, tj)) return;
  if (!update_k_range(nc, step, defer, tj, kSimtTile, kbeg, kend)) return;
  const int K = kend - kbeg;
  const int i0 = base + ti * kSimtTile, j0 = base + tj * kSimtTile;
  T* P = panel + F.panel_off[f];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  T acc[4][4];
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int n = 0; n < 4; ++n) acc[m][n] = T(0);
  for (int k0 = 0; k0 < K; k0 += kSimtK) {
    const int kw = min(kSimtK, K - k0);
    __syncthreads();
    batched_loop(
        2 * kSimtTile * kw,
        [&](int e) {
          const int op = e / (kSimtTile * kw), rem = e - op * (kSimtTile * kw);
          const int k = rem / kSimtTile, g = (op ? j0 : i0) + rem % kSimtTile;
          return g < nf ? P[g + (size_t)(kbeg + k0 + k) * nf] : T(0);
        },
        [&](int e, T v) {
          const int op = e / (kSimtTile * kw), rem = e - op * (kSimtTile * kw);
          (op ? Bs : As)[(rem / kSimtTile) * LDK + rem % kSimtTile] = v;
        });
    __syncthreads();
    for (int k = 0; k < kw; ++k) {
      T av[4], bv[4];
#pragma unroll
      for (int m = 0; m < 4; ++m) av[m] = As[k * LDK + ty + 16 * m];
#pragma unroll
      for (int n = 0; n < 4; ++n) bv[n] = Bs[k * LDK + tx + 16 * n];
#pragma unroll
      for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int n = 0; n < 4; ++n) acc[m][n] += av[m] * bv[n];
    }
  }
  T* U = upool + F.u_off[f];
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      int gi = i0 + ty + 16 * m, gj = j0 + tx + 16 * n;
      if (gi < nf && gj < nf && gi >= gj) *trailing_addr(P, U, nc, nr, nf, gi, gj) -= acc[m][n];
    }
}

// ============================================================================
// solves
// ============================================================================

// ---- large fronts: the solve vector of front f lives in V (nf per RHS) --------
// Panel steps of kSolveB = 128 columns use the inverted diagonal blocks kept
// from the factorization (Li = L_ss^{-1}), one launch per step:
//   forward : v_rest -= L_rest,s y_s over 32-row chunks (k_fwd_large_rest);
//             the last CTA of the front to finish (ticket) then forms the next
//             step's y_{s+1} = Li v_{s+1}; y_0 is formed by the gather kernel
//   backward: t_s = v_s - L_rest,s^T x_rest, partial sums per 64-row chunk;
//             the last CTA sums them in chunk order (deterministic) and forms
//             x_s = Li^T t_s (k_bwd_large_step)
// The diagonal solves write the front's own entries of X directly.  Grid z takes kRhsG right-hand
// sides, with a ticket of its own: one group after another in the same CTAs, 64 right-hand sides on
// the 64^3 Laplacian took 91.9 ms (FP64) and 130 ms (FP32 + refinement), side by side 38 and 53.
constexpr int kFwdRows = 32;  // rows per CTA of k_fwd_large_rest

// y_s = Li v_s by one CTA of 256 threads: thread (row i, half h) sums k in
// [64h, 64h + 64) for a group of 8 right-hand sides (Li is zero above its
// diagonal and outside w x w, so the loops have fixed trip counts and the
// loads pipeline); halves meet in shared memory.  v is read past L1: other
// CTAs wrote it.
template <typename T>
__device__ void fwd_diag_cta(const DevFronts& F, int f, int step, int slot, const T* __restrict__ dinv, T* X,
                             int64_t ldx, T* Vf, int nf, int rb, int re, T* vs, T* hs) {
  const int nc = F.nc[f];
  const int c0 = step * kSolveB;
  const int w = min(kSolveB, nc - c0);
  const T* Li = inv_block(F, dinv, f, step);
  const int first = F.first[f];
  const int tid = threadIdx.x, i = tid & (kSolveB - 1), h = tid >> 7;
  for (int r0 = rb; r0 < re; r0 += kRhsG) {
    const int g = min(kRhsG, re - r0);
    __syncthreads();
    for (int e = tid; e < kSolveB * kRhsG; e += blockDim.x) {
      const int k = e % kSolveB, r = e / kSolveB;
      vs[k * kRhsG + r] = (k < w && r < g) ? __ldcg(&Vf[(int64_t)(r0 + r) * nf + c0 + k]) : T(0);
    }
    __syncthreads();
    T acc[kRhsG];
#pragma unroll
    for (int u = 0; u < kRhsG; ++u) acc[u] = T(0);
#pragma unroll 16
    for (int kk = 0; kk < kSolveB / 2; ++kk) {
      const int k = h * (kSolveB / 2) + kk;
      const T l = Li[i + k * kSolveB];
#pragma unroll
      for (int u = 0; u < kRhsG; ++u) acc[u] += l * vs[k * kRhsG + u];
    }
    if (h == 1)
#pragma unroll
      for (int u = 0; u < kRhsG; ++u) hs[i * kRhsG + u] = acc[u];
    __syncthreads();
    if (h == 0 && i < w) {
#pragma unroll
      for (int u = 0; u < kRhsG; ++u) {
        if (u < g) {
          const T y = acc[u] + hs[i * kRhsG + u];
          const int r = r0 + u;
          Vf[(int64_t)r * nf + c0 + i] = y;
          X[first + c0 + i + r * ldx] = y;
        }
      }
    }
  }
}

// The vectors of fronts with many children before their panel steps (sweep_sync.cuh
// has the other fronts' form): own X entries plus the children's update vectors in
// child order, in FP64.  A warp takes 32 rows of R right-hand sides in shared
// memory; its lanes look for rows in their range in 32 children at a time, and the
// entries of C of those that have some, at most one per lane and child, are in
// flight together.  Front of 300 columns, 20,000 children of five rows: one
// right-hand side 7.0 -> 2.2 ms a solve (each row looked up in every child before),
// five 5.6 -> 3.3 (one child after another: 11.6).
constexpr int kGatherRows = 32, kGatherWarps = 4;
template <typename T, int R, int C>
__global__ void __launch_bounds__(32 * kGatherWarps) k_gather_many(DevFronts F, const int32_t* list, const T* X, int64_t ldx,
                                                                   const T* V, double* G, int nrhs) {
  __shared__ double acc[kGatherWarps][R][kGatherRows];
  const int f = list[blockIdx.y];
  const int nc = F.nc[f], nf = nc + F.nr[f], first = F.first[f];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int i0 = (blockIdx.x * kGatherWarps + warp) * kGatherRows, i1 = min(nf, i0 + kGatherRows);
  const int r0 = blockIdx.z * R, rn = min(R, nrhs - r0);
  if (i0 >= nf) return;
  double (*a)[kGatherRows] = acc[warp];
#pragma unroll
  for (int r = 0; r < R; ++r)
    a[r][lane] = r < rn && i0 + lane < nc ? (double)X[first + i0 + lane + (int64_t)(r0 + r) * ldx] : 0.0;
  __syncwarp();
  const int cb = F.child_ptr[f], ce = F.child_ptr[f + 1];
  for (int t0 = cb; t0 < ce; t0 += 32) {
    int cnr = 0, cnc = 0, clo = 0, at = 0;
    long long cvo = 0;
    bool has = false;
    if (t0 + lane < ce) {
      const ChildRec c = F.crec[t0 + lane];
      cnr = c.nr; cnc = c.nc; clo = c.lrow_off; cvo = c.v_off;
      at = lower_bound_dev(F.local + clo, cnr, i0 + 1);
      has = at < cnr && F.local[clo + at] <= i1;
    }
    unsigned m = __ballot_sync(0xffffffffu, has);
    while (m) {
      int i[C];
      T v[C][R];
#pragma unroll
      for (int u = 0; u < C; ++u) {
        const int s = m ? __ffs(m) - 1 : 0;
        const int n = __shfl_sync(0xffffffffu, cnr, s), cols = __shfl_sync(0xffffffffu, cnc, s);
        const int e = __shfl_sync(0xffffffffu, at, s) + lane;
        const int32_t* loc = F.local + __shfl_sync(0xffffffffu, clo, s);
        const T* vc = V + __shfl_sync(0xffffffffu, cvo, s) * nrhs + (int64_t)r0 * (cols + n) + cols;
        i[u] = m && e < n ? loc[e] - 1 : i1;
#pragma unroll
        for (int r = 0; r < R; ++r) v[u][r] = i[u] < i1 && r < rn ? vc[(int64_t)r * (cols + n) + e] : T(0);
        m &= m - 1;                                      // stays 0
      }
#pragma unroll
      for (int u = 0; u < C; ++u) {
        if (i[u] < i1)
#pragma unroll
          for (int r = 0; r < R; ++r) a[r][i[u] - i0] += (double)v[u][r];
        __syncwarp();
      }
    }
  }
  double* g = G + F.g_off[f] * nrhs + (int64_t)r0 * nf + i0 + lane;
  if (i0 + lane < nf)
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (r < rn) g[(int64_t)r * nf] = a[r][lane];
}

// gather v (own X entries + the children's update vectors), then y_0
template <typename T>
__global__ void __launch_bounds__(256) k_fwd_large_gather(DevFronts F, const int32_t* list,
                                                          const T* __restrict__ dinv, T* X, int64_t ldx, T* V,
                                                          int nrhs) {
  __shared__ T vs[kSolveB * kRhsG];
  __shared__ T hs[kSolveB * kRhsG];
  const int f = list[blockIdx.x];
  const int nc = F.nc[f], nf = nc + F.nr[f], first = F.first[f];
  T* Vbase = V + F.v_off[f] * nrhs;
  const int rb = blockIdx.z * kRhsG, re = min(nrhs, rb + kRhsG);
  // loads batched kGU per thread (in flight together); each entry takes one
  // add per child, children in order
  constexpr int kGU = 4;
  const int nt = blockDim.x;
  for (int r = rb; r < re; ++r) {
    T* Vf = Vbase + (int64_t)r * nf;
    for (int i0 = threadIdx.x; i0 < nf; i0 += kGU * nt) {
      T xv[kGU];
#pragma unroll
      for (int u = 0; u < kGU; ++u) {
        const int i = i0 + u * nt;
        xv[u] = i < nc ? X[first + i + r * ldx] : T(0);
      }
#pragma unroll
      for (int u = 0; u < kGU; ++u)
        if (i0 + u * nt < nf) Vf[i0 + u * nt] = xv[u];
    }
    __syncthreads();
    for (int t = F.child_ptr[f]; t < F.child_ptr[f + 1]; ++t) {
      const int c = F.child[t];
      const int ncc = F.nc[c], nrc = F.nr[c];
      const T* Vc = V + F.v_off[c] * nrhs + (int64_t)r * (ncc + nrc) + ncc;
      const int32_t* loc = F.local + F.lrow_off[c];
      for (int i0 = threadIdx.x; i0 < nrc; i0 += kGU * nt) {
        int li[kGU];
        T cv[kGU], ov[kGU];
#pragma unroll
        for (int u = 0; u < kGU; ++u) {
          const int i = i0 + u * nt;
          li[u] = i < nrc ? loc[i] - 1 : -1;
          cv[u] = i < nrc ? Vc[i] : T(0);
        }
#pragma unroll
        for (int u = 0; u < kGU; ++u) ov[u] = li[u] >= 0 ? Vf[li[u]] : T(0);
#pragma unroll
        for (int u = 0; u < kGU; ++u)
          if (li[u] >= 0) Vf[li[u]] = ov[u] + cv[u];
      }
      __syncthreads();
    }
  }
  __threadfence_block();
  fwd_diag_cta(F, f, 0, blockIdx.x, dinv, X, ldx, Vbase, nf, rb, re, vs, hs);
}

// v_rest -= L_rest,s y_s: 32 rows per CTA (lane = row), warp q takes panel
// columns 16q .. 16q+15 (held in registers), partial sums reduced in shared
// memory; the front's last CTA then forms y_{s+1}
template <typename T>
__global__ void __launch_bounds__(256) k_fwd_large_rest(DevFronts F, const int32_t* list, int step,
                                                        const T* __restrict__ panel, const T* __restrict__ dinv,
                                                        T* X, int64_t ldx, T* V, int32_t* cnt, int nrhs) {
  __shared__ T part[8][kRhsG][32];
  __shared__ T vs[kSolveB * kRhsG];
  __shared__ T hs[kSolveB * kRhsG];
  __shared__ int last;
  const int f = list[blockIdx.y];
  const int nc = F.nc[f], nf = nc + F.nr[f];
  pdl_wait();            // the previous step (or gather) of the sweep has completed
  pdl_trigger();
  const int c0 = step * kSolveB;
  if (c0 >= nc) return;
  const int w = min(kSolveB, nc - c0);
  const int rs0 = c0 + w;
  const int rbase = rs0 + blockIdx.x * kFwdRows;
  if (rbase >= nf) return;
  const int nchunks = (nf - rs0 + kFwdRows - 1) / kFwdRows;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int i = rbase + lane;
  const bool valid = i < nf;
  const T* P = panel + F.panel_off[f];
  T* Vf = V + F.v_off[f] * nrhs;
  T lr[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    const int col = warp * 16 + k;
    lr[k] = (valid && col < w) ? P[i + (size_t)(c0 + col) * nf] : T(0);
  }
  const int r0 = blockIdx.z * kRhsG, g = min(kRhsG, nrhs - r0);
#pragma unroll
  for (int u = 0; u < kRhsG; ++u) {
    T s = T(0);
    if (u < g) {
      const T* y = Vf + (int64_t)(r0 + u) * nf + c0 + warp * 16;
#pragma unroll
      for (int k = 0; k < 16; ++k)
        if (warp * 16 + k < w) s += lr[k] * y[k];
    }
    part[warp][u][lane] = s;
  }
  __syncthreads();
  {
    const int u = threadIdx.x >> 5;
    if (u < g && valid) {
      T s = T(0);
#pragma unroll
      for (int q = 0; q < 8; ++q) s += part[q][u][lane];
      Vf[(int64_t)(r0 + u) * nf + i] -= s;
    }
  }
  int32_t* ticket = cnt + blockIdx.y * gridDim.z + blockIdx.z;
  if (rs0 >= nc) return;                                 // no next step for this front
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(ticket, 1) == nchunks - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  fwd_diag_cta(F, f, step + 1, blockIdx.y, dinv, X, ldx, Vf, nf, r0, r0 + g, vs, hs);
  if (threadIdx.x == 0) *ticket = 0;
}

template <typename T>
__global__ void k_bwd_large_gather(DevFronts F, const int32_t* list, const T* X, int64_t ldx, T* V, int nrhs) {
  const int f = list[blockIdx.x];
  const int nc = F.nc[f], nf = nc + F.nr[f], first = F.first[f];
  const int32_t* lr = F.lrow + F.lrow_off[f];
  constexpr int kGU = 4;                     // loads in flight per thread
  const int nt = blockDim.x;
  for (int r = blockIdx.z * kRhsG; r < min(nrhs, (int)(blockIdx.z + 1) * kRhsG); ++r) {
    T* Vf = V + F.v_off[f] * nrhs + (int64_t)r * nf;
    for (int i0 = threadIdx.x; i0 < nf; i0 += kGU * nt) {
      int gi[kGU];
#pragma unroll
      for (int u = 0; u < kGU; ++u) {
        const int i = i0 + u * nt;
        gi[u] = i < nc ? first + i : (i < nf ? lr[i - nc] : -1);
      }
      T xv[kGU];
#pragma unroll
      for (int u = 0; u < kGU; ++u) xv[u] = gi[u] >= 0 ? X[gi[u] + r * ldx] : T(0);
#pragma unroll
      for (int u = 0; u < kGU; ++u)
        if (gi[u] >= 0) Vf[i0 + u * nt] = xv[u];
    }
  }
}

constexpr int kBwdG = 4;   // right-hand sides per pass of the backward partial sums

// ---- fused backward step (one launch per panel step) -------------------------
// Backward, any number of right-hand sides: every CTA writes its chunk's
// partial sums (64 rows; warp (g, q) takes rows 32g .. 32g+31 against the
// block's columns 32q .. 32q+31, lane = row, coalesced column reads, 16
// columns at a time, then a butterfly transpose-reduce leaves column kb +
// (l mod 16)'s sum in lane l); the last CTA of the front to finish (its group's ticket)
// sums them in chunk order (deterministic), forms x_s = Li^T t_s, writes V_s
// and X, and resets the ticket.  A front without rows below the block is
// finished by CTA 0 alone.  The finish reads Li straight from memory rather
// than caching a slice per thread, so the whole kernel fits 80 registers and
// three CTAs per SM (measured: 64^3 Laplacian FP64 solve 5.7 -> 5.1 ms).
template <typename T>
__global__ void __launch_bounds__(256, 3) k_bwd_large_step(DevFronts F, const int32_t* list, int step,
                                                        const T* __restrict__ panel, const T* __restrict__ dinv,
                                                        T* X, int64_t ldx, T* V, T* scratch, int32_t* cnt,
                                                        int nrhs) {
  constexpr int CW = kSolveB / 8;
  __shared__ T part[2][kBwdG][kSolveB];
  __shared__ T ts[kSolveB];
  __shared__ int last;
  const int f = list[blockIdx.y];
  const int nc = F.nc[f], nf = nc + F.nr[f];
  pdl_wait();            // the previous step (or gather) of the sweep has completed
  pdl_trigger();
  const int c0 = step * kSolveB;
  if (c0 >= nc) return;
  const int w = min(kSolveB, nc - c0);
  const int rs0 = c0 + w;
  const int nchunks = nf > rs0 ? (nf - rs0 + kSolveRows - 1) / kSolveRows : 0;
  const int rbase = rs0 + blockIdx.x * kSolveRows;
  if ((int)blockIdx.x >= max(nchunks, 1)) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const T* P = panel + F.panel_off[f];
  T* Vf = V + F.v_off[f] * nrhs;
  const int rb = blockIdx.z * kRhsG, re = min(nrhs, rb + kRhsG);
  int32_t* ticket = cnt + blockIdx.y * gridDim.z + blockIdx.z;
  if (nchunks > 0) {
    const int rg = warp & 1, cq = warp >> 1;
    const int i = rbase + rg * 32 + lane;
    const bool valid = i < nf;
    for (int r0 = rb; r0 < re; r0 += kBwdG) {
      const int g = min(kBwdG, re - r0);
      T xi[kBwdG];
#pragma unroll
      for (int u = 0; u < kBwdG; ++u) xi[u] = (valid && u < g) ? Vf[(int64_t)(r0 + u) * nf + i] : T(0);
#pragma unroll 1
      for (int kb = 32 * cq; kb < 32 * cq + 32; kb += 16) {
        T pv[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) pv[j] = (valid && kb + j < w) ? P[i + (size_t)(c0 + kb + j) * nf] : T(0);
#pragma unroll
        for (int u = 0; u < kBwdG; ++u) {
          if (u >= g) break;
          T v[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] = pv[j] * xi[u];
#pragma unroll
          for (int s = 8; s >= 1; s >>= 1) {
            const bool up = (lane & s) != 0;
#pragma unroll
            for (int j = 0; j < s; ++j) {
              const T send = up ? v[j] : v[j + s];
              const T keep = up ? v[j + s] : v[j];
              v[j] = keep + __shfl_xor_sync(0xffffffffu, send, s);
            }
          }
          v[0] += __shfl_xor_sync(0xffffffffu, v[0], 16);
          if (lane < 16) part[rg][u][kb + lane] = v[0];
        }
      }
      __syncthreads();
      for (int e = threadIdx.x; e < g * kSolveB; e += blockDim.x) {
        const int u = e / kSolveB, k = e % kSolveB;
        const T s = part[0][u][k] + part[1][u][k];
        scratch[F.s_off[f] * nrhs + ((int64_t)(r0 + u) * nchunks + blockIdx.x) * kSolveB + k] = s;
      }
      __syncthreads();
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(ticket, 1) == nchunks - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
  }
  // finish: x_s = Li^T (v_s - sum of partials)
  const T* Li = inv_block(F, dinv, f, step);
  const int first = F.first[f];
  for (int r = rb; r < re; ++r) {
    __syncthreads();
    if (threadIdx.x < kSolveB) {
      T s = T(0);
      if (threadIdx.x < w) {
        s = Vf[(int64_t)r * nf + c0 + threadIdx.x];
        const T* pr = scratch + F.s_off[f] * nrhs + (int64_t)r * nchunks * kSolveB + threadIdx.x;
        for (int q0 = 0; q0 < nchunks; q0 += 8) {   // other CTAs' partials (read past L1), 8 loads in flight,
          T pv[8];                                   // subtracted in chunk order
#pragma unroll
          for (int q = 0; q < 8; ++q) pv[q] = q0 + q < nchunks ? __ldcg(pr + (int64_t)(q0 + q) * kSolveB) : T(0);
#pragma unroll
          for (int q = 0; q < 8; ++q) s -= pv[q];
        }
      }
      ts[threadIdx.x] = s;
    }
    __syncthreads();
    T tv[kSolveB / 32];
#pragma unroll
    for (int q = 0; q < kSolveB / 32; ++q) tv[q] = ts[lane + 32 * q];
#pragma unroll 4
    for (int cc = 0; cc < CW; ++cc) {   // Li(lane + 32q, warp*CW + cc), read here (registers for the partial phase)
      const T* lcol = Li + (size_t)(warp * CW + cc) * kSolveB + lane;
      T s = T(0);
#pragma unroll
      for (int q = 0; q < kSolveB / 32; ++q) s += lcol[32 * q] * tv[q];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      const int i = warp * CW + cc;
      if (lane == 0 && i < w) {
        Vf[(int64_t)r * nf + c0 + i] = s;
        X[first + c0 + i + r * ldx] = s;
      }
    }
  }
  if (nchunks > 0 && threadIdx.x == 0) *ticket = 0;
}

// ============================================================================
// vectors
// ============================================================================
template <typename T>
__global__ void k_permute_in(const double* b, int64_t ldb, const int32_t* perm, T* X, int64_t ldx, int64_t n, int nrhs) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    int64_t src = perm[i];
    for (int r = 0; r < nrhs; ++r) X[i + r * ldx] = T(b[src + r * ldb]);
  }
}
template <typename T>
__global__ void k_permute_out(const T* X, int64_t ldx, const int32_t* perm, double* b, int64_t ldb, int64_t n, int nrhs) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    int64_t dst = perm[i];
    for (int r = 0; r < nrhs; ++r) b[dst + r * ldb] = double(X[i + r * ldx]);
  }
}
__global__ void k_gather_values(const double* a, const int32_t* src, double* out, int64_t count) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = a[src[i]];
}
__global__ void k_residual(const int64_t* rowptr, const int32_t* col, const double* val, const double* x,
                           const double* b, double* r, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    double s = 0.0;
    for (int64_t e = rowptr[i]; e < rowptr[i + 1]; ++e) s += val[e] * x[col[e]];
    r[i] = b[i] - s;
  }
}
__device__ __forceinline__ void atomic_max_nonneg(double* addr, double v) {
  atomicMax(reinterpret_cast<unsigned long long*>(addr), __double_as_longlong(v));
}
// r = b - A x for k columns at once (x row-major: xt[i * k + c]): one warp per
// row, lanes over columns (32 at a time), the row's entries loaded 32 at a
// time and broadcast by shuffles; A is read once for all columns and the
// lanes' reads of a row of x are contiguous.  Entries are summed in row order,
// as in k_residual.
__global__ void k_residual_multi(const int64_t* rowptr, const int32_t* col, const double* val, const double* xt,
                                 const double* b, double* r, int64_t n, int k) {
  const int lane = threadIdx.x & 31;
  const int64_t w0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t i = w0; i < n; i += nw) {
    const int64_t e0 = rowptr[i], e1 = rowptr[i + 1];
    for (int c0 = 0; c0 < k; c0 += 32) {
      const int c = c0 + lane;
      double s = 0.0;
      for (int64_t eb = e0; eb < e1; eb += 32) {
        const int m = (int)min((int64_t)32, e1 - eb);
        int cj = 0;
        double av = 0.0;
        if (lane < m) {
          cj = col[eb + lane];
          av = val[eb + lane];
        }
        for (int t = 0; t < m; ++t) {
          const int j = __shfl_sync(0xffffffffu, cj, t);
          const double a = __shfl_sync(0xffffffffu, av, t);
          if (c < k) s += a * xt[(int64_t)j * k + c];
        }
      }
      if (c < k) r[i + (int64_t)c * n] = b[i + (int64_t)c * n] - s;
    }
  }
}
// column-major n x k (ld n) -> row-major, 32 x 32 tiles through shared memory
__global__ void k_to_rows(const double* x, double* xt, int64_t n, int k) {
  __shared__ double t[32][33];
  const int64_t i0 = (int64_t)blockIdx.x * 32;
  const int c0 = blockIdx.y * 32, tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  for (int c = ty; c < 32; c += 8) t[c][tx] = (i0 + tx < n && c0 + c < k) ? x[i0 + tx + (int64_t)(c0 + c) * n] : 0.0;
  __syncthreads();
  for (int q = ty; q < 32; q += 8)
    if (i0 + q < n && c0 + tx < k) xt[(i0 + q) * k + c0 + tx] = t[tx][q];
}
// per column (grid y): out + 8 c gets max|r|, max|x|, max|b|, sum r^2, sum x^2
__global__ void k_norms(const double* r, const double* x, const double* b, int64_t n, double* out) {
  r += (int64_t)blockIdx.y * n;
  x += (int64_t)blockIdx.y * n;
  b += (int64_t)blockIdx.y * n;
  out += 8 * blockIdx.y;
  double mr = 0, mx = 0, mb = 0, sr = 0, sx = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    double a = fabs(r[i]), c = fabs(x[i]), d = fabs(b[i]);
    mr = fmax(mr, a); mx = fmax(mx, c); mb = fmax(mb, d);
    sr += r[i] * r[i]; sx += x[i] * x[i];
  }
  for (int o = 16; o > 0; o >>= 1) {
    mr = fmax(mr, __shfl_xor_sync(0xffffffffu, mr, o));
    mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    mb = fmax(mb, __shfl_xor_sync(0xffffffffu, mb, o));
    sr += __shfl_xor_sync(0xffffffffu, sr, o);
    sx += __shfl_xor_sync(0xffffffffu, sx, o);
  }
  if ((threadIdx.x & 31) == 0) {
    atomic_max_nonneg(out + 0, mr);
    atomic_max_nonneg(out + 1, mx);
    atomic_max_nonneg(out + 2, mb);
    atomicAdd(out + 3, sr);
    atomicAdd(out + 4, sx);
  }
}
__global__ void k_row_abs_max(const int64_t* rowptr, const double* val, int64_t n, double* out) {
  double m = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    double s = 0;
    for (int64_t e = rowptr[i]; e < rowptr[i + 1]; ++e) s += fabs(val[e]);
    m = fmax(m, s);
  }
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) atomic_max_nonneg(out, m);
}
template <typename T>
__global__ void k_to_t(const double* in, T* out, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = T(in[i]);
}
template <typename T>
__global__ void k_axpy_from_t(const T* d, double* x, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    x[i] += double(d[i]);
}
__global__ void k_fill_int(int32_t* p, int32_t v, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) p[i] = v;
}

inline int grid_1d(int64_t n, int threads = 256) { return clamp_grid(ceil_div(n, threads), kNumSms * 16); }

// Dynamic shared memory above 48 KB is opted into once per kernel at handle
// creation (prepare_kernels), never inside a stream capture.
constexpr int kMaxDynSmem = 227 * 1024;
template <typename KernelT>
cudaError_t opt_in(KernelT k) {
  return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynSmem);
}

}  // namespace

// ============================================================================
// launch wrappers
// ============================================================================
cudaError_t prepare_kernels() {
  cudaError_t e = cudaSuccess;
  auto chk = [&](cudaError_t r) { if (r != cudaSuccess && e == cudaSuccess) e = r; };
  chk(opt_in(k_update_dmma));
  chk(prepare_small_fronts());
  chk(prepare_small_solve());
  chk(prepare_solve_single());
  chk(prepare_panel());
  chk(prepare_update_tc());
  chk(prepare_update_tcq());
  chk(prepare_update_dp());
  chk(opt_in(k_update_simt<double>)); chk(opt_in(k_update_simt<float>));
  chk(opt_in(k_update_dmma2<4, 2>)); chk(opt_in(k_update_dmma2<2, 1>));
  return e;
}

void launch_local_index(const DevFronts& F, int32_t* local, int num_front, cudaStream_t st) {
  if (num_front > 0) k_local_index<<<num_front, 128, 0, st>>>(F, local, num_front);
}
void launch_assembly_map(const DevFronts& F, const int32_t* col_front, const int32_t* acol_ptr, const int32_t* arow,
                         const int32_t* ccs_src, int32_t* sidx, int32_t* a_src, int32_t* a_pos, int n_total,
                         cudaStream_t st) {
  if (n_total > 0)
    k_assembly_map<<<ceil_div(n_total, 256), 256, 0, st>>>(F, col_front, acol_ptr, arow, ccs_src, sidx, a_src, a_pos,
                                                           n_total);
}
void launch_records(const DevFronts& F, const int32_t* lists, int list_len, FrontRec* rec, int num_child,
                    ChildRec* crec, cudaStream_t st) {
  if (list_len > 0) k_front_records<<<ceil_div(list_len, 256), 256, 0, st>>>(F, lists, list_len, rec);
  if (num_child > 0) k_child_records<<<ceil_div(num_child, 256), 256, 0, st>>>(F, num_child, crec);
}
void launch_bli_count(const DevFronts& F, const int32_t* fronts, int count, int nb, int32_t* groups, cudaStream_t st) {
  if (count > 0) k_bli_count<<<ceil_div(count, 128), 128, 0, st>>>(F, fronts, count, nb, groups);
}
void launch_bli_fill(const DevFronts& F, const int32_t* fronts, int count, int nb, const int32_t* group_base,
                     const int32_t* index_base, int32_t* block_ptr, int32_t* pnum, int32_t* cnum, int32_t* offset,
                     int32_t* rebuilt, cudaStream_t st) {
  if (count > 0)
    k_bli_fill<<<ceil_div(count, 128), 128, 0, st>>>(F, fronts, count, nb, group_base, index_base, block_ptr, pnum,
                                                     cnum, offset, rebuilt);
}

void launch_inverse_index(const DevFronts& F, const int32_t* kids, int count, int32_t* inv, cudaStream_t st) {
  if (count > 0) k_inverse_index<<<count, 128, 0, st>>>(F, kids, inv);
}
template <typename T>
void launch_build_large(const DevFronts& F, const int32_t* list, int count, int max_nf, T* panel, T* upool,
                        cudaStream_t st) {
  if (count <= 0) return;
  // one warp per column pair of the largest front, at most 1,024 CTAs per front
  const int gx = std::max(1, std::min(ceil_div((max_nf + 1) / 2, 8), 1024));
  k_gather_children<T><<<dim3(gx, count), 256, 0, st>>>(F, list, panel, upool);
}
template <typename T>
void launch_assemble_large(const DevFronts& F, const int32_t* list, int count, int max_entries, const double* a,
                           T* panel, const T* upool, cudaStream_t st) {
  if (count <= 0) return;
  dim3 grid(clamp_grid(ceil_div(max_entries, 256), 256), count);
  k_assemble_large<T><<<grid, 256, 0, st>>>(F, list, a, panel, upool);
}
template <typename T>
void launch_add_children(const DevFronts& F, const int32_t* many, int count, int max_nf, T* panel, T* upool,
                         cudaStream_t st) {
  if (count <= 0) return;
  const int gx = std::max(1, std::min(ceil_div((max_nf + 1) / 2, 8), 1024));
  k_add_children<T><<<dim3(gx, count), 256, 0, st>>>(F, many, panel, upool);
}
template <typename T>
void launch_gather_many(const DevFronts& F, const int32_t* many, int count, int max_nf, const T* X, int64_t ldx, const T* V,
                        double* G, int nrhs, cudaStream_t st) {
  if (count <= 0) return;
  const int gx = ceil_div(max_nf, kGatherWarps * kGatherRows);
  if (nrhs == 1)
    k_gather_many<T, 1, 8><<<dim3(gx, count), 32 * kGatherWarps, 0, st>>>(F, many, X, ldx, V, G, nrhs);
  else
    k_gather_many<T, 8, 4><<<dim3(gx, count, ceil_div(nrhs, 8)), 32 * kGatherWarps, 0, st>>>(F, many, X, ldx, V, G, nrhs);
}
int update_grid(int T, int tw, UpdBand band) {
  const int c1 = kFactB / tw, jlo = band.blo * c1;
  if (T <= 0 || jlo >= T) return 0;
  if (band.bhi < 0) return (T - jlo) * (T - jlo + 1) / 2;
  return (T - jlo) * ((band.bhi - band.blo) * c1);
}

template <typename T>
int launch_update(const DevFronts& F, const int32_t* list, int count, int step, int T128, int T64, T* panel,
                  T* upool, int kind, cudaStream_t st, UpdBand band, int defer, bool pdl) {
  if (count <= 0) return 0;
  if constexpr (sizeof(T) == 8) {
    if (kind == 0) {
      const int g = update_grid(T128, kUT, band);
      if (g <= 0) return 0;
      auto go = [&](auto kern, auto sh) {
        using Sh = decltype(sh);
        launch_k(kern, dim3(Sh::kPerTile * g, count), dim3(Sh::kThreads), Sh::kSmem, st, pdl, F, list, step,
                 reinterpret_cast<double*>(panel), reinterpret_cast<double*>(upool), band.blo, band.bhi, defer);
      };
      // at most one 128 x 64 piece per SM: four 64 x 32 pieces in its place still fit one wave
      // (four per SM) and take a fourth of its MMAs each
      if ((int64_t)2 * g * count <= kNumSms) go(k_update_dmma2<2, 1>, UpdShape<2, 1>{});
      else go(k_update_dmma2<4, 2>, UpdShape<4, 2>{});
      return 1;
    }
    if (kind == 3) {                                   // whole 128 x 128 tiles, one CTA per SM
      const int g = update_grid(T128, kUT, band);
      if (g <= 0) return 0;
      size_t sm = 2 * 2 * (size_t)kUK * kULD * sizeof(double);
      launch_k(k_update_dmma, dim3(g, count), dim3(kUThreads), sm, st, pdl, F, list, step, reinterpret_cast<double*>(panel),
               reinterpret_cast<double*>(upool), band.blo, band.bhi, defer);
      return 1;
    }
  }
  const int g = update_grid(T64, kSimtTile, band);
  if (g <= 0) return 0;
  size_t sm = 2 * (size_t)kSimtK * (kSimtTile + 4) * sizeof(T);
  k_update_simt<T><<<dim3(g, count), 256, sm, st>>>(F, list, step, panel, upool, band.blo, band.bhi, defer);
  return 1;
}

template <typename T>
void launch_fwd_large(const DevFronts& F, const int32_t* list, int count, int max_nc, int max_nf, const T* panel,
                      const T* dinv, T* X, int64_t ldx, T* V, int32_t* cnt, int nrhs, cudaStream_t st,
                      int64_t* launches, bool pdl) {
  if (count <= 0) return;
  const int gz = ceil_div(nrhs, kRhsG);
  k_fwd_large_gather<T><<<dim3(count, 1, gz), 256, 0, st>>>(F, list, dinv, X, ldx, V, nrhs);
  const int steps = ceil_div(max_nc, kSolveB);
  const int chunks = std::max(1, ceil_div(max_nf, kFwdRows));
  for (int s = 0; s < steps; ++s)
    launch_k(k_fwd_large_rest<T>, dim3(chunks, count, gz), dim3(256), 0, st, pdl, F, list, s, panel, dinv, X, ldx, V, cnt,
             nrhs);
  if (launches) *launches += 1 + steps;
}
template <typename T>
void launch_bwd_large(const DevFronts& F, const int32_t* list, int count, int max_nc, int max_nf, const T* panel,
                      const T* dinv, T* X, int64_t ldx, T* V, T* scratch, int32_t* cnt, int nrhs, cudaStream_t st,
                      int64_t* launches, bool pdl) {
  if (count <= 0) return;
  const int gz = ceil_div(nrhs, kRhsG);
  k_bwd_large_gather<T><<<dim3(count, 1, gz), 256, 0, st>>>(F, list, X, ldx, V, nrhs);
  const int steps = ceil_div(max_nc, kSolveB);
  const int chunks = std::max(1, ceil_div(max_nf, kSolveRows));
  for (int s = steps - 1; s >= 0; --s)
    launch_k(k_bwd_large_step<T>, dim3(chunks, count, gz), dim3(256), 0, st, pdl, F, list, s, panel, dinv, X, ldx, V,
             scratch, cnt, nrhs);
  if (launches) *launches += 1 + steps;
}
template <typename T>
void launch_permute_in(const double* b, int64_t ldb, const int32_t* perm, T* X, int64_t ldx, int64_t n, int nrhs,
                       cudaStream_t st) {
  k_permute_in<T><<<grid_1d(n), 256, 0, st>>>(b, ldb, perm, X, ldx, n, nrhs);
}
template <typename T>
void launch_permute_out(const T* X, int64_t ldx, const int32_t* perm, double* b, int64_t ldb, int64_t n, int nrhs,
                        cudaStream_t st) {
  k_permute_out<T><<<grid_1d(n), 256, 0, st>>>(X, ldx, perm, b, ldb, n, nrhs);
}
void launch_gather_values(const double* a, const int32_t* src, double* out, int64_t count, cudaStream_t st) {
  if (count > 0) k_gather_values<<<grid_1d(count), 256, 0, st>>>(a, src, out, count);
}
void launch_residual(const int64_t* rowptr, const int32_t* col, const double* val, const double* x, const double* b,
                     double* r, int64_t n, cudaStream_t st) {
  k_residual<<<grid_1d(n), 256, 0, st>>>(rowptr, col, val, x, b, r, n);
}
void launch_norms(const double* r, const double* x, const double* b, int64_t n, double* out, cudaStream_t st) {
  cudaMemsetAsync(out, 0, 5 * sizeof(double), st);
  k_norms<<<grid_1d(n), 256, 0, st>>>(r, x, b, n, out);
}
void launch_residual_multi(const int64_t* rowptr, const int32_t* col, const double* val, const double* x,
                           double* xt, const double* b, double* r, int64_t n, int k, double* out, cudaStream_t st) {
  if (n <= 0 || k <= 0) return;
  k_to_rows<<<dim3((unsigned)ceil_div(n, 32), (unsigned)ceil_div(k, 32)), 256, 0, st>>>(x, xt, n, k);
  k_residual_multi<<<grid_1d(n * 32), 256, 0, st>>>(rowptr, col, val, xt, b, r, n, k);
  cudaMemsetAsync(out, 0, 8 * sizeof(double) * k, st);
  k_norms<<<dim3(grid_1d(n), k), 256, 0, st>>>(r, x, b, n, out);
}
void launch_row_abs_max(const int64_t* rowptr, const double* val, int64_t n, double* out, cudaStream_t st) {
  cudaMemsetAsync(out, 0, sizeof(double), st);
  k_row_abs_max<<<grid_1d(n), 256, 0, st>>>(rowptr, val, n, out);
}
template <typename T>
void launch_to_t(const double* in, T* out, int64_t n, cudaStream_t st) {
  k_to_t<T><<<grid_1d(n), 256, 0, st>>>(in, out, n);
}
template <typename T>
void launch_axpy_from_t(const T* d, double* x, int64_t n, cudaStream_t st) {
  k_axpy_from_t<T><<<grid_1d(n), 256, 0, st>>>(d, x, n);
}
void launch_fill_int(int32_t* p, int32_t v, int64_t n, cudaStream_t st) {
  if (n > 0) k_fill_int<<<grid_1d(n), 256, 0, st>>>(p, v, n);
}
__global__ void k_ir_init(int32_t* st_i, double* st_d, double* prev, int nrhs) {
  for (int c = threadIdx.x; c < nrhs; c += blockDim.x) prev[c] = 1e300;
  if (threadIdx.x == 0) {
    st_i[0] = 0;
    st_i[1] = 1;
    st_d[0] = st_d[1] = 0.0;
  }
}
void launch_ir_init(int32_t* st_i, double* st_d, double* prev, int nrhs, cudaStream_t st) {
  k_ir_init<<<1, 128, 0, st>>>(st_i, st_d, prev, nrhs);
}
// one thread: the per-column test in column order, as the host loop does it
__global__ void k_ir_check(const double* norms, const double* anorm, int nrhs, double tol, int maxit, double* prev,
                           int32_t* st_i, double* st_d, cudaGraphConditionalHandle cond) {
  if (threadIdx.x != 0) return;
  const int it = st_i[0];                 // 0-based index of the sweep just done
  bool all_ok = true, all_stalled = it > 2;
  double worst = 0.0, worst_ref = 0.0;
  for (int c = 0; c < nrhs; ++c) {
    const double* v = norms + 8 * c;
    const double denom = anorm[0] * v[1] + v[2];
    const double cur = denom > 0 ? v[0] / denom : v[0];
    if (cur > tol) {
      all_ok = false;
      if (cur <= 0.9 * prev[c]) all_stalled = false;
    }
    if (cur >= worst) {
      worst = cur;
      worst_ref = v[4] > 0 ? sqrt(v[3]) / sqrt(v[4]) : sqrt(v[3]);
    }
    prev[c] = cur;
  }
  st_i[0] = it + 1;
  st_d[0] = worst;
  st_d[1] = worst_ref;
  const bool more = !(all_ok || all_stalled) && it + 1 < maxit;
  st_i[1] = more ? 1 : 0;
  cudaGraphSetConditional(cond, more ? 1u : 0u);
}
void launch_ir_check(const double* norms, const double* anorm, int nrhs, double tol, int maxit, double* prev,
                     int32_t* st_i, double* st_d, cudaGraphConditionalHandle cond, cudaStream_t st) {
  k_ir_check<<<1, 32, 0, st>>>(norms, anorm, nrhs, tol, maxit, prev, st_i, st_d, cond);
}

__global__ void k_factor_begin(int32_t* info) {
  info[0] = INT_MAX;
  info[1] = 0;
  info[3] = 0;
}
void launch_factor_begin(int32_t* info, cudaStream_t st) { k_factor_begin<<<1, 1, 0, st>>>(info); }
__global__ void k_factor_report(const int32_t* info, const double* anorm, int32_t* h_info, double* h_anorm) {
  if (threadIdx.x < 4) h_info[threadIdx.x] = info[threadIdx.x];
  if (threadIdx.x == 4) *h_anorm = *anorm;
}
void launch_factor_report(const int32_t* info, const double* anorm, int32_t* h_info, double* h_anorm, cudaStream_t st) {
  k_factor_report<<<1, 32, 0, st>>>(info, anorm, h_info, h_anorm);
}
__global__ void k_solve_report(const double* norms, const int32_t* ir_i, const double* ir_d, const int32_t* expired,
                               double* h_norms, int32_t* h_ir_i, double* h_ir_d, int32_t* h_expired) {
  const int t = threadIdx.x;
  if (norms && t < 5) h_norms[t] = norms[t];
  if (ir_i && t < 2) {
    h_ir_i[t] = ir_i[t];
    h_ir_d[t] = ir_d[t];
  }
  if (expired && t == 5) *h_expired = *expired;
}
void launch_solve_report(const double* norms, const int32_t* ir_i, const double* ir_d, const int32_t* expired,
                         double* h_norms, int32_t* h_ir_i, double* h_ir_d, int32_t* h_expired, cudaStream_t st) {
  k_solve_report<<<1, 32, 0, st>>>(norms, ir_i, ir_d, expired, h_norms, h_ir_i, h_ir_d, h_expired);
}

__global__ void k_remap_int(const int32_t* map, int32_t* a, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    a[i] = map[a[i]];
}
void launch_remap_int(const int32_t* map, int32_t* a, int64_t n, cudaStream_t st) {
  if (n > 0) k_remap_int<<<grid_1d(n), 256, 0, st>>>(map, a, n);
}

#define MFD_INSTANTIATE(T)                                                                                          \
  template void launch_build_large<T>(const DevFronts&, const int32_t*, int, int, T*, T*, cudaStream_t);            \
  template void launch_assemble_large<T>(const DevFronts&, const int32_t*, int, int, const double*, T*, const T*,   \
                                         cudaStream_t);                                                            \
  template void launch_add_children<T>(const DevFronts&, const int32_t*, int, int, T*, T*, cudaStream_t);           \
  template void launch_gather_many<T>(const DevFronts&, const int32_t*, int, int, const T*, int64_t, const T*,      \
                                      double*, int, cudaStream_t);                                                 \
  template int launch_update<T>(const DevFronts&, const int32_t*, int, int, int, int, T*, T*, int, cudaStream_t,    \
                                 UpdBand, int, bool);                                                              \
  template void launch_fwd_large<T>(const DevFronts&, const int32_t*, int, int, int, const T*, const T*, T*,       \
                                    int64_t, T*, int32_t*, int, cudaStream_t, int64_t*, bool);                     \
  template void launch_bwd_large<T>(const DevFronts&, const int32_t*, int, int, int, const T*, const T*, T*,       \
                                    int64_t, T*, T*, int32_t*, int, cudaStream_t, int64_t*, bool);                 \
  template void launch_permute_in<T>(const double*, int64_t, const int32_t*, T*, int64_t, int64_t, int,            \
                                     cudaStream_t);                                                                \
  template void launch_permute_out<T>(const T*, int64_t, const int32_t*, double*, int64_t, int64_t, int,           \
                                      cudaStream_t);                                                               \
  template void launch_to_t<T>(const double*, T*, int64_t, cudaStream_t);                                          \
  template void launch_axpy_from_t<T>(const T*, double*, int64_t, cudaStream_t);

MFD_INSTANTIATE(double)
MFD_INSTANTIATE(float)

}  // namespace mfd
