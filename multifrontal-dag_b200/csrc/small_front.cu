// Fused small fronts (nf <= 160): zero, assemble A, extend-add the children in
// order, partial Cholesky of the nc supernode columns and the Schur complement,
// all on chip; the factor panel and the update matrix are written once.
//
//   k_small_warp  : nf <= 32, one warp per front, one row per lane in registers
//   k_small_block : nf <= 160, one CTA per front on 8 x 8 blocks (chol_smem.cuh)
//
// Both start from the front's record and its children's (FrontRec, ChildRec).
// What bound them was latency: a chain of six dependent loads before the first
// value of a child arrives, and in the one-CTA kernel trailing tiles one after
// another (7 us per eight columns); a front of 102 rows and columns took 94 us.
// With the records, the block layout and two panels per update pass the whole
// steps take: 100 x 100 Laplacian 975 -> 554 us, batch of 1000 2D systems 12.35
// -> 8.37 ms (1.5 TFLOP/s, 0.9 TB/s).  160 rows is the line to the blocked path:
// up to there a front's blocks (105 KB) leave room for a second CTA on the SM, and
// the blocked path's two panel steps cost ~37 us each whatever their width.  Line
// at 128 / 160 rows: batch of 1000 8.90 / 8.39 ms, batch solve 802 / 774 us, 100 x
// 100 Laplacian 598 / 573 us, 21^3 elasticity 5.90 / 5.88 ms, 37 x 41 x 43 solve
// 798 / 810 us.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "chol_smem.cuh"
#include "kernels.cuh"

namespace mfd {

namespace {

template <typename T>
__device__ __forceinline__ T rsqrt_of(T x);
template <>
__device__ __forceinline__ double rsqrt_of<double>(double x) { return rsqrt(x); }
template <>
__device__ __forceinline__ float rsqrt_of<float>(float x) { return rsqrtf(x); }

// ---- nf <= NF <= 32: one warp per front ------------------------------------------
// The front is assembled in a per-warp shared buffer (A entries four per lane
// in flight, then the children, lanes over rows, eight columns in flight, the
// next child's first columns and its local index loaded ahead), loaded one row
// per lane into registers and partially factored there (nc pivots: shuffle for
// the pivot, rsqrt, rank-1 update with the column broadcast through a
// double-buffered shared vector); panel and update matrix are written one
// column per step, lanes over rows.  No CTA-wide barrier.  NF in {16, 24, 32}
// sets registers, shared memory and the length of the rank-1 updates.
constexpr int kWarps = 4;

template <typename T, int NF>
__global__ void __launch_bounds__(kWarps * 32, NF <= 24 ? 8 : 6) k_small_warp(DevFronts F, const FrontRec* __restrict__ recs, int count,
                                                            const double* __restrict__ a, T* __restrict__ panel,
                                                            T* __restrict__ upool, int32_t* info) {
  constexpr int LD = NF + 1, CU = 4;
  __shared__ T sbuf[kWarps][NF * LD];
  __shared__ T cbuf[kWarps][2][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int slot = blockIdx.x * kWarps + warp;
  if (slot >= count) return;
  const FrontRec rec = recs[slot];
  const int nc = rec.nc, nr = rec.nr, nf = nc + nr;
  T* S = sbuf[warp];
  const int nch = rec.child_end - rec.child_beg;
  // children's records one per lane (broadcast by shuffles), in flight with A's entries
  int cnr = 0, clo = 0;
  long long cuo = 0;
  if (lane < nch) {
    const ChildRec c = F.crec[rec.child_beg + lane];
    cnr = c.nr; clo = c.lrow_off; cuo = c.u_off;
  }
  for (int e = lane; e < NF * LD; e += 32) S[e] = T(0);
  __syncwarp();
  for (int k0 = rec.a_beg + lane; k0 < rec.a_end; k0 += 4 * 32) {
    int pos[4], src[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int k = k0 + 32 * u;
      pos[u] = k < rec.a_end ? F.a_pos[k] : -1;
      src[u] = k < rec.a_end ? F.a_src[k] : 0;
    }
    double v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = pos[u] >= 0 ? a[src[u]] : 0.0;
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (pos[u] >= 0) {
        const int c = pos[u] / nf;
        S[pos[u] - c * nf + c * LD] = T(v[u]);
      }
  }
  __syncwarp();
  if (nch > 0) {
    int nrc = __shfl_sync(0xffffffffu, cnr, 0), li;
    const T* U = upool + __shfl_sync(0xffffffffu, cuo, 0);
    T u[CU];
    auto fetch = [&](int m, const T* Um, int lo, int& l, T (&x)[CU]) {      // local row and the first CU columns
      l = lane < m ? F.local[lo + lane] - 1 : 0;
#pragma unroll
      for (int c = 0; c < CU; ++c) x[c] = c < m && lane >= c && lane < m ? Um[(size_t)c * m + lane] : T(0);
    };
    fetch(nrc, U, __shfl_sync(0xffffffffu, clo, 0), li, u);
    for (int t = 0; t < nch; ++t) {
      int nrn = 0, lin = 0;
      const T* Un = upool;
      T un[CU];
      if (t + 1 < nch) {
        if (((t + 1) & 31) == 0) {                       // the next 32 children's records
          cnr = 0; clo = 0; cuo = 0;
          if (t + 1 + lane < nch) {
            const ChildRec c = F.crec[rec.child_beg + t + 1 + lane];
            cnr = c.nr; clo = c.lrow_off; cuo = c.u_off;
          }
        }
        const int q = (t + 1) & 31;
        nrn = __shfl_sync(0xffffffffu, cnr, q);
        Un = upool + __shfl_sync(0xffffffffu, cuo, q);
        fetch(nrn, Un, __shfl_sync(0xffffffffu, clo, q), lin, un);
      }
      for (int j0 = 0; j0 < nrc; j0 += CU) {
        if (j0 > 0)
#pragma unroll
          for (int c = 0; c < CU; ++c)
            u[c] = j0 + c < nrc && lane >= j0 + c && lane < nrc ? U[(size_t)(j0 + c) * nrc + lane] : T(0);
#pragma unroll
        for (int c = 0; c < CU; ++c) {
          const int lj = __shfl_sync(0xffffffffu, li, (j0 + c) & 31);
          if (j0 + c < nrc && lane >= j0 + c && lane < nrc) S[lj * LD + li] += u[c];
        }
      }
      __syncwarp();
      nrc = nrn;
      li = lin;
      U = Un;
#pragma unroll
      for (int c = 0; c < CU; ++c) u[c] = un[c];
    }
  }
  T row[NF];
  const int lr = min(lane, NF - 1);
#pragma unroll
  for (int j = 0; j < NF; ++j) row[j] = S[lr + j * LD];
  int bad = 0;
#pragma unroll
  for (int k = 0; k < NF; ++k) {
    if (k >= nc) break;
    T d = __shfl_sync(0xffffffffu, row[k], k);
    if (!(d > T(0))) {                    // uniform across the warp
      if (!bad) bad = k + 1;
      d = T(1);
    }
    const T y = rsqrt_of<T>(d);
    const T l = row[k] * y;
    T* cb = cbuf[warp][k & 1];
    cb[lane] = l;
    __syncwarp();
    row[k] = lane == k ? d * y : l;
#pragma unroll
    for (int j = k + 1; j < NF; ++j) row[j] -= l * cb[j];
  }
  if (bad && lane == 0) atomicMin(info, rec.first + bad);
  T* P = panel + rec.panel_off;
  T* Uf = upool + rec.u_off;
#pragma unroll
  for (int j = 0; j < NF; ++j) {
    if (j >= nf) break;
    if (lane >= j && lane < nf) {
      if (j < nc) P[lane + (size_t)j * nf] = row[j];
      else Uf[(lane - nc) + (size_t)(j - nc) * nr] = row[j];
    }
  }
}

// ---- nf <= 160: one CTA per front ------------------------------------------------
// The nc pivot columns are padded to a multiple of eight with an identity, so
// that the pivot and the update part split at a block boundary (dummy columns
// couple to nothing).  Shared memory in FP64 for either storage type.
constexpr int kChildBatch = 4;    // children whose local indices are staged together
constexpr int kStageRows = kSmallFrontMax;

template <int NF>
__host__ __device__ constexpr int block_rows() { return (NF + 7 + 7) / 8; }      // block rows with the padding
template <int NF>
__host__ __device__ constexpr int block_warps() { return NF <= 64 ? 4 : NF <= 96 ? 6 : 8; }
template <int NF>
__host__ __device__ constexpr int block_threads() { return 32 * block_warps<NF>(); }
// shared memory for fronts of at most nf rows
template <int NF>
size_t block_smem(int nf) {
  return sizeof(double) * ((size_t)blk_count((nf + 14) / 8) * kBlkElems + chol_scratch_elems(8 * block_rows<NF>(), false)) +
         sizeof(uint8_t) * kChildBatch * kStageRows;
}

// S(local) += U (nrc x nrc, lower): warps over columns, lanes over rows, CU
// columns x RI row passes of loads in flight.
template <int RI, int CU, typename T>
__device__ __forceinline__ void extend_add(double* S, int nbt, const T* __restrict__ U, const uint8_t* loc, int nrc,
                                           int lane, int warp, int nw) {
  for (int j0 = warp; j0 < nrc; j0 += CU * nw) {
    T u[CU][RI];
#pragma unroll
    for (int c = 0; c < CU; ++c) {
      const int j = j0 + c * nw;
#pragma unroll
      for (int v = 0; v < RI; ++v) {
        const int i = j + lane + 32 * v;
        u[c][v] = j < nrc && i < nrc ? U[(size_t)j * nrc + i] : T(0);
      }
    }
#pragma unroll
    for (int c = 0; c < CU; ++c) {
      const int j = j0 + c * nw;
      if (j < nrc) {
        const int lj = loc[j];
#pragma unroll
        for (int v = 0; v < RI; ++v) {
          const int i = j + lane + 32 * v;
          if (i < nrc) S[blk_addr(loc[i], lj, nbt)] += (double)u[c][v];
        }
      }
    }
  }
}

template <typename T, int NF>
__global__ void __launch_bounds__(block_threads<NF>(), NF <= 64 ? 6 : NF <= 96 ? 3 : NF <= 128 ? 2 : 1)
    k_small_block(DevFronts F, const FrontRec* __restrict__ recs, const double* __restrict__ a, T* __restrict__ panel,
                  T* __restrict__ upool, int32_t* info) {
  constexpr int NW = block_warps<NF>(), NT = 32 * NW;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const FrontRec rec = recs[blockIdx.x];
  const int nc = rec.nc, nr = rec.nr, nf = nc + nr;
  const int nbp = (nc + 7) >> 3, pad = 8 * nbp - nc, nbt = (nf + pad + 7) >> 3;
  double* S = reinterpret_cast<double*>(smem_raw);
  double* scratch = S + blk_count(nbt) * kBlkElems;
  uint8_t* sloc = reinterpret_cast<uint8_t*>(scratch + chol_scratch_elems(8 * block_rows<NF>(), false));   // kChildBatch x kStageRows
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nch = rec.child_end - rec.child_beg;
  // A's first entries and the first children's local indices are in flight while the front is zeroed
  int pos = -1;
  double av = 0.0;
  if (rec.a_beg + tid < rec.a_end) {
    pos = F.a_pos[rec.a_beg + tid];
    av = a[F.a_src[rec.a_beg + tid]];
  }
  auto stage = [&](int t0) {                             // children t0 .. t0 + kChildBatch - 1, a warp each
    for (int t = t0 + warp; t < min(nch, t0 + kChildBatch); t += NW) {
      const ChildRec c = F.crec[rec.child_beg + t];
      for (int i = lane; i < c.nr; i += 32) {
        const int l = F.local[c.lrow_off + i] - 1;
        sloc[(t - t0) * kStageRows + i] = (uint8_t)(l < nc ? l : l + pad);
      }
    }
  };
  stage(0);
  for (int e = tid; e < blk_count(nbt) * (kBlkElems / 2); e += NT) reinterpret_cast<double2*>(S)[e] = make_double2(0.0, 0.0);
  __syncthreads();
  if (tid < pad) S[blk_addr(nc + tid, nc + tid, nbt)] = 1.0;
  auto put = [&](int ps, double v) {                     // entry of A: row >= column, column < nc
    const int c = ps / nf, r = ps - c * nf;
    S[blk_addr(r < nc ? r : r + pad, c, nbt)] = v;
  };
  if (pos >= 0) put(pos, av);
  for (int k = rec.a_beg + tid + NT; k < rec.a_end; k += NT) put(F.a_pos[k], a[F.a_src[k]]);
  __syncthreads();
  for (int t0 = 0; t0 < nch; t0 += kChildBatch) {
    if (t0 > 0) {
      stage(t0);
      __syncthreads();
    }
    for (int t = t0; t < min(nch, t0 + kChildBatch); ++t) {
      const ChildRec c = F.crec[rec.child_beg + t];
      const T* U = upool + c.u_off;
      const uint8_t* loc = sloc + (t - t0) * kStageRows;
      switch ((c.nr + 31) >> 5) {                        // row passes a column needs
        case 0: break;
        case 1: extend_add<1, 8>(S, nbt, U, loc, c.nr, lane, warp, NW); break;
        case 2: extend_add<2, 8>(S, nbt, U, loc, c.nr, lane, warp, NW); break;
        case 3: extend_add<3, 5>(S, nbt, U, loc, c.nr, lane, warp, NW); break;
        case 4: extend_add<4, 4>(S, nbt, U, loc, c.nr, lane, warp, NW); break;
        default: extend_add<5, 3>(S, nbt, U, loc, c.nr, lane, warp, NW); break;
      }
      __syncthreads();
    }
  }
  chol_panels<NW, false>(
      S, scratch, nbp, nbt, [&](int j) { if (j < nc) atomicMin(info, rec.first + j + 1); }, [] {});
  T* P = panel + rec.panel_off;
  for (int j = warp; j < nc; j += NW)
    for (int i = j + lane; i < nf; i += 32) P[i + (size_t)j * nf] = (T)S[blk_addr(i < nc ? i : i + pad, j, nbt)];
  T* U = upool + rec.u_off;
  const int n0 = 8 * nbp;
  for (int j = warp; j < nr; j += NW)
    for (int i = j + lane; i < nr; i += 32) U[i + (size_t)j * nr] = (T)S[blk_addr(n0 + i, n0 + j, nbt)];
}

}  // namespace

cudaError_t prepare_small_fronts() {
  cudaError_t e = cudaSuccess;
  auto chk = [&](auto k, size_t bytes) {
    cudaError_t r = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (r != cudaSuccess && e == cudaSuccess) e = r;
  };
  chk(k_small_block<double, 64>, block_smem<64>(64)); chk(k_small_block<float, 64>, block_smem<64>(64));
  chk(k_small_block<double, 96>, block_smem<96>(96)); chk(k_small_block<float, 96>, block_smem<96>(96));
  chk(k_small_block<double, 128>, block_smem<128>(128)); chk(k_small_block<float, 128>, block_smem<128>(128));
  chk(k_small_block<double, 160>, block_smem<160>(160)); chk(k_small_block<float, 160>, block_smem<160>(160));
  return e;
}

template <typename T>
void launch_small_fronts(const DevFronts& F, const FrontRec* rec, int count, int nf_max, const double* a, T* panel,
                         T* upool, int32_t* info, cudaStream_t st) {
  if (count <= 0) return;
  const int wgrid = (count + kWarps - 1) / kWarps;
  if (nf_max <= 16) k_small_warp<T, 16><<<wgrid, 32 * kWarps, 0, st>>>(F, rec, count, a, panel, upool, info);
  else if (nf_max <= 24) k_small_warp<T, 24><<<wgrid, 32 * kWarps, 0, st>>>(F, rec, count, a, panel, upool, info);
  else if (nf_max <= 32) k_small_warp<T, 32><<<wgrid, 32 * kWarps, 0, st>>>(F, rec, count, a, panel, upool, info);
  else if (nf_max <= 64)
    k_small_block<T, 64><<<count, block_threads<64>(), block_smem<64>(nf_max), st>>>(F, rec, a, panel, upool, info);
  else if (nf_max <= 96)
    k_small_block<T, 96><<<count, block_threads<96>(), block_smem<96>(nf_max), st>>>(F, rec, a, panel, upool, info);
  else if (nf_max <= 128)
    k_small_block<T, 128><<<count, block_threads<128>(), block_smem<128>(nf_max), st>>>(F, rec, a, panel, upool, info);
  else
    k_small_block<T, 160><<<count, block_threads<160>(), block_smem<160>(nf_max), st>>>(F, rec, a, panel, upool, info);
}

#define MFD_INSTANTIATE_SMALL(T)                                                                                \
  template void launch_small_fronts<T>(const DevFronts&, const FrontRec*, int, int, const double*, T*, T*,      \
                                       int32_t*, cudaStream_t);
MFD_INSTANTIATE_SMALL(double)
MFD_INSTANTIATE_SMALL(float)

}  // namespace mfd
