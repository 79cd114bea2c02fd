// Panel step of the blocked large-front factorization (128 columns):
//   k_potrf  : one CTA per front: Cholesky of the w x w diagonal block in shared
//              memory (chol_smem.cuh); L11 to the panel and, with the 8 x 8
//              diagonal blocks inverted, in packed blocks to a scratch slot
//   k_trsm   : the rows below, X <- A L11^{-T}, by block substitution on DMMA
//              from that slot, eight rows per warp in registers
//   k_invert : L11^{-1} of every panel step of a level, for the solves; off the
//              panel chain (nothing in the factorization reads it)
// All arithmetic is FP64 whatever the storage type.
//
// What bounds a step is latency on the one CTA (few at most) that holds the
// block: POTRF 53 -> 20 us (the pivot chain at one FP64 instruction per 4.5
// cycles and warp), TRSM 15-18 -> 8 us (substitution instead of the product with
// an inverse that had to be formed first); a whole step 88 -> ~37 us with the next
// panel's update.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "chol_smem.cuh"
#include "kernels.cuh"

namespace mfd {

namespace {

// Widest block of a k_potrf class: 32 NSB columns, one row per thread of the
// first NSB warps, more warps for the trailing updates of the wider ones.
template <int NSB>
__host__ __device__ constexpr int potrf_warps() {
  return NSB == 1 ? 1 : NSB == 2 ? 4 : NSB == 3 ? 8 : 12;
}
template <int NSB>
__host__ __device__ constexpr int potrf_threads() {
  return 32 * potrf_warps<NSB>();
}
template <int NSB>
__host__ __device__ constexpr size_t potrf_smem() {
  return sizeof(double) * ((size_t)blk_count(4 * NSB) * kBlkElems + (size_t)4 * NSB * kBlkElems +
                           chol_scratch_elems(32 * NSB, true));
}

// Column-major lower w x w block (ld) -> packed blocks in shared memory, zero
// above the diagonal, identity on the padding up to 8 nb.  A warp takes four
// columns at a time, 16 loads per lane in flight.
template <typename T>
__device__ __forceinline__ void load_block(const T* P, size_t ld, int w, int nb, double* S, int warps) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n = 8 * nb;
  for (int j0 = 4 * warp; j0 < n; j0 += 4 * warps) {     // the four columns share a block column
    const int i0 = j0 & ~7;
    T v[4][4];
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int i = i0 + lane + 32 * u, j = j0 + c;
        v[c][u] = (i >= j && i < w && j < w) ? P[i + (size_t)j * ld] : T(i == j && j >= w ? 1 : 0);
      }
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int i = i0 + lane + 32 * u, j = j0 + c;
        if (i < n) S[blk_index(i >> 3, j >> 3, nb) * kBlkElems + blk_elem(i & 7, j & 7)] = (double)v[c][u];
      }
  }
}

// info_stride 0: every front reports into info[0]; 1: list slot i reports into info[i].
// fallbacks (may be null; counted for FP32 storage): 32-column groups with a small pivot.
template <typename T, int NSB>
__global__ void __launch_bounds__(potrf_threads<NSB>(), 1) k_potrf(DevFronts F, const int32_t* list, int slot0,
                                                                   int step, T* panel, double* packed, int slot_elems,
                                                                   int32_t* info, int info_stride, int32_t* fallbacks) {
  constexpr int NW = potrf_warps<NSB>(), NT = 32 * NW;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* S = reinterpret_cast<double*>(smem_raw);
  double* Dinv = S + (size_t)blk_count(4 * NSB) * kBlkElems;
  double* scratch = Dinv + 4 * NSB * kBlkElems;
  const int slot = slot0 + blockIdx.x, f = list[slot];
  const int nc = F.nc[f], nf = nc + F.nr[f];
  const int c0 = step * kFactB;
  if (c0 >= nc) return;
  const int w = min(kFactB, nc - c0), nb = (w + 7) >> 3;   // w <= 32 NSB by the launch's choice of NSB
  T* P = panel + F.panel_off[f] + c0 + (size_t)c0 * nf;
  pdl_wait();
  pdl_trigger();          // after the wait: every kernel before this one has completed
  load_block(P, nf, w, nb, S, NW);
  __syncthreads();
  int32_t* my_info = info + (size_t)info_stride * slot;
  chol_panels<NW, sizeof(T) == 4>(
      S, scratch, nb, nb,
      [&](int j) {
        if (j < w) atomicMin(my_info, F.first[f] + c0 + j + 1);
      },
      [&] {
        if (fallbacks) atomicAdd(fallbacks, 1);
      });
  invert_diagonal_blocks(S, scratch + kCholRq, Dinv, nb, nb);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double2* Q = reinterpret_cast<double2*>(packed + (size_t)slot * slot_elems);
  for (int e = tid; e < blk_count(nb) * 32; e += NT) Q[e] = reinterpret_cast<const double2*>(S)[e];
  __syncthreads();        // the diagonal blocks of the slot are rewritten below
  for (int e = tid; e < nb * 32; e += NT)
    Q[blk_index(e >> 5, e >> 5, nb) * 32 + (e & 31)] = reinterpret_cast<const double2*>(Dinv)[e];
  for (int j = warp; j < w; j += NW)
    for (int i = j + lane; i < w; i += 32)
      P[i + (size_t)j * nf] = (T)S[blk_index(i >> 3, j >> 3, nb) * kBlkElems + blk_elem(i & 7, j & 7)];
}

// 32 rows per CTA, eight per warp.  The rows go from global memory straight
// into accumulator fragments (eight lanes read eight consecutive rows of a
// column) before the wait on the diagonal block, and back from there; only the
// packed block passes through shared memory.
constexpr int kTrWarps = 4;
template <typename T>
__global__ void __launch_bounds__(32 * kTrWarps, 3) k_trsm(DevFronts F, const int32_t* list, int step, T* panel,
                                                        const double* packed, int slot_elems, T* q) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* L = reinterpret_cast<double*>(smem_raw);
  const int f = list[blockIdx.y];
  const int nc = F.nc[f], nf = nc + F.nr[f];
  const int c0 = step * kFactB;
  if (c0 >= nc) return;
  const int w = min(kFactB, nc - c0), nb = (w + 7) >> 3;
  const int rel = blockIdx.x * 8 * kTrWarps;               // first row relative to c0 + w
  if (c0 + w + rel >= nf) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, c2 = 2 * (lane & 3);
  const int row = c0 + w + rel + 8 * warp + g;
  const bool ok = row < nf;
  T* P = panel + F.panel_off[f] + row + (size_t)c0 * nf;   // column c of the row at P[c nf]
  // the rows below the diagonal block do not depend on the POTRF that precedes this kernel
  // (no event wait sits between the two launches)
  double2 acc[16];
#pragma unroll
  for (int b = 0; b < 16; ++b) {
    const int c = 8 * b + c2;
    acc[b].x = ok && c < w ? (double)P[(size_t)c * nf] : 0.0;
    acc[b].y = ok && c + 1 < w ? (double)P[(size_t)(c + 1) * nf] : 0.0;
  }
  pdl_wait();
  pdl_trigger();
  const double* Q = packed + (size_t)blockIdx.y * slot_elems;
  for (int e = threadIdx.x; e < blk_count(nb) * 32; e += 32 * kTrWarps) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(L + 2 * e);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(Q + 2 * e));
  }
  asm volatile("cp.async.commit_group;\n" ::);
  asm volatile("cp.async.wait_group 0;\n" ::);
  __syncthreads();
  trsm_rows8(acc, L, nb, 0, lane);
#pragma unroll
  for (int b = 0; b < 16; ++b) {
    const int c = 8 * b + c2;
    if (ok && c < w) P[(size_t)c * nf] = (T)acc[b].x;
    if (ok && c + 1 < w) P[(size_t)(c + 1) * nf] = (T)acc[b].y;
  }
  if constexpr (sizeof(T) == 8) {
    if (q != nullptr) {     // the same rows as packed operands of the update
      double* Qf = q + F.q_off[f];
      const int r = rel + 8 * warp + g;
#pragma unroll
      for (int b = 0; b < 16; ++b) {
        const int c = 8 * b + c2;
        Qf[packed_dp_offset(r, c)] = ok && c < w ? acc[b].x : 0.0;
        Qf[packed_dp_offset(r, c + 1)] = ok && c + 1 < w ? acc[b].y : 0.0;
      }
    }
  } else {
    if (q != nullptr) {     // the same rows as packed TF32 hi / lo operands of the tensor-core update
      float* Qf = q + F.q_off[f];
#pragma unroll
      for (int b = 0; b < 16; ++b) {
        const int c = 8 * b + c2;
        float2 hi, lo;
        const float v0 = ok && c < w ? (float)acc[b].x : 0.0f, v1 = ok && c + 1 < w ? (float)acc[b].y : 0.0f;
        uint32_t h0, h1;
        asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(h0) : "f"(v0));
        asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(h1) : "f"(v1));
        hi = make_float2(__uint_as_float(h0), __uint_as_float(h1));
        lo = make_float2(v0 - hi.x, v1 - hi.y);
        *reinterpret_cast<float2*>(Qf + packed_offset(rel + 8 * warp + g, c, 0)) = hi;
        *reinterpret_cast<float2*>(Qf + packed_offset(rel + 8 * warp + g, c, 1)) = lo;
      }
    }
  }
}

// X = L11^{-1} of panel step blockIdx.y of front list[blockIdx.x], from the
// panel: eight warps, warp v the rows of the identity in block rows v and
// 15 - v (as many blocks in any pair); row k of I L^{-T} is column k of X.
// linv was zeroed once: only the lower w x w part is written.
template <typename T>
__global__ void __launch_bounds__(256) k_invert(DevFronts F, const int32_t* list, const T* panel, T* linv) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* S = reinterpret_cast<double*>(smem_raw);
  const int f = list[blockIdx.x], step = blockIdx.y;
  const int nc = F.nc[f], nf = nc + F.nr[f];
  const int c0 = step * kFactB;
  if (c0 >= nc) return;
  const int w = min(kFactB, nc - c0), nb = (w + 7) >> 3;
  load_block(panel + F.panel_off[f] + c0 + (size_t)c0 * nf, nf, w, nb, S, 8);
  __syncthreads();
  const int tid = threadIdx.x;
  double z[8];
  if (tid < 8 * nb) {                                      // diagonal block tid / 8, column tid % 8 of its inverse
    const double* D = S + blk_index(tid >> 3, tid >> 3, nb) * kBlkElems;
#pragma unroll
    for (int k = 0; k < 8; ++k) z[k] = k == (tid & 7) ? 1.0 : 0.0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      z[k] /= D[blk_elem(k, k)];
#pragma unroll
      for (int i = k + 1; i < 8; ++i) z[i] = fma(-D[blk_elem(i, k)], z[k], z[i]);
    }
  }
  __syncthreads();
  if (tid < 8 * nb) {
    double* D = S + blk_index(tid >> 3, tid >> 3, nb) * kBlkElems;
#pragma unroll
    for (int k = 0; k < 8; ++k) D[blk_elem(k, tid & 7)] = z[k];
  }
  __syncthreads();
  T* X = linv + F.d_off[f] + (size_t)step * kFactB * kFactB;
  const int lane = tid & 31, warp = tid >> 5, g = lane >> 2, c2 = 2 * (lane & 3);
#pragma unroll 1
  for (int hh = 0; hh < 2; ++hh) {
    const int v = hh ? 15 - warp : warp;
    if (v >= nb) continue;
    double2 acc[16];
#pragma unroll
    for (int b = 0; b < 16; ++b)
      acc[b] = make_double2(b == v && c2 == g ? 1.0 : 0.0, b == v && c2 + 1 == g ? 1.0 : 0.0);
    trsm_rows8(acc, S, nb, v, lane);
    const int k = 8 * v + g;
#pragma unroll
    for (int b = 0; b < 16; ++b) {
      const int n = 8 * b + c2;
      if (b >= v && k < w && n < w && n >= k) X[n + (size_t)k * kFactB] = (T)acc[b].x;
      if (b >= v && k < w && n + 1 < w && n + 1 >= k) X[n + 1 + (size_t)k * kFactB] = (T)acc[b].y;
    }
  }
}

constexpr size_t kPanelSmem = (size_t)blk_count(16) * kBlkElems * sizeof(double);   // 69,632: three CTAs per SM

template <typename KernelT>
cudaError_t max_smem(KernelT k, size_t bytes) {
  return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

}  // namespace

cudaError_t prepare_panel() {
  cudaError_t e = cudaSuccess;
  auto chk = [&](cudaError_t r) { if (r != cudaSuccess && e == cudaSuccess) e = r; };
  chk(max_smem(k_potrf<double, 4>, potrf_smem<4>())); chk(max_smem(k_potrf<float, 4>, potrf_smem<4>()));
  chk(max_smem(k_potrf<double, 3>, potrf_smem<3>())); chk(max_smem(k_potrf<float, 3>, potrf_smem<3>()));
  chk(max_smem(k_potrf<double, 2>, potrf_smem<2>())); chk(max_smem(k_potrf<float, 2>, potrf_smem<2>()));
  chk(max_smem(k_potrf<double, 1>, potrf_smem<1>())); chk(max_smem(k_potrf<float, 1>, potrf_smem<1>()));
  chk(max_smem(k_trsm<double>, kPanelSmem)); chk(max_smem(k_trsm<float>, kPanelSmem));
  chk(max_smem(k_invert<double>, kPanelSmem)); chk(max_smem(k_invert<float>, kPanelSmem));
  return e;
}

template <typename T>
void launch_potrf(const DevFronts& F, const int32_t* list, int count, int step, T* panel, double* packed, int slot_elems,
                  int32_t* info, cudaStream_t st, bool pdl, int info_stride, int32_t* fallbacks, const int32_t* cls) {
  if (count <= 0) return;
  int off = 0;
  auto go = [&](auto kern, int nt, size_t smem, int cnt) {
    if (cnt > 0)
      launch_k(kern, dim3(cnt), dim3(nt), smem, st, pdl, F, list, off, step, panel, packed, slot_elems, info,
               info_stride, fallbacks);
    off += cnt;
  };
  if (cls == nullptr) {                   // one launch, any block width
    go(k_potrf<T, 4>, potrf_threads<4>(), potrf_smem<4>(), count);
    return;
  }
  // cls[k]: fronts of the list (in order, block widths non-increasing) whose block needs 4 - k groups of 32 columns
  go(k_potrf<T, 4>, potrf_threads<4>(), potrf_smem<4>(), cls[0]);
  go(k_potrf<T, 3>, potrf_threads<3>(), potrf_smem<3>(), cls[1]);
  go(k_potrf<T, 2>, potrf_threads<2>(), potrf_smem<2>(), cls[2]);
  go(k_potrf<T, 1>, potrf_threads<1>(), potrf_smem<1>(), cls[3]);
}

template <typename T>
void launch_trsm(const DevFronts& F, const int32_t* list, int count, int step, int row_blocks, int max_w, T* panel,
                 const double* packed, int slot_elems, cudaStream_t st, bool pdl, T* q) {
  if (count <= 0 || row_blocks <= 0) return;
  // row_blocks counts 64-row blocks; shared memory for the widest block of the launch
  const size_t smem = (size_t)blk_count((max_w + 7) / 8) * kBlkElems * sizeof(double);
  launch_k(k_trsm<T>, dim3(row_blocks * (kTrRowsH / (8 * kTrWarps)), count), dim3(32 * kTrWarps), smem, st, pdl, F, list,
           step, panel, packed, slot_elems, q);
}

template <typename T>
void launch_invert(const DevFronts& F, const int32_t* list, int count, int steps, int max_w, const T* panel, T* linv,
                   cudaStream_t st) {
  if (count <= 0 || steps <= 0) return;
  const size_t smem = (size_t)blk_count((max_w + 7) / 8) * kBlkElems * sizeof(double);
  k_invert<T><<<dim3(count, steps), 256, smem, st>>>(F, list, panel, linv);
}

#define MFD_INSTANTIATE_PANEL(T)                                                                                   \
  template void launch_potrf<T>(const DevFronts&, const int32_t*, int, int, T*, double*, int, int32_t*, cudaStream_t,  \
                                bool, int, int32_t*, const int32_t*);                                              \
  template void launch_trsm<T>(const DevFronts&, const int32_t*, int, int, int, int, T*, const double*, int,           \
                               cudaStream_t, bool, T*);                                                        \
  template void launch_invert<T>(const DevFronts&, const int32_t*, int, int, int, const T*, T*, cudaStream_t);

MFD_INSTANTIATE_PANEL(double)
MFD_INSTANTIATE_PANEL(float)

}  // namespace mfd
