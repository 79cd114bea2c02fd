// FP64 trailing update of large fronts from packed operands.
//
// C -= P_i P_j^T over the step's K range in 128 x 64 pieces of the lower tiles
// (the tiles, bands and K ranges of k_update_dmma2, and its arithmetic: the same
// mma.m16n8k16.f64 over the same groups of 16 k in the same order, so the results
// are the same bits).  The TRSM of a panel step also writes its rows packed: per
// 128-row block eight chunks of 16 columns, a chunk being 128 rows of 16 doubles,
//   column k of a row at position 4 (k % 4) + k / 4  -- the four values that lane
//   q = k % 4 of a fragment needs are 32 contiguous bytes --
//   with the row's eight 16-byte pairs XORed by (row & 1), so that the two rows
//   a quarter-warp reads at once use different banks.
// A chunk of an operand is then one bulk copy (cp.async.bulk, issued by one
// thread, completion on an mbarrier) and a fragment two 16-byte loads.
//
// What bounds it: the FP64 tensor pipe once the pieces fill the chip.  Staging
// the operands from the panel itself takes 12 8- or 16-byte cp.async per thread
// and 32 columns with their addresses, and 8-byte fragment loads: 24.6 TFLOP/s on
// a 43-tile trailing matrix with K = 256, of 36.9 of the pipe.  With packed
// operands the 64^3 Laplacian's whole step goes from 33.0 to 29.2 ms, 30^3
// elasticity with 64 right-hand sides from 15.7 to 14.6 ms; the pipe is active in
// 60-63 % of a bulk launch's cycles (50 before).  One barrier per chunk for the
// whole CTA: refilling a stage on a barrier of its own, warp by warp, was no faster
// (29.5 ms, more registers spilled).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "kernels.cuh"

namespace mfd {

namespace {

constexpr int kThreads = 256, kN = 64, kKc = 16, kStages = 4;
constexpr uint32_t kABytes = kFactB * kKc * 8, kBBytes = kN * kKc * 8, kStageBytes = kABytes + kBBytes;   // 16 + 8 KB
constexpr size_t kSmem = kStages * (size_t)kStageBytes;       // 96 KB: two CTAs per SM
constexpr long long kWait = 1ll << 31;                        // cycles (~1.1 s)
constexpr long long kProbeWait = 1ll << 21;                   // the test request's (~1 ms)
constexpr int kChunks = kFactB / kKc;                         // of one step's block
constexpr int kMaxGroup = kPackedDefer;
static_assert(kMaxGroup == 2, "q and qprev");

__device__ __forceinline__ void dmma16(double (&d)[4], const double (&a)[8], const double (&b)[4]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7,%8,%9,%10,%11}, "
      "{%12,%13,%14,%15}, {%0,%1,%2,%3};\n"
      : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(a[4]), "d"(a[5]), "d"(a[6]), "d"(a[7]), "d"(b[0]), "d"(b[1]),
        "d"(b[2]), "d"(b[3]));
}
// completion of the barrier's phase `parity`, bounded by the cycles at `limit`
__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity, const volatile long long* limit) {
  const long long t0 = clock64();
  while (true) {
    uint32_t done;
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t"
        "}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
    if (clock64() - t0 > *limit) return false;
  }
}
__device__ __forceinline__ void bulk_copy(uint32_t dst, const double* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

// q, qprev: the packed rows of the step and of the one before (read where its group has two);
// err[0] is raised if a wait expires; err[1] != 0 (a test of that path): the first chunk's barrier
// expects one arrival more than it gets, and the limit is short.
__global__ void __launch_bounds__(kThreads, 2) k_update_dp(DevFronts F, const int32_t* list, int step, const double* q,
                                                           const double* qprev, double* panel, double* upool,
                                                           int32_t* err, int blo, int bhi, int defer) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ __align__(8) unsigned long long full[kStages];
  __shared__ long long limit;
  __shared__ const double* src[2][kMaxGroup];            // thread 0's: operand (A, B) rows in each step of the group
  const bool probe = threadIdx.x == 0 && err[1] != 0;    // in flight with the front's sizes
  const int f = list[blockIdx.y];
  const int nc = F.nc[f], nr = F.nr[f], nf = nc + nr;
  const int c0 = step * kFactB;
  if (c0 >= nc) return;
  const int w = min(kFactB, nc - c0), base = c0 + w, nrem = nf - base;
  if (nrem <= 0) return;
  const int T = (nrem + kUpdTile - 1) / kUpdTile, hf = blockIdx.x & 1;
  int ti, tj, kbeg, kend;
  if (!select_tile(T, kUpdTile, blo, bhi, blockIdx.x >> 1, ti, tj)) return;
  if (!update_k_range(nc, step, defer, tj, kUpdTile, kbeg, kend)) return;
  const int i0 = base + ti * kUpdTile, j0 = base + tj * kUpdTile + hf * kN;
  if (j0 >= nf) return;
  const int g0 = kbeg / kFactB, nchunk = (kend - kbeg + kKc - 1) / kKc;
  const bool diag = ti == tj;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t sb = (uint32_t)__cvta_generic_to_shared(smem_raw), fb = (uint32_t)__cvta_generic_to_shared(full);
  if (tid == 0) {
    limit = probe ? kProbeWait : kWait;
    for (int s = 0; s < kStages; ++s)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(fb + 8 * s), "r"(probe && s == 0 ? 2 : 1));
    // a 128-row block relative to `base` lies (step - s) blocks further down in the rows of step s
    // (every step of a group but its last is 128 wide)
    for (int s = g0; s <= step; ++s) {
      const double* b = (s == step ? q : qprev) + F.q_off[f] + (int64_t)(step - s) * (kFactB * kFactB);
      src[0][s - g0] = b + (int64_t)ti * (kFactB * kFactB);
      src[1][s - g0] = b + (int64_t)tj * (kFactB * kFactB) + hf * kN * kKc;
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  pdl_wait();
  pdl_trigger();
  __syncthreads();
  auto issue = [&](int c) {                              // by thread 0
    const int s = c % kStages;
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(fb + 8 * s),
                 "r"(diag ? kABytes : kStageBytes)
                 : "memory");
    bulk_copy(sb + s * kStageBytes, src[0][c / kChunks] + (c % kChunks) * (kFactB * kKc), kABytes, fb + 8 * s);
    if (!diag)
      bulk_copy(sb + s * kStageBytes + kABytes, src[1][c / kChunks] + (c % kChunks) * (kFactB * kKc), kBBytes, fb + 8 * s);
  };
  if (tid == 0)
    for (int c = 0; c < min(kStages, nchunk); ++c) issue(c);

  const int wm = warp >> 1, wn = warp & 1, g = lane >> 2, qq = lane & 3;
  const int rbase = i0 + wm * 32 + g, cbase = j0 + wn * 32 + 2 * qq;
  const bool idle = i0 + wm * 32 + 31 < j0 + wn * 32;    // rows all above the diagonal
  // every entry of C this thread holds, op(entry of acc, where it is in memory); its addresses are
  // formed here twice (kept live through the K loop they would spill)
  double acc[2][4][4];
  auto for_c = [&](auto op) {
    const int nc = F.nc[f], nr = F.nr[f], nf = nc + nr;
    double* P = panel + F.panel_off[f];
    double* U = upool + F.u_off[f];
    const bool whole = i0 + kUpdTile <= nf && j0 + kN <= nf && i0 >= j0 + kN && (j0 + kN <= nc || j0 >= nc);
    const int ldc = j0 < nc ? nf : nr;
    double* Cb = j0 < nc ? P + (size_t)j0 * nf : U + (size_t)(j0 - nc) * nr - nc;   // C(gi, gj) = Cb[gi + (gj - j0) ldc]
#pragma unroll
    for (int mi = 0; mi < 2; ++mi)
#pragma unroll
      for (int ni = 0; ni < 4; ++ni)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int gi = rbase + mi * 16 + 8 * (e >> 1), gj = cbase + ni * 8 + (e & 1);
          if (whole) op(acc[mi][ni][e], Cb + gi + (size_t)(gj - j0) * ldc);
          else if (gi < nf && gj < nf && gi >= gj)
            op(acc[mi][ni][e], gj < nc ? P + gi + (size_t)gj * nf : U + (gi - nc) + (size_t)(gj - nc) * nr);
        }
  };
#pragma unroll
  for (int mi = 0; mi < 2; ++mi)
#pragma unroll
    for (int ni = 0; ni < 4; ++ni)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[mi][ni][e] = 0.0;
  for_c([](double& a, const double* at) { a = *at; });
  // this lane's 32 bytes of a row (two pairs, swapped in odd rows) and its rows in the operands
  const int p0 = 4 * qq + 2 * (g & 1), p1 = p0 ^ 2;
  bool ok = true;
  int c = 0;
  for (; c < nchunk; ++c) {
    const int s = c % kStages;
    ok = bar_wait(fb + 8 * s, (c / kStages) & 1, &limit);
    if (!idle && ok) {
      const double* As = reinterpret_cast<const double*>(smem_raw + s * kStageBytes);
      const double* Bs = diag ? As + hf * kN * kKc : As + kABytes / 8;
      double av[2][8];
#pragma unroll
      for (int mi = 0; mi < 2; ++mi)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const double* r = As + (wm * 32 + mi * 16 + 8 * h + g) * kKc;
          const double2 lo = *reinterpret_cast<const double2*>(r + p0), hi = *reinterpret_cast<const double2*>(r + p1);
          av[mi][h] = -lo.x;
          av[mi][2 + h] = -lo.y;
          av[mi][4 + h] = -hi.x;
          av[mi][6 + h] = -hi.y;
        }
#pragma unroll
      for (int ni = 0; ni < 4; ++ni) {
        const double* r = Bs + (wn * 32 + ni * 8 + g) * kKc;
        const double2 lo = *reinterpret_cast<const double2*>(r + p0), hi = *reinterpret_cast<const double2*>(r + p1);
        const double bv[4] = {lo.x, lo.y, hi.x, hi.y};
#pragma unroll
        for (int mi = 0; mi < 2; ++mi) dmma16(acc[mi][ni], av[mi], bv);
      }
    }
    if (!__syncthreads_and(ok)) break;                   // everyone is done with the stage
    if (tid == 0 && c + kStages < nchunk) issue(c + kStages);
  }
  if (c < nchunk) {                                      // a wait expired: leave C alone, let the copies land
    if (tid == 0) {
      atomicExch(err, 1);
      if (err[1] != 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(fb) : "memory");   // the arrival held back
      for (int d = c; d < min(nchunk, c + kStages); ++d) bar_wait(fb + 8 * (d % kStages), (d / kStages) & 1, &limit);
    }
    return;
  }
  for_c([](const double& a, double* at) { *at = a; });
}

}  // namespace

cudaError_t prepare_update_dp() {
  return cudaFuncSetAttribute(k_update_dp, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
}

int launch_update_dp(const DevFronts& F, const int32_t* list, int count, int step, int T128, const double* q,
                     const double* qprev, double* panel, double* upool, int32_t* err, cudaStream_t st, UpdBand band,
                     int defer, bool pdl) {
  const int g = update_grid(T128, kUpdTile, band);
  if (count <= 0 || g <= 0) return 0;
  launch_k(k_update_dp, dim3(2 * g, count), dim3(kThreads), kSmem, st, pdl, F, list, step, q, qprev, panel, upool, err,
           band.blo, band.bhi, defer);
  return 1;
}

}  // namespace mfd
