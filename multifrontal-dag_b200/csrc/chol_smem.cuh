// Partial Cholesky of a dense symmetric matrix held in shared memory, and the
// block layout its kernels share.
//
// Layout: the lower triangle in 8 x 8 blocks of doubles (512 bytes), packed by
// block columns: block (bi, bj), bi >= bj, of an nb x nb block matrix is number
// bj nb - bj (bj - 1) / 2 + bi - bj.  Inside a block, row r holds its four
// 16-byte column pairs with pair c stored at position c ^ ((r >> 1) & 3):
//   - eight lanes reading pair c of the eight rows hit all 32 banks once,
//   - a warp reading pair q of row g (g = lane / 4, q = lane % 4) reads the
//     block's 512 bytes, each once.
// The second pattern is at the same time the accumulator layout of
// mma.m8n8k4.f64 and, with the contraction index taken in the order 0 2 4 6,
// 1 3 5 7, the fragment of both of its operands (A row g, B column g): a
// fragment of any role is one 16-byte load, and an accumulator can be the A
// operand of the next multiplication without a shuffle.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace mfd {

constexpr int kBlkElems = 64;

__device__ __forceinline__ int blk_index(int bi, int bj, int nb) { return bj * nb - bj * (bj - 1) / 2 + bi - bj; }
__device__ __forceinline__ int blk_elem(int r, int c) { return r * 8 + ((((c >> 1) ^ (r >> 1)) & 3) << 1) + (c & 1); }
// entry (i, j), i >= j (or both in one diagonal block), of an nb x nb block matrix
__device__ __forceinline__ int blk_addr(int i, int j, int nb) {
  const int bj = j >> 3;
  return kBlkElems * (bj * nb - bj * (bj + 1) / 2) + 8 * i + ((((j >> 1) ^ (i >> 1)) & 3) << 1) + (j & 1);
}
// where lane (g, q) finds its 16 bytes of a block
__device__ __forceinline__ int blk_frag(int lane) { return blk_elem(lane >> 2, 2 * (lane & 3)); }
__host__ __device__ constexpr int blk_count(int nb) { return nb * (nb + 1) / 2; }

__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}
// c += a b^T over 8 contraction indices, all three as block fragments
__device__ __forceinline__ void dmma8(double2& c, const double2& a, const double2& b) {
  dmma(c.x, c.y, a.x, b.x);
  dmma(c.x, c.y, a.y, b.y);
}

__device__ __forceinline__ void blk_load_row(const double* b, int r, double (&x)[8]) {
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const double2 v = *reinterpret_cast<const double2*>(b + blk_elem(r, 2 * c));
    x[2 * c] = v.x;
    x[2 * c + 1] = v.y;
  }
}
__device__ __forceinline__ void blk_store_row(double* b, int r, const double (&x)[8]) {
#pragma unroll
  for (int c = 0; c < 4; ++c) *reinterpret_cast<double2*>(b + blk_elem(r, 2 * c)) = make_double2(x[2 * c], x[2 * c + 1]);
}
template <int ID>
__device__ __forceinline__ void named_barrier(int threads) {
  asm volatile("bar.sync %0, %1;" ::"n"(ID), "r"(threads) : "memory");
}

// One warp's share (warp u of nu) of the rank-8 update of block columns js ..
// nbt - 1 by panel p: block rows in a there-and-back order, so that two rows of
// a warp have as many blocks as any other two.  row_done(i) follows block row i.
template <typename RowDone>
__device__ __forceinline__ void panel_update(double* S, int p, int js, int nbt, int u, int nu, int lane,
                                             RowDone&& row_done) {
  const int fo = blk_frag(lane);
  const double* Lp = S + blk_index(p, p, nbt) * kBlkElems + fo;       // block (i, p) at Lp + 64 (i - p)
  for (int m = 0; js + m < nbt; m += 2 * nu) {
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
      const int i = js + m + (hh ? 2 * nu - 1 - u : u);
      if (i >= nbt) continue;
      double2 a = *reinterpret_cast<const double2*>(Lp + (i - p) * kBlkElems);
      a.x = -a.x;
      a.y = -a.y;
      for (int j0 = js; j0 <= i; j0 += 4) {
        double2 b[4], c[4];
#pragma unroll
        for (int v = 0; v < 4; ++v)
          if (j0 + v <= i) {
            b[v] = *reinterpret_cast<const double2*>(Lp + (j0 + v - p) * kBlkElems);
            c[v] = *reinterpret_cast<const double2*>(S + blk_index(i, j0 + v, nbt) * kBlkElems + fo);
          }
#pragma unroll
        for (int v = 0; v < 4; ++v)
          if (j0 + v <= i) dmma8(c[v], a, b[v]);
#pragma unroll
        for (int v = 0; v < 4; ++v)
          if (j0 + v <= i) *reinterpret_cast<double2*>(S + blk_index(i, j0 + v, nbt) * kBlkElems + fo) = c[v];
      }
      row_done(i);
    }
  }
}

// Scratch of chol_panels in shared memory, in doubles: two staged diagonal
// blocks and the pivots' reciprocal roots; with small-pivot tracking the
// diagonal entries its test compares with.
__host__ __device__ constexpr int chol_scratch_elems(int max_rows, bool track) {
  return 2 * kBlkElems + max_rows * (track ? 2 : 1);
}

// Right-looking partial Cholesky of the first nbp of nbt block columns of S,
// in place: L in the first nbp block columns, the Schur complement of the rest.
// Run by (PW + UW) warps, nbt <= 4 PW.  Two roles:
//   panel warps (the first PW, thread t owns row t): every thread factors the
//     current 8 x 8 diagonal block redundantly in registers, its own row
//     carried along as a ninth one, so that a pivot costs one 1/sqrt, one
//     product and one multiply-add of latency and no exchange between lanes;
//     then, with the finished panel visible, its row of the next block column;
//   update warps: the panel's rank-8 update of the block columns after the
//     next, on m8n8k4 DMMA, while the panel warps factor the next panel.
// The last panel's update is shared by all warps.
// Dinv (optional, nbp blocks): the inverses of the diagonal blocks.
// track: dgs holds, per 32-column group, the diagonal as it stood when the
// group was reached, and on_small() is called once per group with a pivot not
// above 2^-12 of it; on_bad(j) with the first non-positive pivot (0-based).
// The caller synchronises before (S complete) and after.
//
// What bounds it: the pivot chain, 73 cycles per column (rsqrt 55, DMUL 9,
// DFMA 9) plus about 400 per 8 columns for the exchange of the next diagonal
// block and two barriers.
template <int PW, int UW, bool kInv, bool kTrack, typename OnBad, typename OnSmall>
__device__ __forceinline__ void chol_panels(double* S, double* scratch, double* Dinv, int nbp, int nbt, OnBad&& on_bad,
                                            OnSmall&& on_small) {
  double* Dst = scratch;                       // 2 x 64: the diagonal block being factored, by panel parity
  double* rq = scratch + 2 * kBlkElems;         // 8 per panel: 1 / L_kk
  double* dgs = rq + 32 * PW;                   // kTrack: reference diagonal
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  if (warp < PW) {
    const int R = t >> 3, rr = t & 7;
    double x[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) x[k] = 0.0;
    if (R < nbt) blk_load_row(S + blk_index(R, 0, nbt) * kBlkElems, rr, x);
    if (R == 0) blk_store_row(Dst, rr, x);
    if (kTrack && R < 4 && R < nbp) dgs[t] = S[blk_index(R, R, nbt) * kBlkElems + blk_elem(rr, rr)];
    named_barrier<1>(32 * PW);
    bool reported = false, small = false;
    for (int p = 0; p < nbp; ++p) {
      if (4 * warp + 3 >= p && 4 * warp < nbt) {         // the warp still has rows at or below the diagonal block
        double a[8][8];
        const double* D = Dst + (p & 1) * kBlkElems;
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int c = 0; c <= i / 2; ++c) {
            const double2 v = *reinterpret_cast<const double2*>(D + blk_elem(i, 2 * c));
            a[i][2 * c] = v.x;
            if (2 * c + 1 <= i) a[i][2 * c + 1] = v.y;
          }
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          double d = a[k][k];
          if constexpr (kTrack) small |= !(d > dgs[8 * p + k] * (1.0 / 4096.0));
          if (!(d > 0.0)) {                              // uniform: every thread holds the same block
            if (!reported) {
              if (t == 8 * p) on_bad(8 * p + k);
              reported = true;
            }
            d = 1.0;
          }
          const double y = rsqrt(d);
          if (t == 8 * p) rq[8 * p + k] = y;
          x[k] *= y;
          double l[8];
#pragma unroll
          for (int i = k + 1; i < 8; ++i) l[i] = a[i][k] * y;
#pragma unroll
          for (int j = k + 1; j < 8; ++j) {
#pragma unroll
            for (int i = j; i < 8; ++i) a[i][j] = fma(-l[i], l[j], a[i][j]);
            x[j] = fma(-x[k], l[j], x[j]);
          }
        }
        if (R >= p && R < nbt) blk_store_row(S + blk_index(R, p, nbt) * kBlkElems, rr, x);
        if constexpr (kTrack)
          if ((p & 3) == 3 || p + 1 == nbp) {
            if (small && t == 8 * p) on_small();
            small = false;
          }
      }
      __syncwarp();
      named_barrier<0>(32 * (PW + UW));                  // panel p complete; every update up to panel p - 1 applied
      if (p + 1 < nbp) {
        if (4 * warp + 3 > p && 4 * warp < nbt) {
          double c[8];
          const int Rc = R > p && R < nbt ? R : p + 1;
          blk_load_row(S + blk_index(Rc, p + 1, nbt) * kBlkElems, rr, c);
          const double* Lj = S + blk_index(p + 1, p, nbt) * kBlkElems;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            double l[8];
            blk_load_row(Lj, j, l);
#pragma unroll
            for (int k = 0; k < 8; ++k) c[j] = fma(-x[k], l[k], c[j]);
          }
          if (R == p + 1) {
            blk_store_row(Dst + ((p + 1) & 1) * kBlkElems, rr, c);
            if constexpr (kTrack)
              if ((p & 3) == 3) {
#pragma unroll
                for (int k = 0; k < 8; ++k)
                  if (k == rr) dgs[t] = c[k];
              }
          }
#pragma unroll
          for (int k = 0; k < 8; ++k) x[k] = c[k];
        }
        __syncwarp();
        named_barrier<1>(32 * PW);
      } else {
        panel_update(S, p, p + 1, nbt, warp, PW + UW, lane, [](int) {});
      }
    }
  } else {
    const int u = warp - PW;
    for (int p = 0; p < nbp; ++p) {
      named_barrier<0>(32 * (PW + UW));
      if (p + 1 < nbp) {                                 // the panel warps take block column p + 1
        panel_update(S, p, p + 2, nbt, u, UW, lane, [&](int i) {
          if constexpr (kTrack)                          // the next group's reference diagonal (its first block: above)
            if ((p & 3) == 3 && i <= p + 4 && i < nbp) {
              __syncwarp();
              if (lane < 8) dgs[8 * i + lane] = S[blk_index(i, i, nbt) * kBlkElems + blk_elem(lane, lane)];
            }
        });
      } else {
        panel_update(S, p, p + 1, nbt, warp, PW + UW, lane, [](int) {});
      }
      if constexpr (kInv) {
        if (u == p % UW && lane < 8) {                   // column `lane` of the inverse of the diagonal block
          const double* L = S + blk_index(p, p, nbt) * kBlkElems;
          double z[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) z[k] = k == lane ? 1.0 : 0.0;
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            z[k] *= rq[8 * p + k];
#pragma unroll
            for (int i = k + 1; i < 8; ++i) z[i] = fma(-L[blk_elem(i, k)], z[k], z[i]);
          }
#pragma unroll
          for (int k = 0; k < 8; ++k) Dinv[p * kBlkElems + blk_elem(k, lane)] = z[k];
        }
        __syncwarp();
      }
    }
  }
}

// One warp, eight rows: acc (8 x 8 nb, fragments) <- acc L^{-T}, L packed with
// the inverses of its diagonal blocks in their place; block columns before
// `b0` of acc are zero and stay as they are.  Right-looking: 2 + 2 (nb - 1 - b)
// m8n8k4 per block column, no shuffles.
__device__ __forceinline__ void trsm_rows8(double2 (&acc)[16], const double* L, int nb, int b0, int lane) {
  const double* Lf = L + blk_frag(lane);
#pragma unroll
  for (int b = 0; b < 16; ++b) {
    if (b >= b0 && b < nb) {
      const double* col = Lf + blk_index(b, b, nb) * kBlkElems;
      double2 xb = make_double2(0.0, 0.0);
      dmma8(xb, acc[b], *reinterpret_cast<const double2*>(col));
      acc[b] = xb;
      const double2 n = make_double2(-xb.x, -xb.y);
#pragma unroll
      for (int j = b + 1; j < 16; ++j)
        if (j < nb) dmma8(acc[j], n, *reinterpret_cast<const double2*>(col + (j - b) * kBlkElems));
    }
  }
}

}  // namespace mfd
