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

// Row and column of the t-th tile of a lower triangle, row by row (the same for every size).
__device__ __forceinline__ void tile_table(uint16_t* tab, int rows) {
  for (int i = threadIdx.x >> 5; i < rows; i += blockDim.x >> 5)
    for (int j = threadIdx.x & 31; j <= i; j += 32) tab[i * (i + 1) / 2 + j] = (uint16_t)(i << 8 | j);
}

// Block columns js .. nbt - 1 -= the K panels p .. p + K - 1, warp u of nu, in 2 x 2
// blocks.  Shared memory bounds it (a block moves in 4 cycles): single blocks a
// panel at a time take 16 cycles per block and panel, 2 x 2 of two panels 8.
template <int K>
__device__ __forceinline__ void panel_update(double* S, const uint16_t* tab, int p, int js, int nbt, int u, int nu,
                                             int lane) {
  const int fo = blk_frag(lane), T = (nbt - js + 1) / 2;
  for (int t = u; t < T * (T + 1) / 2; t += nu) {
    const int ij = tab[t], i0 = js + 2 * (ij >> 8), j0 = js + 2 * (ij & 255);
    double2 a[K][2], b[K][2], c[2][2];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const double* L = S + (blk_index(p + k, p + k, nbt) - (p + k)) * kBlkElems + fo;   // block (i, p + k) at L + 64 i
#pragma unroll
      for (int v = 0; v < 2; ++v) {
        a[k][v] = *reinterpret_cast<const double2*>(L + min(i0 + v, nbt - 1) * kBlkElems);
        b[k][v] = *reinterpret_cast<const double2*>(L + min(j0 + v, nbt - 1) * kBlkElems);
        a[k][v] = make_double2(-a[k][v].x, -a[k][v].y);
      }
    }
    // block (i0 + v, j0 + w); above the diagonal or past the last block: not there
    auto there = [&](int v, int w) { return i0 + v < nbt && j0 + w < nbt && i0 + v >= j0 + w; };
    auto at = [&](int v, int w) { return reinterpret_cast<double2*>(S + blk_index(i0 + v, j0 + w, nbt) * kBlkElems + fo); };
#pragma unroll
    for (int v = 0; v < 2; ++v)
#pragma unroll
      for (int w = 0; w < 2; ++w)
        if (there(v, w)) c[v][w] = *at(v, w);
#pragma unroll
    for (int k = 0; k < K; ++k)
#pragma unroll
      for (int v = 0; v < 2; ++v)
#pragma unroll
        for (int w = 0; w < 2; ++w)
          if (there(v, w)) dmma8(c[v][w], a[k][v], b[k][w]);
#pragma unroll
    for (int v = 0; v < 2; ++v)
#pragma unroll
      for (int w = 0; w < 2; ++w)
        if (there(v, w)) *at(v, w) = c[v][w];
  }
}
// Block column p + 1 alone, one block per warp at a time.
__device__ __forceinline__ void next_column_update(double* S, int p, int nbt, int u, int nu, int lane) {
  const int fo = blk_frag(lane);
  const double* L = S + (blk_index(p, p, nbt) - p) * kBlkElems + fo;
  for (int i = p + 1 + u; i < nbt; i += nu) {
    double2* C = reinterpret_cast<double2*>(S + blk_index(i, p + 1, nbt) * kBlkElems + fo);
    double2 a = *reinterpret_cast<const double2*>(L + i * kBlkElems), c = *C;
    dmma8(c, make_double2(-a.x, -a.y), *reinterpret_cast<const double2*>(L + (p + 1) * kBlkElems));
    *C = c;
  }
}

// Scratch of chol_panels in shared memory, in doubles: two 4 x 4 exchange blocks,
// the pivots' reciprocal roots, with small-pivot tracking the diagonal its test
// compares with, and the tile table.
__host__ __device__ constexpr int chol_scratch_elems(int max_rows, bool track) {
  return 32 + max_rows * (track ? 2 : 1) + (blk_count((max_rows / 8 + 1) / 2) + 3) / 4;
}

// Cholesky of the N x N lower block a (redundantly by every thread that calls
// it), the thread's own row x carried along: x <- x L^{-T}.  a[k][k] ends as the
// pivots (a non-positive one counts as 1), y as their 1 / sqrt; nothing but the
// arithmetic is on the chain, the caller looks at the pivots afterwards.
template <int N>
__device__ __forceinline__ void chol_row(double (&a)[N][N], double* x, double (&y)[N]) {
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const double r = rsqrt(a[k][k]);
    y[k] = a[k][k] > 0.0 ? r : 1.0;
    x[k] *= y[k];
    double l[N];
#pragma unroll
    for (int i = k + 1; i < N; ++i) l[i] = a[i][k] * y[k];
#pragma unroll
    for (int j = k + 1; j < N; ++j) {
#pragma unroll
      for (int i = j; i < N; ++i) a[i][j] = fma(-l[i], l[j], a[i][j]);
      x[j] = fma(-x[k], l[j], x[j]);
    }
  }
}

// Right-looking partial Cholesky of the first nbp of nbt block columns of S,
// in place: L in the first nbp block columns, the Schur complement of the rest.
// Run by NW warps with 8 nbt <= 32 NW; thread t owns row t.  Per block column:
//   factor, by the warps with rows at or below the diagonal block: every thread
//     factors it redundantly in registers, its own row carried along, so that a
//     pivot needs no exchange between lanes; in two 4 x 4 blocks, rows 4..7 of L
//     and the second block exchanged through shared memory;
//   update: all warps, on m8n8k4 DMMA, two panels at a time.
// rq (in scratch): 1 / L_kk.  track: on_small() once per 32-column group with a
// pivot not above 2^-12 of the diagonal entry it had when the group was reached;
// on_bad(j): a non-positive pivot (0-based; the first one counts).  The caller
// synchronises before (S complete) and after.
//
// What bounds it: the chain of pivots, 105 cycles each (rsqrt 55, DMUL 9, DFMA 9,
// the issue of one warp's FP64 at 4.5 cycles per instruction), 1,330 cycles per
// eight columns with the exchanges; then the update's shared-memory traffic.
// Measured alternatives, 128 x 128: factor and update side by side in different
// warps 2,450 cycles per panel (both slow each other down), 8 x 8 blocks without
// the exchanges 1,500 per factor and 175 registers for 110.
constexpr int kCholRq = 32;       // offset of rq in the scratch
template <int NW, bool kTrack, typename OnBad, typename OnSmall>
__device__ __forceinline__ void chol_panels(double* S, double* scratch, int nbp, int nbt, OnBad&& on_bad,
                                            OnSmall&& on_small) {
  constexpr int N = 4;
  double* low = scratch;                                 // rows 4..7 of the diagonal block: L's first four columns
  double* next = scratch + 16;                            // and their last four, before the second 4 x 4 block
  double* rq = scratch + kCholRq;
  double* dgs = rq + 8 * nbp;                            // kTrack
  uint16_t* tab = reinterpret_cast<uint16_t*>(dgs + (kTrack ? 8 * nbp : 0));
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int R = t >> 3, rr = t & 7;
  tile_table(tab, (nbt + 1) / 2);
  bool small = false;
  for (int p = 0; p < nbp; ++p) {
    if (4 * warp + 3 >= p && 4 * warp < nbt) {           // the warp has rows at or below the diagonal block
      const int bar = 32 * ((nbt + 3) / 4 - p / 4);      // threads of such warps
      const double* D = S + blk_index(p, p, nbt) * kBlkElems;
      const bool mine = R >= p && R < nbt;
      double a[N][N], x[8], dg[N];
      auto load = [&](auto at) {                         // at(i, c): columns 2 c, 2 c + 1 of row i
#pragma unroll
        for (int i = 0; i < N; ++i)
#pragma unroll
          for (int c = 0; c <= i / 2; ++c) {
            const double2 v = at(i, c);
            a[i][2 * c] = v.x;
            a[i][2 * c + 1] = v.y;
          }
      };
      load([&](int i, int c) { return *reinterpret_cast<const double2*>(D + blk_elem(i, 2 * c)); });
      blk_load_row(S + blk_index(mine ? R : p, p, nbt) * kBlkElems, rr, x);
      if constexpr (kTrack) {
#pragma unroll
        for (int k = 0; k < N; ++k) dg[k] = (p & 3) == 0 ? a[k][k] : dgs[8 * p + k];
        if ((p & 3) == 0 && mine && R < min(p + 4, nbp)) dgs[t] = S[blk_index(R, R, nbt) * kBlkElems + blk_elem(rr, rr)];
      }
      auto factor = [&](int o) {                         // columns o .. o + N - 1 of the panel
        double y[N];
        chol_row<N>(a, x + o, y);
        bool good = true;
#pragma unroll
        for (int k = 0; k < N; ++k) {
          good &= a[k][k] > 0.0;
          if constexpr (kTrack) small |= !(a[k][k] > dg[k] * (1.0 / 4096.0));
        }
        if (t == 8 * p) {
#pragma unroll
          for (int k = 0; k < N; k += 2) *reinterpret_cast<double2*>(rq + 8 * p + o + k) = make_double2(y[k], y[k + 1]);
          if (!good)
#pragma unroll
            for (int k = N - 1; k >= 0; --k)             // the first one last: the caller keeps the smallest
              if (!(a[k][k] > 0.0)) on_bad(8 * p + o + k);
        }
      };
      factor(0);
      if (R == p && rr >= 4) {
        *reinterpret_cast<double2*>(low + 4 * (rr - 4)) = make_double2(x[0], x[1]);
        *reinterpret_cast<double2*>(low + 4 * (rr - 4) + 2) = make_double2(x[2], x[3]);
      }
      __syncwarp();
      named_barrier<1>(bar);                           // also: every thread has read the diagonal block
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const double2 l0 = *reinterpret_cast<const double2*>(low + 4 * j), l1 = *reinterpret_cast<const double2*>(low + 4 * j + 2);
        x[4 + j] = fma(-x[0], l0.x, x[4 + j]);
        x[4 + j] = fma(-x[1], l0.y, x[4 + j]);
        x[4 + j] = fma(-x[2], l1.x, x[4 + j]);
        x[4 + j] = fma(-x[3], l1.y, x[4 + j]);
      }
      if (R == p && rr >= 4) {
        *reinterpret_cast<double2*>(next + 4 * (rr - 4)) = make_double2(x[4], x[5]);
        *reinterpret_cast<double2*>(next + 4 * (rr - 4) + 2) = make_double2(x[6], x[7]);
      }
      __syncwarp();
      named_barrier<1>(bar);
      load([&](int i, int c) { return *reinterpret_cast<const double2*>(next + 4 * i + 2 * c); });
      if constexpr (kTrack) {
#pragma unroll
        for (int k = 0; k < 4; ++k) dg[k] = dgs[8 * p + 4 + k];
      }
      factor(4);
      if (mine) blk_store_row(S + blk_index(R, p, nbt) * kBlkElems, rr, x);
      if constexpr (kTrack)
        if ((p & 3) == 3 || p + 1 == nbp) {
          if (small && t == 8 * p) on_small();
          small = false;
        }
    }
    __syncthreads();
    // two panels at a time: after the first of a pair only the second's block column
    if ((p & 1) == 0 && p + 1 < nbp) next_column_update(S, p, nbt, warp, NW, lane);
    else if ((p & 1) == 0) panel_update<1>(S, tab, p, p + 1, nbt, warp, NW, lane);
    else panel_update<2>(S, tab, p - 1, p + 1, nbt, warp, NW, lane);
    __syncthreads();
  }
}

// Dinv (nbp blocks): the inverses of the diagonal blocks of L, one column per thread.
__device__ __forceinline__ void invert_diagonal_blocks(const double* S, const double* rq, double* Dinv, int nbp, int nbt) {
  const int t = threadIdx.x, p = t >> 3, c = t & 7;
  if (p >= nbp) return;
  const double* L = S + blk_index(p, p, nbt) * kBlkElems;
  double z[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) z[k] = k == c ? 1.0 : 0.0;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    z[k] *= rq[8 * p + k];
#pragma unroll
    for (int i = k + 1; i < 8; ++i) z[i] = fma(-L[blk_elem(i, k)], z[k], z[i]);
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) Dinv[p * kBlkElems + blk_elem(k, c)] = z[k];
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
