// Large-front solves with one right-hand side: each level's forward and
// backward sweep as one launch over its task list (plan order: a task only
// waits for tasks earlier in the list, which CTAs already running hold, so the
// sweep always progresses; every wait is bounded).
//
// What bounds a sweep is the chain of 128-column steps: at the top of the tree
// one front has the level to itself and y_{s+1} needs y_s.  A step's latency was
// 8 us: a flag's release and acquire, the vector's load behind it, the inverted
// diagonal block from L2 in four rounds, chains of 64 dependent multiply-adds.
// Here the vectors travel in exchange words that carry their own tag (the
// sweep's number), so that waiting for a value is reading it; the inverted
// block is in shared memory before the wait, the factor's entries in
// registers; sums run in four chains.  The gathers (children's vectors forward,
// ancestors' entries backward) are part of the tasks, each row once, instead of
// a launch per level and sweep.  A step now takes 5-6 us: solve of a 37 x 41 x 43
// Laplacian 1147 -> 831 us, 64^3 3.36 -> 2.48 ms.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "kernels.cuh"
#include "sweep_sync.cuh"

namespace mfd {

namespace {

// ---- exchange words -----------------------------------------------------------------
// A value travels with the sweep's tag in the same 64-bit word (FP64: its two
// halves in two words, each with the tag), read and written as one access each:
// no fence, no separate flag.
template <typename T>
struct Exchange;
template <>
struct Exchange<float> {
  using Word = unsigned long long;
  static __device__ __forceinline__ void put(Word* p, float v, uint32_t tag) {
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p),
                 "l"(((unsigned long long)tag << 32) | __float_as_uint(v))
                 : "memory");
  }
  static __device__ __forceinline__ bool get(const Word* p, uint32_t tag, float& v) {
    unsigned long long w;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(w) : "l"(p) : "memory");
    v = __uint_as_float((uint32_t)w);
    return (uint32_t)(w >> 32) == tag;
  }
};
template <>
struct Exchange<double> {
  using Word = ulonglong2;
  static __device__ __forceinline__ void put(Word* p, double v, uint32_t tag) {
    const unsigned long long b = __double_as_longlong(v), t = (unsigned long long)tag << 32;
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(t | (uint32_t)b), "l"(t | (b >> 32)) : "memory");
  }
  static __device__ __forceinline__ bool get(const Word* p, uint32_t tag, double& v) {
    unsigned long long lo, hi;
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(lo), "=l"(hi) : "l"(p) : "memory");
    v = __longlong_as_double((long long)((hi << 32) | (uint32_t)lo));
    return (uint32_t)(lo >> 32) == tag && (uint32_t)(hi >> 32) == tag;
  }
};

// Waits for the value at p (bounded; gives up when another CTA's wait expired).
template <typename T>
__device__ __forceinline__ bool wait_value(const typename Exchange<T>::Word* p, uint32_t tag, T& v, int32_t* expired,
                                           bool probe) {
  if (probe) tag ^= 0x80000000u;             // a test request: a tag that no task writes
  if (Exchange<T>::get(p, tag, v)) return true;
  const long long t0 = clock64(), limit = probe ? kSolveProbeLimit : kSolveWaitLimit;
  for (int n = 1;; ++n) {
    if (Exchange<T>::get(p, tag, v)) return true;
    if ((n & 31) == 0 && (clock64() - t0 > limit || ld_acquire_i32(expired) != 0)) {
      atomicExch(expired, 1);
      return false;
    }
  }
}

// ---- the inverted diagonal block in shared memory ---------------------------------------
// Lower triangle, columns contiguous, column k < 64 and column 127 - k sharing a
// row of 129 words: 64 x 129 words instead of 128 x 128.
constexpr int kFoldElems = 64 * 129;
__device__ __forceinline__ int fold_col(int k) { return k < 64 ? k * 128 : (127 - k) * 129 + 1; }   // entry (i, k) at + i

template <typename T>
__device__ __forceinline__ void stage_inverse(T* S, const T* Li, int w) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int k = warp; k < w; k += 8)
    for (int i = k + lane; i < w; i += 32) {
      const unsigned sa = (unsigned)__cvta_generic_to_shared(S + fold_col(k) + i);
      if constexpr (sizeof(T) == 8) asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(Li + i + (size_t)k * kSolveB));
      else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(sa), "l"(Li + i + (size_t)k * kSolveB));
    }
  asm volatile("cp.async.commit_group;\n" ::);
}
__device__ __forceinline__ void copies_done() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// ---- forward ---------------------------------------------------------------------------
// Task (f, s): y_s = Li (v_s - sum_{t<s} L_st y_t); rest tasks (128 rows below
// the columns): v -= sum_t L_rest,t y_t.  Thread (row r0 + (t mod 128), half
// t / 128) takes its half of each step's 128 columns.
//
// N: columns per half step in flight: 64, all of them, before the wait; in FP64 32
// where the level has more tasks than SMs, so that two CTAs share an SM (in FP32
// two do with 64).
template <typename T, int N, bool kMany>
__global__ void __launch_bounds__(256, N == 64 && sizeof(T) == 8 ? 1 : 2) k_fwd_single(DevFronts F, const int4* __restrict__ tasks, int ntask,
                                                    int32_t* ticket, int32_t* expired, const int32_t* epoch,
                                                    const T* __restrict__ panel, const T* __restrict__ dinv, T* X, T* V,
                                                    const double* __restrict__ G, typename Exchange<T>::Word* E,
                                                    const int32_t* test_req) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* Ls = reinterpret_cast<T*>(smem_raw);
  __shared__ int sh_t;
  __shared__ T ys[2][kSolveB], vs[kSolveB], part[2][kSolveB];
  const bool probe = *test_req != 0;
  const uint32_t tag = 2u * (uint32_t)*epoch;
  if (threadIdx.x == 0) sh_t = atomicAdd(ticket, 1);
  __syncthreads();
  const int t = sh_t;
  if (t >= ntask) return;
  const int4 tk = tasks[t];
  const int f = tk.x, code = tk.y;
  const int nc = F.nc[f], nf = nc + F.nr[f], first = F.first[f];
  const int r0 = code >= 0 ? code * kSolveB : nc + (-1 - code) * kSolveB;
  const int r1 = min(code >= 0 ? nc : nf, r0 + kSolveB);
  const int nsteps = code >= 0 ? code : (nc + kSolveB - 1) / kSolveB;   // steps whose y this task consumes
  const T* P = panel + F.panel_off[f];
  const int tid = threadIdx.x, ri = tid & (kSolveB - 1), h = tid >> 7;
  const int i = r0 + ri;
  const bool valid = i < r1;
  if (code >= 0) stage_inverse(Ls, dinv + F.d_off[f] + (size_t)code * kSolveB * kSolveB, r1 - r0);
  T v = T(0);
  if (h == 0 && valid) v = gather_row<kMany>(F, f, tk.w != 0, i, nf, nc, X + first, V, G, 1, 0);
  T acc[4] = {T(0), T(0), T(0), T(0)};
  for (int s = 0; s < nsteps; ++s) {
    const int c0 = s * kSolveB, w = min(kSolveB, nc - c0);
    T l[N];
    const T* pc = P + (valid ? i : 0) + (size_t)(c0 + 64 * h) * nf;
    auto load = [&](int o) {
#pragma unroll
      for (int k = 0; k < N; ++k) l[k] = (valid && 64 * h + o + k < w) ? pc[(size_t)(o + k) * nf] : T(0);
    };
    load(0);
    bool ok = true;
    if (tid < kSolveB) {
      T y = T(0);
      if (tid < w) ok = wait_value<T>(E + first + c0 + tid, tag, y, expired, probe);
      ys[s & 1][tid] = y;
    }
    if (!__syncthreads_and(ok)) {
      copies_done();
      return;
    }
    const T* y = ys[s & 1] + 64 * h;
#pragma unroll
    for (int o = 0; o < 64; o += N) {
      if (o > 0) load(o);
#pragma unroll
      for (int k = 0; k < N; ++k) acc[k & 3] += l[k] * y[o + k];
    }
  }
  const T a = (acc[0] + acc[1]) + (acc[2] + acc[3]);
  if (h == 1) part[0][ri] = a;
  copies_done();
  __syncthreads();
  if (h == 0) v = valid ? v - (a + part[0][ri]) : T(0);
  if (code < 0) {
    if (h == 0 && valid) V[F.v_off[f] + i] = v;
    return;
  }
  if (h == 0) vs[ri] = v;
  __syncthreads();
  // y = Li v: columns k <= ri of this half
  T b[4] = {T(0), T(0), T(0), T(0)};
  const int k0 = 64 * h;
#pragma unroll 16
  for (int kk = 0; kk < 64; ++kk) {
    const int k = k0 + kk;
    if (k <= ri && valid) b[kk & 3] += Ls[(h ? (127 - k) * 129 + 1 : k * 128) + ri] * vs[k];
  }
  const T p = (b[0] + b[1]) + (b[2] + b[3]);
  if (h == 1) part[1][ri] = p;
  __syncthreads();
  if (h == 0 && valid) {
    const T y = p + part[1][ri];
    Exchange<T>::put(E + first + i, y, tag);
    X[first + i] = y;
  }
}

// butterfly transpose-reduce of 16 per-lane column sums: lane l ends with column (l mod 16)'s sum
template <typename T>
__device__ __forceinline__ T transpose_reduce16(T (&acc)[16], int lane) {
#pragma unroll
  for (int sft = 8; sft >= 1; sft >>= 1) {
    const bool up = (lane & sft) != 0;
#pragma unroll
    for (int j = 0; j < sft; ++j) {
      const T send = up ? acc[j] : acc[j + sft];
      const T keep = up ? acc[j + sft] : acc[j];
      acc[j] = keep + __shfl_xor_sync(0xffffffffu, send, sft);
    }
  }
  return acc[0] + __shfl_xor_sync(0xffffffffu, acc[0], 16);
}

// ---- backward --------------------------------------------------------------------------
// First the partial sums over the update rows (chunks of kBwdRestRows against a
// column block, their x known from the ancestors), then the column blocks from
// the last down: x_s = Li^T (v_s - L_below,s^T x_below), the chunks' partials
// added in chunk order, before the wait on the later blocks.  Warp w takes
// columns 16 w .. 16 w + 15 of the block, lanes rows.
//
// Q: 32-row pieces of a later block in flight: 4, the block, before the wait, or 2
// (as N above).
template <typename T, int Q>
__global__ void __launch_bounds__(256, Q == 4 && sizeof(T) == 8 ? 1 : 2) k_bwd_single(DevFronts F, const int4* __restrict__ tasks, int ntask,
                                                    int32_t* ticket, int32_t* expired, const int32_t* epoch,
                                                    const T* __restrict__ panel, const T* __restrict__ dinv, T* X,
                                                    typename Exchange<T>::Word* E, T* part, int32_t* counters,
                                                    const int32_t* test_req) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* Ls = reinterpret_cast<T*>(smem_raw);
  __shared__ int sh_t, sh_ok;
  __shared__ T ts[kSolveB];
  const bool probe = *test_req != 0;
  const uint32_t tag = 2u * (uint32_t)*epoch + 1u;
  if (threadIdx.x == 0) sh_t = atomicAdd(ticket, 1);
  __syncthreads();
  const int t = sh_t;
  if (t >= ntask) return;
  const int4 tk = tasks[t];
  const int f = tk.x;
  const int nc = F.nc[f], nr = F.nr[f], nf = nc + nr, first = F.first[f];
  const int nsteps = (nc + kSolveB - 1) / kSolveB;
  const int nch = (nr + kBwdRestRows - 1) / kBwdRestRows;
  const T* P = panel + F.panel_off[f];
  T* Pt = part + tk.w;                        // the front's partial sums: [step][chunk][128]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wc = 16 * warp;
  T acc[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) acc[j] = T(0);
  if (tk.y < 0) {                             // update-row chunk j against column block s
    const int code = -1 - tk.y, s = code >> 16, j = code & 0xffff;
    const int c0 = s * kSolveB, w = min(kSolveB, nc - c0);
    const int ra = nc + j * kBwdRestRows, rb = min(nf, ra + kBwdRestRows);
    const int32_t* lr = F.lrow + F.lrow_off[f] - nc;
#pragma unroll 2
    for (int rr = ra; rr < rb; rr += 32) {
      const int r = rr + lane;
      const bool ok = r < rb;
      const T xv = ok ? X[lr[r]] : T(0);
      const T* pr = P + (ok ? r : ra) + (size_t)(c0 + wc) * nf;
#pragma unroll
      for (int q = 0; q < 16; ++q) acc[q] += (ok && wc + q < w ? pr[(size_t)q * nf] : T(0)) * xv;
    }
    const T sum = transpose_reduce16(acc, lane);
    if (lane < 16) Pt[((size_t)s * nch + j) * kSolveB + wc + lane] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      atomicAdd(&counters[tk.z + s], 1);
    }
    return;
  }
  const int s = tk.y;
  const int c0 = s * kSolveB, w = min(kSolveB, nc - c0);
  stage_inverse(Ls, dinv + F.d_off[f] + (size_t)s * kSolveB * kSolveB, w);
  if (nch > 0 && !cta_wait_flag(counters + tk.z + s, expired, &sh_ok, probe, nch)) {
    copies_done();
    return;
  }
  T own = T(0), rsum = T(0);
  if (lane < 16 && wc + lane < w) {
    own = X[first + c0 + wc + lane];
    for (int j = 0; j < nch; ++j) rsum += __ldcg(&Pt[((size_t)s * nch + j) * kSolveB + wc + lane]);
  }
  bool good = true;
  for (int b = nsteps - 1; b > s && good; --b) {                           // later diagonal blocks
    const int ra = b * kSolveB, rb = min(nc, ra + kSolveB);
#pragma unroll
    for (int o = 0; o < 4; o += Q) {
      T l[Q][16];
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const int r = ra + lane + 32 * (o + q);
        const T* pr = P + (r < rb ? r : ra) + (size_t)(c0 + wc) * nf;
#pragma unroll
        for (int j = 0; j < 16; ++j) l[q][j] = (r < rb && wc + j < w) ? pr[(size_t)j * nf] : T(0);
      }
      T xv[Q];
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const int r = ra + lane + 32 * (o + q);
        xv[q] = T(0);
        if (r < rb && good) good = wait_value<T>(E + first + r, tag, xv[q], expired, probe);
      }
#pragma unroll
      for (int q = 0; q < Q; ++q)
#pragma unroll
        for (int j = 0; j < 16; ++j) acc[j] += l[q][j] * xv[q];
    }
    good = __all_sync(0xffffffffu, good);
  }
  const T dsum = transpose_reduce16(acc, lane);           // lane l: column wc + (l mod 16), diagonal blocks
  if (lane < 16) ts[wc + lane] = wc + lane < w ? own - (rsum + dsum) : T(0);
  copies_done();
  if (!__syncthreads_and(good)) return;
  // x = Li^T t: column i of Li against t, lanes over k
  T tv[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) tv[q] = ts[lane + 32 * q];
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    const int i = wc + j;
    const T* col = Ls + fold_col(i);
    T sum = T(0);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int k = lane + 32 * q;
      if (k >= i && k < w) sum += col[k] * tv[q];
    }
    acc[j] = sum;
  }
  const T x = transpose_reduce16(acc, lane);
  if (lane < 16 && wc + lane < w) {
    Exchange<T>::put(E + first + c0 + wc + lane, x, tag);
    X[first + c0 + wc + lane] = x;
  }
}

// zeroes the sweep's tickets, flags and counters and starts the next one's tag
__global__ void k_solve_begin(int32_t* sync, int64_t n, int32_t* epoch) {
  const int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (int64_t i = i0; i < n; i += (int64_t)gridDim.x * blockDim.x) sync[i] = 0;
  if (i0 == 0) *epoch += 1;
}

}  // namespace

cudaError_t prepare_solve_single() {
  cudaError_t e = cudaSuccess;
  auto chk = [&](auto k, size_t bytes) {
    cudaError_t r = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (r != cudaSuccess && e == cudaSuccess) e = r;
  };
  auto fwd = [&](auto k, auto k_many, size_t bytes) { chk(k, bytes); chk(k_many, bytes); };
  fwd(k_fwd_single<double, 64, false>, k_fwd_single<double, 64, true>, kFoldElems * sizeof(double)); chk(k_bwd_single<double, 4>, kFoldElems * sizeof(double));
  fwd(k_fwd_single<double, 32, false>, k_fwd_single<double, 32, true>, kFoldElems * sizeof(double)); chk(k_bwd_single<double, 2>, kFoldElems * sizeof(double));
  fwd(k_fwd_single<float, 64, false>, k_fwd_single<float, 64, true>, kFoldElems * sizeof(float)); chk(k_bwd_single<float, 4>, kFoldElems * sizeof(float));
  return e;
}

void launch_solve_begin(int32_t* sync, int64_t n, int32_t* epoch, cudaStream_t st) {
  k_solve_begin<<<(int)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, kNumSms * 4)), 256, 0, st>>>(sync, n, epoch);
}

template <typename T>
void launch_large_fused(const DevFronts& F, const int4* tasks, int ntask, bool backward, int32_t* ticket,
                        int32_t* expired, const int32_t* epoch, const T* panel, const T* dinv, T* X, T* V, const double* G,
                        void* exch, cudaStream_t st, const int32_t* test_req, T* part, int32_t* counters) {
  if (ntask <= 0) return;
  auto* E = static_cast<typename Exchange<T>::Word*>(exch);
  const size_t sm = kFoldElems * sizeof(T);
  auto bwd = [&](auto k) {
    k<<<ntask, 256, sm, st>>>(F, tasks, ntask, ticket, expired, epoch, panel, dinv, X, E, part, counters, test_req);
  };
  auto fwd = [&](auto k) {
    k<<<ntask, 256, sm, st>>>(F, tasks, ntask, ticket, expired, epoch, panel, dinv, X, V, G, E, test_req);
  };
  if constexpr (sizeof(T) == 8) {
    if (ntask > kNumSms) {
      if (backward) bwd(k_bwd_single<T, 2>);
      else if (G) fwd(k_fwd_single<T, 32, true>);
      else fwd(k_fwd_single<T, 32, false>);
      return;
    }
  }
  if (backward) bwd(k_bwd_single<T, 4>);
  else if (G) fwd(k_fwd_single<T, 64, true>);
  else fwd(k_fwd_single<T, 64, false>);
}

#define MFD_INSTANTIATE_SINGLE(T)                                                                                  \
  template void launch_large_fused<T>(const DevFronts&, const int4*, int, bool, int32_t*, int32_t*, const int32_t*, \
                                      const T*, const T*, T*, T*, const double*, void*, cudaStream_t, const int32_t*,  \
                                      T*, int32_t*);
MFD_INSTANTIATE_SINGLE(double)
MFD_INSTANTIATE_SINGLE(float)

}  // namespace mfd
