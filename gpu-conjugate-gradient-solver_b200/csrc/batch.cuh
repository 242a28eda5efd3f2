// Kernels of the batched AMG-PCG solver: many independent systems of uneven
// sizes, each with up to four right-hand sides, advanced together.
//
// Storage. Level k of the batch is the block-diagonal matrix of every
// system's level-k matrix, systems one after another, each system's rows in
// its own colour-contiguous order. The R right-hand sides of a system share
// its matrix: vectors are stored row-interleaved ([row][R]), so one read of a
// matrix entry serves R updates and a neighbour gather is one R-wide load.
//
// Work lists. Every launch walks a list of items (system, begin, end, aux):
// a range of SELL-32 slices or of rows of one system (never crossing systems
// or colours), with aux the first row of the item's colour where it matters.
// The blocks of a launch loop over the list (grid-stride), so one launch
// carries the same pass of every system: colour j of the forward sweep is
// colour j of each system, colour C_s - 1 - j of the backward sweep. An item
// whose system has finished (every right-hand side converged) is skipped.
//
// Outer CG (FP64). Per (system, right-hand side) pair the scalars live in
// BPair on the device. Item kernels write per-item partial sums; one block
// per system then adds its items' partials in a fixed order (deterministic)
// and updates the pair scalars and the convergence flags.
#pragma once

#include "kernels.cuh"

namespace gsb {

template <typename T, int R>
struct alignas(sizeof(T) * R) Rv {
  T v[R];
};

template <typename T, int R>
__device__ __forceinline__ Rv<T, R> rv_zero() {
  Rv<T, R> z;
#pragma unroll
  for (int j = 0; j < R; ++j) z.v[j] = T(0);
  return z;
}

// Read-only (non-coherent) load of the R values of one row.
template <typename T, int R>
__device__ __forceinline__ Rv<T, R> ldg_rv(const Rv<T, R> *p) {
  Rv<T, R> r;
  if constexpr (R == 4 && sizeof(T) == 4) {
    const float4 q = __ldg(reinterpret_cast<const float4 *>(p));
    r.v[0] = q.x, r.v[1] = q.y, r.v[2] = q.z, r.v[3] = q.w;
  } else if constexpr (R == 4 && sizeof(T) == 8) {
    const double2 a = __ldg(reinterpret_cast<const double2 *>(p));
    const double2 b = __ldg(reinterpret_cast<const double2 *>(p) + 1);
    r.v[0] = a.x, r.v[1] = a.y, r.v[2] = b.x, r.v[3] = b.y;
  } else {
#pragma unroll
    for (int j = 0; j < R; ++j) r.v[j] = __ldg(&p->v[j]);
  }
  return r;
}

template <typename T, int R>
__device__ __forceinline__ void fma_rv(T a, const Rv<T, R> &x, Rv<T, R> &acc) {
#pragma unroll
  for (int j = 0; j < R; ++j) acc.v[j] = fma(a, x.v[j], acc.v[j]);
}

// Items: x = system, y = begin, z = end, w = aux.
using BItem = int4;

// Entry of every kernel of an iteration (kernels.cuh: pass_entry, without the
// stop flag: a finished system's items are skipped one by one). Whatever an
// earlier kernel of the iteration writes -- vectors, pair scalars, sys_done --
// is read after it, through pointers that are not const __restrict__ (which
// would promise that nobody writes the data while the kernel runs) or that
// after_wait holds back; items and matrices never change during a solve.
__device__ __forceinline__ void bpass_entry() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

__device__ __forceinline__ bool item_skipped(const int *sys_done, int sys) {
  return sys_done != nullptr && reinterpret_cast<const volatile int *>(sys_done)[sys] != 0;
}

// ---- SELL-32, one lane per row -------------------------------------------
// kHead of the kernels below: with it the first item's matrix entries are loaded
// before the wait on the predecessor and held in registers, which is what a
// short list of items waits for; on a long list, bound by bandwidth, the
// registers halve the warps in flight (FP32, 4 right-hand sides: 64 a thread
// against 32 in the colour pass, 48 against 32 in the product). The lists are
// told apart by their items in blocks that fill the device (148 SMs x 8): up to
// 4 times as many slice items or 8 times as many row items take the head.
// Measured (one B200, 64 systems of 16^3 to 96^3, 4 FP32 right-hand sides, head /
// no head): slices: sweep of 31,600 items a pass 397 / 331 us, product of 9,300
// 61 / 47, product of 1,300 8.6 / 10.5, sweep of 585 a pass 541 / 565; rows: sweep
// of 2,300 a pass 482 / 516, of 4,700 505 / 514, product of 5,300 48 / 52, of
// 10,500 102 / 91, of 39,700 369 / 325. The solve: 176.3 ms with the head
// throughout, 182.7 without, 169.5 by this rule.
constexpr int kHeadSliceItems = 4;
constexpr int kHeadRowItems = 8;

template <typename T, int R, bool kSkip>
__device__ __forceinline__ Rv<T, R> bsell_offdiag(const SellView<T> &A, int s, int lane,
                                                  const Rv<T, R> *__restrict__ x, int skip_from) {
  using P2 = typename Pair<T>::type;
  const int p0 = A.sptr[s], p1 = kSkip && A.lo != nullptr ? A.lo[s] : A.sptr[s + 1];
  Rv<T, R> sum = rv_zero<T, R>();
#pragma unroll 2
  for (int p = p0 + 2 * lane; p < p1; p += 64) {
    const P2 v = __ldg(reinterpret_cast<const P2 *>(A.val + p));
    const int2 c = __ldg(reinterpret_cast<const int2 *>(A.col + p));
    if (!kSkip || c.x < skip_from) fma_rv<T, R>(v.x, ldg_rv<T, R>(x + c.x), sum);
    if (!kSkip || c.y < skip_from) fma_rv<T, R>(v.y, ldg_rv<T, R>(x + c.y), sum);
  }
  return sum;
}

// bsell_offdiag with the first slot pairs taken from a head loaded earlier
// (kernels.cuh): the same sums in the same order.
template <typename T, int R, bool kSkip>
__device__ __forceinline__ Rv<T, R> bsell_offdiag_head(const SellView<T> &A, const SellHead<T> &h, int lane,
                                                       const Rv<T, R> *__restrict__ x, int skip_from) {
  using P2 = typename Pair<T>::type;
  constexpr int kP = SellHead<T>::kPairs;
  Rv<T, R> g[2 * kP];
#pragma unroll
  for (int q = 0; q < kP; ++q) {
    g[2 * q] = h.c[q].x >= 0 && (!kSkip || h.c[q].x < skip_from) ? ldg_rv<T, R>(x + h.c[q].x) : rv_zero<T, R>();
    g[2 * q + 1] = h.c[q].y >= 0 && (!kSkip || h.c[q].y < skip_from) ? ldg_rv<T, R>(x + h.c[q].y) : rv_zero<T, R>();
  }
  Rv<T, R> sum = rv_zero<T, R>();
#pragma unroll
  for (int q = 0; q < kP; ++q) {
    fma_rv<T, R>(h.v[q].x, g[2 * q], sum);
    fma_rv<T, R>(h.v[q].y, g[2 * q + 1], sum);
  }
#pragma unroll 2
  for (int p = h.p0 + 64 * kP + 2 * lane; p < h.p1; p += 64) {
    const P2 v = __ldg(reinterpret_cast<const P2 *>(A.val + p));
    const int2 c = __ldg(reinterpret_cast<const int2 *>(A.col + p));
    if (!kSkip || c.x < skip_from) fma_rv<T, R>(v.x, ldg_rv<T, R>(x + c.x), sum);
    if (!kSkip || c.y < skip_from) fma_rv<T, R>(v.y, ldg_rv<T, R>(x + c.y), sum);
  }
  return sum;
}

// One row of a colour pass from its off-diagonal sum.
template <typename T, typename BT, int R, bool kZero>
__device__ __forceinline__ Rv<T, R> bgs_row(const Rv<T, R> &off, const Rv<BT, R> &b, const Rv<T, R> &old, T d, T w) {
  Rv<T, R> xn;
#pragma unroll
  for (int j = 0; j < R; ++j) {
    const T gs = (T(b.v[j]) - off.v[j]) / d;
    xn.v[j] = kZero ? w * gs : (T(1) - w) * old.v[j] + w * gs;
  }
  return xn;
}

// Gauss-Seidel colour pass, items = slice ranges of one colour of one system
// (aux = first row of that colour), at most one slice per warp:
//     x_i <- (1 - w) x_i + w (b_i - sum_{j != i} a_ij x_j) / a_ii
// for each of the R right-hand sides. kZero: x is an implicit zero vector
// before this forward sweep (columns >= aux hold zero and are not read).
template <typename T, typename BT, int R, bool kZero, bool kHead>
__global__ void __launch_bounds__(256) bsell_gs_kernel(SellView<T> A, const BItem *__restrict__ items,
                                                       int nitems, const Rv<BT, R> *__restrict__ b,
                                                       Rv<T, R> *__restrict__ x, T w,
                                                       const int *__restrict__ sys_done) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  SellHead<T> h;
  BItem q;
  if constexpr (kHead) {
    q = __ldg(items + blockIdx.x);
    if (q.y + warp < q.z) sell_head_ops(A, q.y + warp, lane, h, kZero);
  }
  bpass_entry();
  b = after_wait(b);
  x = after_wait(x);
  for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
    if (!kHead || it != static_cast<int>(blockIdx.x)) {
      q = __ldg(items + it);
      if constexpr (kHead)
        if (q.y + warp < q.z) sell_head_ops(A, q.y + warp, lane, h, kZero);
    }
    if (item_skipped(sys_done, q.x) || q.y + warp >= q.z) continue;
    if constexpr (kHead) {
      const int row = h.r0 + lane;
      const bool valid = row < h.r1;
      T d = T(1);
      Rv<BT, R> bv;
      Rv<T, R> xo = rv_zero<T, R>();
      if (valid) {
        d = __ldg(A.diag + row);
        bv = b[row];
        if (!kZero) xo = x[row];
      }
      const Rv<T, R> off = bsell_offdiag_head<T, R, kZero>(A, h, lane, x, q.w);
      if (valid) x[row] = bgs_row<T, BT, R, kZero>(off, bv, xo, d, w);
    } else {
      const int s = q.y + warp;
      const Rv<T, R> off = bsell_offdiag<T, R, kZero>(A, s, lane, x, q.w);
      const int row = A.srow[s] + lane;
      if (row < A.srow[s + 1]) {
        Rv<T, R> xo = rv_zero<T, R>();
        if (!kZero) xo = x[row];
        x[row] = bgs_row<T, BT, R, kZero>(off, b[row], xo, A.diag[row], w);
      }
    }
  }
}

// One row of y = A x (kSpmvSet), b - A x (kSpmvResid) or y + A x (kSpmvAdd)
// from its off-diagonal sum.
template <typename T, typename BT, int R, int kMode>
__device__ __forceinline__ void bspmv_store(const T *__restrict__ diag, int row, Rv<T, R> sum,
                                            const Rv<T, R> *__restrict__ x, Rv<T, R> *__restrict__ y,
                                            const Rv<BT, R> *__restrict__ b) {
  if (diag != nullptr) fma_rv<T, R>(__ldg(diag + row), x[row], sum);
  if (kMode == kSpmvResid) {
    const Rv<BT, R> bv = b[row];
#pragma unroll
    for (int j = 0; j < R; ++j) sum.v[j] = T(bv.v[j]) - sum.v[j];
  } else if (kMode == kSpmvAdd) {
    const Rv<T, R> old = y[row];
#pragma unroll
    for (int j = 0; j < R; ++j) sum.v[j] = old.v[j] + sum.v[j];
  }
  y[row] = sum;
}

// Items are slice ranges. The first slice's head is loaded before the wait on
// the predecessor, as in the colour passes.
template <typename T, typename BT, int R, int kMode, bool kHead>
__global__ void __launch_bounds__(256) bsell_spmv_kernel(SellView<T> A, const BItem *__restrict__ items,
                                                         int nitems, const Rv<T, R> *__restrict__ x,
                                                         Rv<T, R> *__restrict__ y,
                                                         const Rv<BT, R> *__restrict__ b,
                                                         const int *__restrict__ sys_done) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  BItem q;
  SellHead<T> h;
  if constexpr (kHead) {
    q = __ldg(items + blockIdx.x);
    if (q.y + warp < q.z) sell_head_ops(A, q.y + warp, lane, h);
  }
  bpass_entry();
  x = after_wait(x);
  b = after_wait(b);
  for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
    const bool first = it == static_cast<int>(blockIdx.x);
    if (!kHead || !first) q = __ldg(items + it);
    if (item_skipped(sys_done, q.x)) continue;
    for (int s = q.y + warp; s < q.z; s += nw) {
      if constexpr (kHead) {
        if (!first || s != q.y + warp) sell_head_ops(A, s, lane, h);
        const Rv<T, R> sum = bsell_offdiag_head<T, R, false>(A, h, lane, x, 0);
        const int row = h.r0 + lane;
        if (row < h.r1) bspmv_store<T, BT, R, kMode>(A.diag, row, sum, x, y, b);
      } else {
        const Rv<T, R> sum = bsell_offdiag<T, R, false>(A, s, lane, x, 0);
        const int row = A.srow[s] + lane;
        if (row < A.srow[s + 1]) bspmv_store<T, BT, R, kMode>(A.diag, row, sum, x, y, b);
      }
    }
  }
}

// ---- CSR-vector, G lanes per row -----------------------------------------
// A row's off-diagonal sum from a loaded head, the gathers of four entries
// requested together.
template <typename T, int R, bool kSkip, int G, int kE>
__device__ __forceinline__ Rv<T, R> bcsrv_offdiag_head(const CsrvView<T> &A, const CsrvHead<T, kE> &h,
                                                       const Rv<T, R> *__restrict__ x, int skip_from) {
  Rv<T, R> sum = rv_zero<T, R>();
#pragma unroll
  for (int u0 = 0; u0 < kE; u0 += 4) {
    Rv<T, R> g[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int c = h.c[u0 + u];
      g[u] = c >= 0 && (!kSkip || c < skip_from) ? ldg_rv<T, R>(x + c) : rv_zero<T, R>();
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) fma_rv<T, R>(h.v[u0 + u], g[u], sum);
  }
#pragma unroll 4
  for (int k = h.k0 + kE * G; k < h.k1; k += G) {
    const int c = __ldg(A.ci + k);
    if (!kSkip || c < skip_from) fma_rv<T, R>(__ldg(A.v + k), ldg_rv<T, R>(x + c), sum);
  }
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1)
#pragma unroll
    for (int j = 0; j < R; ++j) sum.v[j] += __shfl_xor_sync(0xffffffffu, sum.v[j], o, G);
  return sum;
}

template <typename T, int R, bool kSkip, int G>
__device__ __forceinline__ Rv<T, R> bcsrv_offdiag(const CsrvView<T> &A, int row, bool valid, int sub,
                                                  const Rv<T, R> *__restrict__ x, int skip_from) {
  Rv<T, R> sum = rv_zero<T, R>();
  if (valid) {
    const int k1 = A.re[row];
#pragma unroll 4
    for (int k = A.rp[row] + sub; k < k1; k += G) {
      const int c = __ldg(A.ci + k);
      if (!kSkip || c < skip_from) fma_rv<T, R>(__ldg(A.v + k), ldg_rv<T, R>(x + c), sum);
    }
  }
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1)
#pragma unroll
    for (int j = 0; j < R; ++j) sum.v[j] += __shfl_xor_sync(0xffffffffu, sum.v[j], o, G);
  return sum;
}

// Items are row ranges of one colour of one system (aux = first row of the
// colour), at most one row per group of G lanes. Coarse passes are
// latency-bound: the first item, its rows' first 8 entries per lane and their
// diagonals are loaded before the wait on the predecessor. Measured (one
// B200, a forward sweep of level 1): 12 systems of 16^3 to 56^3, 4 FP32
// right-hand sides, 17 passes, 105 -> 69 us; 5 systems of 14^3 to 30^3, one
// FP64 right-hand side, 18 passes, 92 -> 43 us.
template <typename T, typename BT, int R, bool kZero, int G, bool kHead>
__global__ void __launch_bounds__(256) bcsrv_gs_kernel(CsrvView<T> A, const BItem *__restrict__ items,
                                                       int nitems, const Rv<BT, R> *__restrict__ b,
                                                       Rv<T, R> *__restrict__ x, T w,
                                                       const int *__restrict__ sys_done) {
  const int sub = threadIdx.x & (G - 1), grp = threadIdx.x / G;
  BItem q;
  CsrvHead<T, 8> h;
  T d = T(1);
  if constexpr (kHead) {
    q = __ldg(items + blockIdx.x);
    csrv_head<T, G>(A, q.y + grp, q.y + grp < q.z, sub, h);
    if (q.y + grp < q.z) d = __ldg(A.diag + q.y + grp);
  }
  bpass_entry();
  b = after_wait(b);
  x = after_wait(x);
  for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
    if (!kHead || it != static_cast<int>(blockIdx.x)) {
      q = __ldg(items + it);
      if constexpr (kHead) {
        csrv_head<T, G>(A, q.y + grp, q.y + grp < q.z, sub, h);
        d = q.y + grp < q.z ? __ldg(A.diag + q.y + grp) : T(1);
      }
    }
    if (item_skipped(sys_done, q.x)) continue;
    const int row = q.y + grp;
    const bool mine = row < q.z && sub == 0;
    if constexpr (kHead) {
      Rv<BT, R> bv;
      Rv<T, R> xo = rv_zero<T, R>();
      if (mine) {
        bv = b[row];
        if (!kZero) xo = x[row];
      }
      const Rv<T, R> off = bcsrv_offdiag_head<T, R, kZero, G>(A, h, x, q.w);
      if (mine) x[row] = bgs_row<T, BT, R, kZero>(off, bv, xo, d, w);
    } else {
      const Rv<T, R> off = bcsrv_offdiag<T, R, kZero, G>(A, row, row < q.z, sub, x, q.w);
      if (mine) {
        Rv<T, R> xo = rv_zero<T, R>();
        if (!kZero) xo = x[row];
        x[row] = bgs_row<T, BT, R, kZero>(off, b[row], xo, A.diag[row], w);
      }
    }
  }
}

// Items are row ranges, at most one row per group of G lanes; the head as in
// the colour passes.
template <typename T, typename BT, int R, int kMode, int G, bool kHead>
__global__ void __launch_bounds__(256) bcsrv_spmv_kernel(CsrvView<T> A, const BItem *__restrict__ items,
                                                         int nitems, const Rv<T, R> *__restrict__ x,
                                                         Rv<T, R> *__restrict__ y,
                                                         const Rv<BT, R> *__restrict__ b,
                                                         const int *__restrict__ sys_done) {
  const int sub = threadIdx.x & (G - 1), grp = threadIdx.x / G;
  BItem q;
  CsrvHead<T, 8> h;
  if constexpr (kHead) {
    q = __ldg(items + blockIdx.x);
    csrv_head<T, G>(A, q.y + grp, q.y + grp < q.z, sub, h);
  }
  bpass_entry();
  x = after_wait(x);
  b = after_wait(b);
  for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
    if (!kHead || it != static_cast<int>(blockIdx.x)) {
      q = __ldg(items + it);
      if constexpr (kHead) csrv_head<T, G>(A, q.y + grp, q.y + grp < q.z, sub, h);
    }
    if (item_skipped(sys_done, q.x)) continue;
    const int row = q.y + grp;
    Rv<T, R> sum;
    if constexpr (kHead) sum = bcsrv_offdiag_head<T, R, false, G>(A, h, x, 0);
    else sum = bcsrv_offdiag<T, R, false, G>(A, row, row < q.z, sub, x, 0);
    if (row < q.z && sub == 0) bspmv_store<T, BT, R, kMode>(A.diag, row, sum, x, y, b);
  }
}

// ---- coarsest levels: x_c = A_c^-1 b_c per system ---------------------------
// Items: x = system, y = its coarsest level, z/w = local row range. A warp
// reads four rows of the system's dense FP64 inverse at once: the right-hand
// sides of a column are loaded and widened to FP64 once for the four rows
// (the conversions, not the inverse's bytes, bounded one row per warp), and
// four rows' loads are in flight. Per row the same sums in the same order.
// Measured (one B200, 11 coarsest levels, 17,234 rows in all, 4 FP32
// right-hand sides): 137 -> 80 us.
constexpr int kBDenseRows = 4;
template <typename T, int R>
__global__ void __launch_bounds__(256) bdense_kernel(const BItem *__restrict__ items, int nitems,
                                                     const double *__restrict__ ainv,
                                                     const long long *__restrict__ ainv_off,
                                                     const int *__restrict__ crow0,
                                                     const int *__restrict__ cn,
                                                     Rv<T, R> *const *__restrict__ xl,
                                                     const Rv<T, R> *const *__restrict__ bl,
                                                     const int *__restrict__ sys_done) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  bpass_entry();
  for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
    const BItem q = items[it];
    if (item_skipped(sys_done, q.x)) continue;
    const int n = cn[q.x], r0 = crow0[q.x];
    const Rv<T, R> *b = bl[q.y] + r0;
    Rv<T, R> *x = xl[q.y] + r0;
    const double *a = ainv + ainv_off[q.x];
    // each warp takes kBDenseRows rows at a time (the last ones clamped and not stored)
    for (int r1 = q.z + kBDenseRows * warp; r1 < q.w; r1 += kBDenseRows * nw) {
      const double *ar[kBDenseRows];
      double acc[kBDenseRows][R];
#pragma unroll
      for (int i = 0; i < kBDenseRows; ++i) {
        ar[i] = a + static_cast<size_t>(min(r1 + i, q.w - 1)) * n;
#pragma unroll
        for (int j = 0; j < R; ++j) acc[i][j] = 0.0;
      }
#pragma unroll 2
      for (int c = lane; c < n; c += 32) {
        double av[kBDenseRows];
#pragma unroll
        for (int i = 0; i < kBDenseRows; ++i) av[i] = __ldg(ar[i] + c);
        const Rv<T, R> bv = ldg_rv<T, R>(b + c);
#pragma unroll
        for (int j = 0; j < R; ++j) {
          const double bj = double(bv.v[j]);
#pragma unroll
          for (int i = 0; i < kBDenseRows; ++i) acc[i][j] = fma(av[i], bj, acc[i][j]);
        }
      }
#pragma unroll
      for (int i = 0; i < kBDenseRows; ++i) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
          for (int j = 0; j < R; ++j) acc[i][j] += __shfl_xor_sync(0xffffffffu, acc[i][j], o);
        if (lane == 0 && r1 + i < q.w) {
          Rv<T, R> out;
#pragma unroll
          for (int j = 0; j < R; ++j) out.v[j] = T(acc[i][j]);
          x[r1 + i] = out;
        }
      }
    }
  }
}

// ---- outer CG (FP64) ------------------------------------------------------
// Scalars of one (system, right-hand side) pair.
struct BPair {
  double rho, alpha, beta, rr, bb, ratio, pAp;
  int iter, done, status, iterations;
};

struct BCgShared {
  double tol2;
  int max_iter;
  int flexible;
  int active;  // systems with at least one pair still running (after the last convergence test)
  int sync_fault;  // a bounded wait of a cluster step gave up
  int arrived;     // systems past the current convergence test
  int tests;       // convergence tests run
};

// Deterministic block sum of kN values per thread into smem-backed totals;
// the result is valid in thread 0.
template <int kN>
__device__ __forceinline__ void bblock_sum(double (&v)[kN], double *smem) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int i = 0; i < kN; ++i)
    for (int o = 16; o > 0; o >>= 1) v[i] += __shfl_down_sync(0xffffffffu, v[i], o);
  __syncthreads();
  if (lane == 0)
#pragma unroll
    for (int i = 0; i < kN; ++i) smem[warp * kN + i] = v[i];
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int i = 0; i < kN; ++i) {
      double t = 0.0;
      for (int q = 0; q < nw; ++q) t += smem[q * kN + i];
      v[i] = t;
    }
  }
}

// CG items: x = system, y/z = slice range of level 0, w unused. Rows are
// [srow[y], srow[z]).

// Ap = A p and the per-item partials of p . Ap (R values per item).
template <int R>
__global__ void __launch_bounds__(256) bcg_spmv_pap_kernel(SellView<double> A, const BItem *__restrict__ items,
                                                           int nitems, const Rv<double, R> *p,
                                                           Rv<double, R> *__restrict__ ap,
                                                           const int *__restrict__ sys_done,
                                                           double *__restrict__ partials) {
  __shared__ double smem[32 * R];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  bpass_entry();
  p = after_wait(p);
  for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
    const BItem q = items[it];
    if (item_skipped(sys_done, q.x)) continue;
    double acc[R];
#pragma unroll
    for (int j = 0; j < R; ++j) acc[j] = 0.0;
    for (int s = q.y + warp; s < q.z; s += nw) {
      Rv<double, R> sum = bsell_offdiag<double, R, false>(A, s, lane, p, 0);
      const int row = A.srow[s] + lane;
      if (row < A.srow[s + 1]) {
        const Rv<double, R> pr = p[row];
        fma_rv<double, R>(A.diag[row], pr, sum);
        ap[row] = sum;
#pragma unroll
        for (int j = 0; j < R; ++j) acc[j] = fma(pr.v[j], sum.v[j], acc[j]);
      }
    }
    bblock_sum<R>(acc, smem);
    if (threadIdx.x == 0)
#pragma unroll
      for (int j = 0; j < R; ++j) partials[static_cast<size_t>(it) * R + j] = acc[j];
  }
}

// x += alpha p, r -= alpha Ap for running pairs; partials of r . r.
template <int R>
__global__ void __launch_bounds__(256) bcg_update_xr_kernel(const int *__restrict__ srow,
                                                            const BItem *__restrict__ items, int nitems,
                                                            Rv<double, R> *__restrict__ x,
                                                            Rv<double, R> *__restrict__ r,
                                                            const Rv<double, R> *p,
                                                            const Rv<double, R> *ap,
                                                            const BPair *__restrict__ pairs,
                                                            const int *__restrict__ sys_done,
                                                            double *__restrict__ partials) {
  __shared__ double smem[32 * R];
  bpass_entry();
  for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
    const BItem q = items[it];
    if (item_skipped(sys_done, q.x)) continue;
    double alpha[R];
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const BPair &pr = pairs[q.x * R + j];
      alpha[j] = pr.done ? 0.0 : pr.alpha;
    }
    double acc[R];
#pragma unroll
    for (int j = 0; j < R; ++j) acc[j] = 0.0;
    const int r1 = srow[q.z];
    for (int i = srow[q.y] + threadIdx.x; i < r1; i += blockDim.x) {
      Rv<double, R> xi = x[i], ri = r[i];
      const Rv<double, R> pi = p[i], api = ap[i];
#pragma unroll
      for (int j = 0; j < R; ++j) {
        if (alpha[j] != 0.0) {
          xi.v[j] = fma(alpha[j], pi.v[j], xi.v[j]);
          ri.v[j] = fma(-alpha[j], api.v[j], ri.v[j]);
        }
        acc[j] = fma(ri.v[j], ri.v[j], acc[j]);
      }
      x[i] = xi;
      r[i] = ri;
    }
    bblock_sum<R>(acc, smem);
    if (threadIdx.x == 0)
#pragma unroll
      for (int j = 0; j < R; ++j) partials[static_cast<size_t>(it) * R + j] = acc[j];
  }
}

// Partials of r . z and (flexible) r . z_old: 2R values per item.
template <typename ZT, int R>
__global__ void __launch_bounds__(256) bcg_dot_rz_kernel(const int *__restrict__ srow,
                                                         const BItem *__restrict__ items, int nitems,
                                                         const Rv<double, R> *r,
                                                         const Rv<ZT, R> *z,
                                                         const Rv<ZT, R> *z_old,
                                                         const int *__restrict__ sys_done,
                                                         double *__restrict__ partials) {
  __shared__ double smem[32 * 2 * R];
  const bool flex = z_old != nullptr;
  bpass_entry();
  for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
    const BItem q = items[it];
    if (item_skipped(sys_done, q.x)) continue;
    double acc[2 * R];
#pragma unroll
    for (int j = 0; j < 2 * R; ++j) acc[j] = 0.0;
    const int r1 = srow[q.z];
    for (int i = srow[q.y] + threadIdx.x; i < r1; i += blockDim.x) {
      const Rv<double, R> ri = r[i];
      const Rv<ZT, R> zi = z[i];
#pragma unroll
      for (int j = 0; j < R; ++j) acc[j] = fma(ri.v[j], double(zi.v[j]), acc[j]);
      if (flex) {
        const Rv<ZT, R> zo = z_old[i];
#pragma unroll
        for (int j = 0; j < R; ++j) acc[R + j] = fma(ri.v[j], double(zo.v[j]), acc[R + j]);
      }
    }
    bblock_sum<2 * R>(acc, smem);
    if (threadIdx.x == 0)
#pragma unroll
      for (int j = 0; j < 2 * R; ++j) partials[static_cast<size_t>(it) * 2 * R + j] = acc[j];
  }
}

// p = z + beta p for running pairs.
template <typename ZT, int R>
__global__ void __launch_bounds__(256) bcg_update_p_kernel(const int *__restrict__ srow,
                                                           const BItem *__restrict__ items, int nitems,
                                                           const Rv<ZT, R> *z,
                                                           Rv<double, R> *__restrict__ p,
                                                           const BPair *__restrict__ pairs,
                                                           const int *__restrict__ sys_done) {
  bpass_entry();
  for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
    const BItem q = items[it];
    if (item_skipped(sys_done, q.x)) continue;
    double beta[R];
    bool run[R];
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const BPair &pr = pairs[q.x * R + j];
      run[j] = pr.done == 0;
      beta[j] = pr.beta;
    }
    const int r1 = srow[q.z];
    for (int i = srow[q.y] + threadIdx.x; i < r1; i += blockDim.x) {
      const Rv<ZT, R> zi = z[i];
      Rv<double, R> pi = p[i];
#pragma unroll
      for (int j = 0; j < R; ++j)
        if (run[j]) pi.v[j] = fma(beta[j], pi.v[j], double(zi.v[j]));
      p[i] = pi;
    }
  }
}

// Start of the solve: p = z; partials of b . b, r . z, r . r (3R per item).
template <typename ZT, int R>
__global__ void __launch_bounds__(256) bcg_init_kernel(const int *__restrict__ srow,
                                                       const BItem *__restrict__ items, int nitems,
                                                       const Rv<double, R> *b,
                                                       const Rv<double, R> *r,
                                                       const Rv<ZT, R> *z,
                                                       Rv<double, R> *__restrict__ p,
                                                       double *__restrict__ partials) {
  __shared__ double smem[32 * 3 * R];
  bpass_entry();
  for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
    const BItem q = items[it];
    double acc[3 * R];
#pragma unroll
    for (int j = 0; j < 3 * R; ++j) acc[j] = 0.0;
    const int r1 = srow[q.z];
    for (int i = srow[q.y] + threadIdx.x; i < r1; i += blockDim.x) {
      const Rv<double, R> bi = b[i], ri = r[i];
      const Rv<ZT, R> zi = z[i];
      Rv<double, R> pi;
#pragma unroll
      for (int j = 0; j < R; ++j) {
        const double zj = double(zi.v[j]);
        pi.v[j] = zj;
        acc[j] = fma(bi.v[j], bi.v[j], acc[j]);
        acc[R + j] = fma(ri.v[j], zj, acc[R + j]);
        acc[2 * R + j] = fma(ri.v[j], ri.v[j], acc[2 * R + j]);
      }
      p[i] = pi;
    }
    bblock_sum<3 * R>(acc, smem);
    if (threadIdx.x == 0)
#pragma unroll
      for (int j = 0; j < 3 * R; ++j) partials[static_cast<size_t>(it) * 3 * R + j] = acc[j];
  }
}

// Sum of one system's item partials (stride kN per item, component i), in a
// fixed order: lane-strided over the items, then a fixed shuffle tree.
template <int kN>
__device__ __forceinline__ double sum_items(const double *partials, int i0, int i1, int comp, int lane) {
  double t = 0.0;
#pragma unroll 8
  for (int i = i0 + lane; i < i1; i += 32) t += partials[static_cast<size_t>(i) * kN + comp];
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  return t;
}

// Finalize kernels: one block of 32*R threads per system, warp j handles the
// pair (system, j). The last system past a convergence test tells the host
// through two words of pinned memory: twice the number of tests so far, plus
// one once nothing is left to run; and whether a cluster step's wait gave up.
// That is ahead of the V-cycle, so the host queues the next iteration while the
// V-cycle runs, and none after the last one. Measured (one B200), with the
// kernels overlapping their launches: 5 systems of 14^3 to 30^3, issued
// launch by launch, 176 -> 159 us an iteration; 12 systems of 16^3 to 56^3 with
// 4 right-hand sides, graph replay, 550 -> 535 us.
enum BFinal : int { kBFinInit = 0, kBFinPap = 1, kBFinXr = 2, kBFinRz = 3 };

template <int R, int kWhich>
__global__ void __launch_bounds__(128) bcg_finalize_kernel(const int *__restrict__ item_first,
                                                           const double *partials,
                                                           BPair *__restrict__ pairs, int *__restrict__ sys_done,
                                                           BCgShared *__restrict__ sh,
                                                           volatile unsigned *host) {
  const int s = blockIdx.x, j = threadIdx.x >> 5, lane = threadIdx.x & 31;
  bpass_entry();
  if (kWhich == kBFinPap && s == 0 && threadIdx.x == 0) sh->active = 0;
  __shared__ int any_running;
  if (threadIdx.x == 0) any_running = 0;
  __syncthreads();
  const bool skip = kWhich != kBFinInit && sys_done[s] != 0;
  if (!skip) {
    const int i0 = item_first[s], i1 = item_first[s + 1];
    BPair &P = pairs[s * R + j];
    if (kWhich == kBFinInit) {
      const double bb = sum_items<3 * R>(partials, i0, i1, j, lane);
      const double rz = sum_items<3 * R>(partials, i0, i1, R + j, lane);
      const double rr = sum_items<3 * R>(partials, i0, i1, 2 * R + j, lane);
      if (lane == 0) {
        P.bb = bb;
        P.rho = rz;
        P.rr = rr;
        P.ratio = rr / bb;
        P.iter = 0;
        P.iterations = 0;
        P.alpha = P.beta = P.pAp = 0.0;
        P.done = 0;
        P.status = kCgRunning;
        if (!(sqrt(bb) >= 1e-12)) {
          // CGSolver::solve: a zero right-hand side returns x = 0
          P.status = isfinite(bb) ? kCgZeroRhs : kCgNotFinite;
          P.done = 1;
        } else if (!isfinite(P.ratio)) {
          P.status = kCgNotFinite;
          P.done = 1;
        } else if (P.ratio < sh->tol2) {
          P.status = kCgInitialConverged;
          P.done = 1;
        }
        if (!P.done) atomicOr(&any_running, 1);
      }
    } else if (kWhich == kBFinPap) {
      const double pap = sum_items<R>(partials, i0, i1, j, lane);
      if (lane == 0 && !P.done) {
        P.pAp = pap;
        if (!isfinite(pap) || pap == 0.0) {
          P.status = pap == 0.0 ? kCgBreakdown : kCgNotFinite;
          P.done = 1;
          P.iterations = P.iter;
          P.alpha = 0.0;
        } else {
          P.alpha = P.rho / pap;
        }
      }
    } else if (kWhich == kBFinXr) {
      const double rr = sum_items<R>(partials, i0, i1, j, lane);
      if (lane == 0 && !P.done) {
        P.rr = rr;
        const double ratio = rr / P.bb;
        P.ratio = ratio;
        if (!isfinite(ratio)) {
          P.status = kCgNotFinite;
          P.done = 1;
          P.iterations = P.iter;
        } else if (ratio < sh->tol2) {
          P.status = kCgConverged;
          P.done = 1;
          P.iterations = P.iter;  // 0-based, as the reference counts
        } else if (P.iter + 1 >= sh->max_iter) {
          P.status = kCgMaxIter;
          P.done = 1;
          P.iterations = sh->max_iter;
        }
        P.iter += 1;
      }
      if (lane == 0 && !P.done) atomicOr(&any_running, 1);
    } else {  // kBFinRz
      const double rz = sum_items<2 * R>(partials, i0, i1, j, lane);
      const double rzo = sum_items<2 * R>(partials, i0, i1, R + j, lane);
      if (lane == 0 && !P.done) {
        P.beta = (sh->flexible ? (rz - rzo) : rz) / P.rho;
        P.rho = rz;
      }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0 && (kWhich == kBFinInit || kWhich == kBFinXr) && !skip) {
    sys_done[s] = any_running ? 0 : 1;
    if (any_running) atomicAdd(&sh->active, 1);
  }
  if (kWhich == kBFinXr && threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&sh->arrived, 1) == static_cast<int>(gridDim.x) - 1) {
      sh->arrived = 0;
      const int tests = sh->tests + 1;
      sh->tests = tests;
      const bool fault = *reinterpret_cast<volatile int *>(&sh->sync_fault) != 0;
      if (fault) host[1] = 1u;
      __threadfence_system();
      host[0] = 2u * static_cast<unsigned>(tests) | (fault || atomicAdd(&sh->active, 0) == 0 ? 1u : 0u);
    }
  }
}

// ---- caller layout <-> internal layout ------------------------------------
// Caller: system s occupies [uoff[s], uoff[s] + nrhs * n[s]), right-hand side
// j of s at uoff[s] + j * n[s], rows in the caller's order. Internal: row
// q0[qoff[s] + i] + off0[s] of level 0, R values per row; columns j >= nrhs
// are set to zero. blockIdx.y = system.
template <int R>
__global__ void bscatter_kernel(const long long *__restrict__ uoff, const int *__restrict__ n,
                                const int *__restrict__ off0, const long long *__restrict__ qoff,
                                const int *__restrict__ q0, int nrhs, const double *__restrict__ in,
                                Rv<double, R> *__restrict__ out) {
  const int s = blockIdx.y, ns = n[s];
  const double *src = in + uoff[s];
  const int *q = q0 + qoff[s];
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ns; i += gridDim.x * blockDim.x) {
    Rv<double, R> v;
#pragma unroll
    for (int j = 0; j < R; ++j) v.v[j] = j < nrhs ? src[static_cast<size_t>(j) * ns + i] : 0.0;
    out[off0[s] + q[i]] = v;
  }
}

// Inverse of bscatter_kernel; pairs that ended with a zero right-hand side
// return x = 0.
template <int R>
__global__ void bgather_kernel(const long long *__restrict__ uoff, const int *__restrict__ n,
                               const int *__restrict__ off0, const long long *__restrict__ qoff,
                               const int *__restrict__ q0, int nrhs, const Rv<double, R> *__restrict__ in,
                               const BPair *__restrict__ pairs, double *__restrict__ out) {
  const int s = blockIdx.y, ns = n[s];
  double *dst = out + uoff[s];
  const int *q = q0 + qoff[s];
  bool zero[R];
#pragma unroll
  for (int j = 0; j < R; ++j) zero[j] = pairs[s * R + j].status == kCgZeroRhs;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ns; i += gridDim.x * blockDim.x) {
    const Rv<double, R> v = in[off0[s] + q[i]];
#pragma unroll
    for (int j = 0; j < R; ++j)
      if (j < nrhs) dst[static_cast<size_t>(j) * ns + i] = zero[j] ? 0.0 : v.v[j];
  }
}

}  // namespace gsb
