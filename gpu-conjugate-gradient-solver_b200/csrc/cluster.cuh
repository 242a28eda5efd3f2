// Whole Gauss-Seidel smoothing steps of a small level in one thread-block
// cluster, the iterate in distributed shared memory.
//
// What bounds such a level. A multicolour sweep is one dependent step per
// colour, and a Galerkin level of a few thousand rows has 15-45 colours of a
// few hundred rows: launched one kernel per colour, a pass is one or two
// blocks whose warps wait on row pointer -> column -> gather -> store -> next
// launch, about 3 us a pass with the GPU idle (ncu: 0.1 % of DRAM, 8-11 % of
// the warps of the SMs in use). Here the step is latency only:
//   * one cluster of up to 16 CTAs owns the level. Each colour's rows are cut
//     into one contiguous piece per CTA, and a CTA keeps in shared memory the
//     entries of x that its rows own or read ("slots", numbered per CTA);
//   * the thread group that updates a row sends the new value straight into
//     the slots of every CTA that reads it (st.async), which also counts the
//     bytes on that CTA's mbarrier of the pass: there is one mbarrier per
//     pass, armed once with the bytes the CTA will receive, so a CTA starts
//     pass p + 1 as soon as the values it reads have arrived: one one-way
//     message, no barrier round trip;
//   * the matrix is stored in the order in which each CTA's threads read it
//     (values and 16-bit slot numbers, slot pairs, threads contiguous), and
//     every thread loads its next row's operands before it waits.
// Measured (one B200, FP64, level 2 of a 61 x 47 x 83 Poisson: 5,103 rows, 37
// colours, 361 k entries): a symmetric step of 73 passes 183 -> 71 us, 0.84 us
// a pass, of which 0.74 us are there with next to no rows. A pass is bound by
// the instructions between two messages (clock: loads issued 360 cycles, wait
// 190, gathers, sums and shuffles 640, quotient 190, messages 300), not by the
// message, so the operands of the next row stay in place (two units change
// roles from pass to pass) and the way to the messages has no branch.
//
// No race. Row j of colour c' is overwritten in CTA B's slots only after the
// owner A of j has waited for every earlier pass of the sweep, and A receives
// every row i that reads j (checked when the layout is built): B's read of j
// for i happened before B sent i. A weighted update also reads the row's own
// slot, in every lane of its group, before any lane sends. Two writes of one row to one slot are
// separated by a direction change or a step's end, where every CTA first
// waits for all its passes and then meets the others at the cluster barrier,
// so the earlier write has landed. Rows of one colour do not read each other
// (or, on a level whose colouring is of the strong couplings only, read the
// copy of x taken where the sweep starts: slot numbers past the zero slot).
// All CTAs meet at the cluster barrier before any of them exits.
//
// Each row is updated with the arithmetic of csrv_gs_kernel with the same
// lanes per row (bsrv_gs_kernel for 3x3 blocks): same sums in the same order,
// same shuffles, same division, so the iterates are the same bits.
//
// Waits on mbarriers are bounded: a wait that gives up records
// CgState::sync_fault and stops the solve; the kernel then runs to its end
// without waiting, sends all its messages, and before it leaves waits (bounded
// as well) for those that are on their way to it.
#pragma once

#include "bulk.cuh"
#include "kernels.cuh"

namespace gsb {

constexpr int kClusterThreads = 512;    // scalar levels
constexpr int kClusterBlockThreads = 256;  // 3x3 levels: two units of 18 block values a thread
constexpr int kClusterPairs = 4;        // slot pairs per lane loaded ahead
constexpr int kClusterBlocks = 2;       // 3x3 blocks per lane loaded ahead
constexpr int kClusterMaxPasses = 512;  // mbarriers
constexpr int kClusterMaxSlots = 32760; // two copies of the slots in 16 bits
constexpr int kClusterMaxColors = 128;
constexpr long long kClusterWaitClocks = 2000000000LL;  // about a second

// One CTA's piece of one colour.
struct __align__(16) ClusterSeg {
  int row0, rows;  // global rows [row0, row0 + rows) (nodes of a block level)
  int trips;       // rows per thread group, at least 1
  int base;        // first slot pair (block slot) of trip 0
  int pairs;       // slot pairs (block slots) per lane and trip
  int stride;      // threads that take part (a multiple of 32; 0: no rows)
  int sbase;       // first send entry
  int schunks;     // send entries per lane and trip
};

template <typename T>
struct ClusterView {
  int ncta, ncolors, threads;
  int max_slots;                               // slots of the widest CTA, without the zero slot
  const ClusterSeg *__restrict__ seg;          // [cta][colour]
  const unsigned *__restrict__ expect;         // [cta][colour]: rows of the colour that the CTA receives
  const int *__restrict__ slot_ptr;            // ncta + 1
  const int *__restrict__ slot_row;            // global row of each slot
  const T *__restrict__ val;                   // slot pairs (scalar), or 9 per block slot, component-major
  const unsigned *__restrict__ col;            // two slots a pair; block slots: 16 bits each. + max_slots + 1: the
                                               // copy taken at the sweep's start
  const unsigned *__restrict__ send;           // cta << 16 | slot, or kNoSend
  const unsigned short *__restrict__ own;      // slot of each row in its owner
  const T *__restrict__ diag;                  // scalar: {d, 1 / d} per row, the latter 0 where it is not safe to
                                               // use; 3x3: the inverse diagonal block per node
  int relaxed;                                 // own-colour reads from the sweep's start
  long long wait_clocks;                       // bound of a wait
  int row0;                                    // first row of this system in the level's vectors (batches)
};

// No message. Its CTA and slot read 0, which every cluster has: the addresses
// are formed ahead of the test whether to send.
constexpr unsigned kNoSend = 0x80000000u;

// The passes of one call: dir 0 symmetric steps, 1 forward sweeps, 2
// backward sweeps; skip drops the colour repeated where a sweep turns.
struct ClusterPasses {
  int ncolors, steps, dir, skip;
  // sweep s of the call: its first colour, direction (+1 / -1) and passes
  __host__ __device__ int sweeps() const { return dir == 0 ? 2 * steps : steps; }
  __host__ __device__ int direction(int s) const { return dir == 1 || (dir == 0 && (s & 1) == 0) ? 1 : -1; }
  __host__ __device__ int first(int s) const {
    const int drop = dir == 0 && skip != 0 && s > 0 ? 1 : 0;
    return direction(s) > 0 ? drop : ncolors - 1 - drop;
  }
  __host__ __device__ int count(int s) const { return ncolors - (dir == 0 && skip != 0 && s > 0 ? 1 : 0); }
  __host__ __device__ int total() const {
    int t = 0;
    for (int s = 0; s < sweeps(); ++s) t += count(s);
    return t;
  }
};

namespace cluster_detail {

__device__ __forceinline__ unsigned cta_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ unsigned remote(unsigned addr, unsigned cta) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(cta));
  return r;
}
__device__ __forceinline__ void send_value(unsigned addr, double v, unsigned bar, bool on) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.u32 p, %3, 0;\n"
      " @p st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];\n}" ::"r"(addr),
      "l"(__double_as_longlong(v)), "r"(bar), "r"(static_cast<unsigned>(on))
      : "memory");
}
__device__ __forceinline__ void send_value(unsigned addr, float v, unsigned bar, bool on) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.u32 p, %3, 0;\n"
      " @p st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];\n}" ::"r"(addr),
      "r"(__float_as_uint(v)), "r"(bar), "r"(static_cast<unsigned>(on))
      : "memory");
}
// The W values of a row, if `on`: 16 bytes a message where they fill it.
template <typename T, int W>
__device__ __forceinline__ void send_row(unsigned addr, const T (&v)[W], unsigned bar, bool on) {
  if constexpr (W == 4 && sizeof(T) == 4) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.u32 p, %6, 0;\n"
        " @p st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];\n}" ::"r"(addr),
        "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])),
        "r"(__float_as_uint(v[3])), "r"(bar), "r"(static_cast<unsigned>(on))
        : "memory");
  } else if constexpr (W == 4) {
#pragma unroll
    for (int j = 0; j < 4; j += 2)
      asm volatile(
          "{\n .reg .pred p;\n setp.ne.u32 p, %4, 0;\n"
          " @p st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];\n}" ::"r"(addr + 8 * j),
          "l"(__double_as_longlong(v[j])), "l"(__double_as_longlong(v[j + 1])), "r"(bar), "r"(static_cast<unsigned>(on))
          : "memory");
  } else {
#pragma unroll
    for (int j = 0; j < W; ++j) send_value(addr + j * static_cast<unsigned>(sizeof(T)), v[j], bar, on);
  }
}

// Read-only loads that keep their place: the operands of the next row are
// requested before the wait on the current pass (a plain load is moved down to
// its first use, which exposes its latency: 770 of 3000 cycles a pass).
__device__ __forceinline__ double2 load_early(const double2 *p) {
  double2 v;
  asm volatile("ld.global.nc.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ float2 load_early(const float2 *p) {
  float2 v;
  asm volatile("ld.global.nc.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ double load_early(const double *p) {
  double v;
  asm volatile("ld.global.nc.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ float load_early(const float *p) {
  float v;
  asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ unsigned load_early(const unsigned *p) {
  unsigned v;
  asm volatile("ld.global.nc.u32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ unsigned short load_early(const unsigned short *p) {
  unsigned short v;
  asm volatile("ld.global.nc.u16 %0, [%1];" : "=h"(v) : "l"(p));
  return v;
}

// Whether the quotient q of an n and a d that has a reciprocal here is finite
// and large enough that the residuals n - q d have all their bits: |n| of at
// least 2^-969. Such a d is above 2^-500 (cluster_values), so n is above 2^-968
// when q is above 2^-468.
__device__ __forceinline__ bool full_residuals(double q) {
  constexpr unsigned lo = (1023u - 968u + 500u) << 20;
  return (static_cast<unsigned>(__double2hiint(q)) & 0x7fffffffu) - lo < 0x7ff00000u - lo;
}

// The quotients n / d of a row's R right-hand sides. FP64: from r = 1 / d, two
// residual corrections of n r (Markstein, IBM J. Res. Dev. 34, 1990), after
// which they are correctly rounded; the division (370 cycles on the critical
// path of every pass) where r is 0 (1 / d may not be a normal number; the result
// is 0 or NaN then), or n or the result is not finite or so small that a residual
// loses bits. Zeros need neither: a batch of two or three right-hand sides is
// padded with them (9 systems of 20^3 to 34^3, two right-hand sides, a sweep: 46
// us, 62 where zeros divide), and only there the test for them pays ahead of the
// branch. FP32: the division itself, which is as fast (two
// right-hand sides: 43 us either way).
template <typename T, int R>
__device__ __forceinline__ void quotients(const T (&n)[R], T d, T r, T (&q)[R]) {
  if constexpr (sizeof(T) == 4) {
#pragma unroll
    for (int j = 0; j < R; ++j) q[j] = n[j] / d;
  } else {
    bool exact = true;
#pragma unroll
    for (int j = 0; j < R; ++j) {
      q[j] = n[j] * r;
      q[j] = fma(fma(-q[j], d, n[j]), r, q[j]);
      q[j] = fma(fma(-q[j], d, n[j]), r, q[j]);
      exact = exact && (full_residuals(q[j]) || (R > 1 && n[j] == T(0)));
    }
    if (!exact) {
#pragma unroll
      for (int j = 0; j < R; ++j)
        if (!full_residuals(q[j]) && n[j] != T(0)) q[j] = n[j] / d;
    }
  }
}

// Bounded wait for the values of a pass (written by other CTAs: acquire at
// cluster scope); false after `clocks`.

__device__ __forceinline__ bool pass_ready(unsigned bar) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], 0;\n"
      " selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(bar)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool pass_wait(unsigned bar, long long clocks) {
  if (pass_ready(bar)) return true;
  const long long t0 = clock64();
  while (clock64() - t0 < clocks)
    if (pass_ready(bar)) return true;
  return false;
}
// After a wait gave up, ahead of the last cluster barrier: what is on its way
// to this CTA lands before it leaves. What is still missing after `clocks` in
// all was not sent.
__device__ __forceinline__ void drain_passes(unsigned bars, int npass, long long clocks) {
  const long long t0 = clock64();
  for (int p = 0; p < npass; ++p)
    while (!pass_ready(bars + 8 * p) && clock64() - t0 < clocks) {
    }
}

}  // namespace cluster_detail

// Rows of a scalar level with R right-hand sides, vectors row-interleaved
// ([row][R]): the arithmetic of csrv_gs_kernel (bcsrv_gs_kernel) with G lanes.
template <typename T, typename BT, int G, int R>
struct ClusterScalar {
  using V = T;
  using B = BT;
  static constexpr int kLanes = G, kW = R, kThreads = kClusterThreads;
  using P2 = typename Pair<T>::type;
  // what one thread needs of one row before the iterate
  struct Unit {
    P2 v[kClusterPairs];
    unsigned c[kClusterPairs];  // two slots
    unsigned send;
    P2 d;
    BT b[R];
  };

  static __device__ __forceinline__ void load(const ClusterView<T> &A, const ClusterSeg &sg, int t, int tid, int row,
                                              Unit &u) {
    using cluster_detail::load_early;
    const P2 *val = reinterpret_cast<const P2 *>(A.val);
    const int e0 = sg.base + t * sg.pairs * sg.stride + tid;
#pragma unroll
    for (int q = 0; q < kClusterPairs; ++q)
      if (q < sg.pairs) {
        u.v[q] = load_early(val + e0 + q * sg.stride);
        u.c[q] = load_early(A.col + e0 + q * sg.stride);
      }
    u.d = load_early(reinterpret_cast<const P2 *>(A.diag) + row);
  }
  static __device__ __forceinline__ void load_b(const BT *b, int row, Unit &u) {
    if constexpr (R == 4 && sizeof(BT) == 4) {
      const float2 *q = reinterpret_cast<const float2 *>(b) + 2 * static_cast<size_t>(row);
      const float2 lo = cluster_detail::load_early(q), hi = cluster_detail::load_early(q + 1);
      u.b[0] = lo.x, u.b[1] = lo.y, u.b[2] = hi.x, u.b[3] = hi.y;
    } else if constexpr (R == 4) {
      const double2 *q = reinterpret_cast<const double2 *>(b) + 2 * static_cast<size_t>(row);
      const double2 lo = cluster_detail::load_early(q), hi = cluster_detail::load_early(q + 1);
      u.b[0] = lo.x, u.b[1] = lo.y, u.b[2] = hi.x, u.b[3] = hi.y;
    } else {
#pragma unroll
      for (int j = 0; j < R; ++j) u.b[j] = cluster_detail::load_early(b + static_cast<size_t>(row) * R + j);
    }
  }
  static __device__ __forceinline__ void add(T v, const T *xs, unsigned slot, T (&sum)[R]) {
    if constexpr (R == 4 && sizeof(T) == 4) {
      const float4 q = *reinterpret_cast<const float4 *>(xs + 4 * slot);
      sum[0] = fma(v, q.x, sum[0]), sum[1] = fma(v, q.y, sum[1]);
      sum[2] = fma(v, q.z, sum[2]), sum[3] = fma(v, q.w, sum[3]);
    } else if constexpr (R == 4) {
      const double2 q0 = *reinterpret_cast<const double2 *>(xs + 4 * slot);
      const double2 q1 = *reinterpret_cast<const double2 *>(xs + 4 * slot + 2);
      sum[0] = fma(v, q0.x, sum[0]), sum[1] = fma(v, q0.y, sum[1]);
      sum[2] = fma(v, q1.x, sum[2]), sum[3] = fma(v, q1.y, sum[3]);
    } else {
#pragma unroll
      for (int j = 0; j < R; ++j) sum[j] = fma(v, xs[slot * R + j], sum[j]);
    }
  }
  // neighbour sums of the row (in every lane of its group)
  static __device__ __forceinline__ void sums(const ClusterView<T> &A, const ClusterSeg &sg, int t, int tid,
                                              const T *xs, const Unit &u, T (&sum)[R]) {
#pragma unroll
    for (int j = 0; j < R; ++j) sum[j] = T(0);
#pragma unroll
    for (int q = 0; q < kClusterPairs; ++q)
      if (q < sg.pairs) {
        add(u.v[q].x, xs, u.c[q] & 0xffffu, sum);
        add(u.v[q].y, xs, u.c[q] >> 16, sum);
      }
    if (sg.pairs > kClusterPairs) {
      const int e0 = sg.base + t * sg.pairs * sg.stride + tid;
#pragma unroll 4
      for (int q = kClusterPairs; q < sg.pairs; ++q) {
        const P2 v = __ldg(reinterpret_cast<const P2 *>(A.val) + e0 + q * sg.stride);
        const unsigned c = __ldg(A.col + e0 + q * sg.stride);
        add(v.x, xs, c & 0xffffu, sum);
        add(v.y, xs, c >> 16, sum);
      }
    }
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1)
#pragma unroll
      for (int j = 0; j < R; ++j) sum[j] += __shfl_xor_sync(0xffffffffu, sum[j], o, G);
  }
  static __device__ __forceinline__ void update(const Unit &u, const T (&sum)[R], T (&xn)[R]) {
    T n[R];
#pragma unroll
    for (int j = 0; j < R; ++j) n[j] = T(u.b[j]) - sum[j];
    cluster_detail::quotients(n, u.d.x, u.d.y, xn);
  }
};

// Node rows of a 3x3 level: the arithmetic of bsrv_gs_kernel with G lanes.
template <typename T, typename BT, int G>
struct ClusterBlock {
  using V = T;
  using B = BT;
  static constexpr int kLanes = G, kW = 3, kThreads = kClusterBlockThreads;
  struct Unit {
    T v[kClusterBlocks][9];
    unsigned short c[kClusterBlocks];
    unsigned send;
    T d[9];
    BT b[3];
  };

  static __device__ __forceinline__ void load(const ClusterView<T> &A, const ClusterSeg &sg, int t, int tid, int row,
                                              Unit &u) {
    using cluster_detail::load_early;
    const unsigned short *col = reinterpret_cast<const unsigned short *>(A.col);
#pragma unroll
    for (int q = 0; q < kClusterBlocks; ++q)
      if (q < sg.pairs) {
        const int e = t * sg.pairs + q;
        u.c[q] = load_early(col + sg.base + e * sg.stride + tid);
#pragma unroll
        for (int k = 0; k < 9; ++k) u.v[q][k] = load_early(A.val + 9 * sg.base + (9 * e + k) * sg.stride + tid);
      }
#pragma unroll
    for (int k = 0; k < 9; ++k) u.d[k] = load_early(A.diag + 9 * static_cast<size_t>(row) + k);
  }
  static __device__ __forceinline__ void load_b(const BT *b, int row, Unit &u) {
#pragma unroll
    for (int j = 0; j < 3; ++j) u.b[j] = cluster_detail::load_early(b + 3 * static_cast<size_t>(row) + j);
  }
  static __device__ __forceinline__ void add(const T (&v)[9], const T *x, T (&sum)[3]) {
    const T x0 = x[0], x1 = x[1], x2 = x[2];
#pragma unroll
    for (int r = 0; r < 3; ++r) sum[r] = fma(v[3 * r], x0, fma(v[3 * r + 1], x1, fma(v[3 * r + 2], x2, sum[r])));
  }
  static __device__ __forceinline__ void sums(const ClusterView<T> &A, const ClusterSeg &sg, int t, int tid,
                                              const T *xs, const Unit &u, T (&sum)[3]) {
    sum[0] = sum[1] = sum[2] = T(0);
#pragma unroll
    for (int q = 0; q < kClusterBlocks; ++q)
      if (q < sg.pairs) add(u.v[q], xs + 3 * static_cast<unsigned>(u.c[q]), sum);
    const unsigned short *col = reinterpret_cast<const unsigned short *>(A.col);
#pragma unroll 2
    for (int q = kClusterBlocks; q < sg.pairs; ++q) {
      const int e = t * sg.pairs + q;
      T v[9];
#pragma unroll
      for (int k = 0; k < 9; ++k) v[k] = __ldg(A.val + 9 * sg.base + (9 * e + k) * sg.stride + tid);
      add(v, xs + 3 * static_cast<unsigned>(__ldg(col + sg.base + e * sg.stride + tid)), sum);
    }
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1)
#pragma unroll
      for (int r = 0; r < 3; ++r) sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], o, G);
  }
  static __device__ __forceinline__ void update(const Unit &u, const T (&sum)[3], T (&xn)[3]) {
    const T r0 = T(u.b[0]) - sum[0], r1 = T(u.b[1]) - sum[1], r2 = T(u.b[2]) - sum[2];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      T nv = u.d[3 * r] * r0;
      nv = fma(u.d[3 * r + 1], r1, nv);
      xn[r] = fma(u.d[3 * r + 2], r2, nv);
    }
  }
};

// Where a launch reads its stop flag and records a fault.
struct ClusterStatus {
  int *stop;   // nonzero: nothing to do
  int *fault;  // set when a wait gave up (and *stop with it)
};

// Smoothing steps of the level (or, in a batch, of one system of the level)
// that A describes; called by every thread of its cluster.
template <typename Row>
__device__ __forceinline__ void cluster_steps(const ClusterView<typename Row::V> &A, const ClusterPasses &P,
                                              const typename Row::B *__restrict__ b, typename Row::V *__restrict__ x,
                                              int zero, const typename Row::V *__restrict__ wts,
                                              const typename Row::V *__restrict__ nw, typename Row::V omega,
                                              ClusterStatus status) {
  using namespace cluster_detail;
  using T = typename Row::V;
  constexpr int W = Row::kW, G = Row::kLanes;
  extern __shared__ __align__(16) unsigned char cluster_smem[];
  __shared__ ClusterSeg seg[kClusterMaxColors];
  __shared__ unsigned long long bars[kClusterMaxPasses];
  // colour of each pass, bit 15 on the last one of a sweep; 0xffff at the end
  __shared__ unsigned short plist[kClusterMaxPasses + 1];
  // max_slots + 1 slots of W values, the last one zero (then the sweep's start)
  T *xs = reinterpret_cast<T *>(cluster_smem);
  const int tid = threadIdx.x, nthr = A.threads;
  const unsigned me = cta_rank();
  const int s0 = __ldg(A.slot_ptr + me), nslots = __ldg(A.slot_ptr + me + 1) - s0;
  T *xp = xs + (A.max_slots + 1) * W;
  for (int c = tid; c < A.ncolors; c += nthr) seg[c] = A.seg[me * A.ncolors + c];
  const int npass = P.total();
  for (int p = tid; p < npass; p += nthr)
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(bars + p)) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  __syncthreads();
  // arm every pass once with the bytes this CTA receives in it
  for (int s = 0, p = 0; s < P.sweeps(); ++s) {
    const int n = P.count(s), f = P.first(s), dr = P.direction(s);
    for (int i = tid; i < n; i += nthr) {
      const int c = f + dr * i;
      mbar_expect_tx(bars + p + i, __ldg(A.expect + me * A.ncolors + c) * static_cast<unsigned>(W * sizeof(T)));
      plist[p + i] = static_cast<unsigned short>(c | (i + 1 == n ? 0x8000 : 0));
    }
    p += n;
  }
  if (tid == 0) plist[npass] = 0xffff;
  __syncthreads();
  // the first row's matrix operands do not change during a solve
  constexpr int kLog = G == 4 ? 2 : (G == 8 ? 3 : (G == 16 ? 4 : 5));
  const int grp = tid >> kLog, groups = nthr >> kLog;
  typename Row::Unit unit0, unit1;
  unit0.send = unit1.send = kNoSend;  // threads without a row
  unsigned code = plist[0];
  ClusterSeg sg = seg[code & 0x7fffu];
  if (tid < sg.stride) {
    Row::load(A, sg, 0, tid, sg.row0 + min(grp, sg.rows - 1), unit0);
    unit0.send = load_early(A.send + sg.sbase + tid);
  }
  const bool stop = pass_entry(status.stop);  // the same in every CTA: only a finished kernel writes it
  if (!stop) {
    if (tid < sg.stride) Row::load_b(b, sg.row0 + min(grp, sg.rows - 1), unit0);
    for (int i = tid; i < (A.max_slots + 1) * W; i += nthr) {
      const int slot = i / W;
      const T v = zero || slot >= nslots ? T(0) : x[static_cast<size_t>(__ldg(A.slot_row + s0 + slot)) * W + i % W];
      xs[i] = v;
      if (A.relaxed) xp[i] = v;
    }
  }
  cluster_barrier();
  if (stop) return;
  const unsigned xs_addr = smem_addr(xs), bar_addr = smem_addr(bars);
  // passes from here on write x back to the level (the last step's)
  const int keep = npass - (P.dir == 0 ? P.count(P.sweeps() - 1) + P.count(P.sweeps() - 2) : A.ncolors);
  int p = 0, t = 0;
  bool fresh = true, dead = false;  // first pass of a sweep; a wait gave up
  const bool weighted = nw != nullptr || wts != nullptr || omega != T(1);
  // One unit (a trip of a pass) from `cur`, the next one's operands into
  // `nxt`; true at the end. The two change places from call to call: moved
  // instead, the operands would have to arrive a unit early.
  const auto step = [&](typename Row::Unit &cur, typename Row::Unit &nxt) __attribute__((always_inline)) {
    // the next unit's operands, before this one waits
    const bool last_trip = t + 1 == sg.trips;
    const int tn = last_trip ? 0 : t + 1;
    const unsigned next_code = plist[last_trip ? p + 1 : p];
    ClusterSeg sn;
    sn.stride = 0;
    nxt.send = kNoSend;
    if (next_code != 0xffffu) {
      sn = seg[next_code & 0x7fffu];
      if (tid < sn.stride) {
        const int row = sn.row0 + min(tn * groups + grp, sn.rows - 1);
        Row::load(A, sn, tn, tid, row, nxt);
        nxt.send = load_early(A.send + sn.sbase + tn * sn.schunks * sn.stride + tid);
        Row::load_b(b, row, nxt);
      }
    }
    const unsigned to_cta = (cur.send >> 16) & 15u;
    const unsigned to_x = remote(xs_addr + static_cast<unsigned>(W * sizeof(T)) * (cur.send & 0xffffu), to_cta);
    const unsigned to_bar = remote(bar_addr + 8 * p, to_cta);
    if (t == 0 && !fresh && !dead) dead = !pass_wait(bar_addr + 8 * (p - 1), A.wait_clocks);
    if (tid < sg.stride) {
      T sum[W], xn[W];
      Row::sums(A, sg, t, tid, xs, cur, sum);
      // lanes past the piece's rows compute along (their sums are zero and
      // they send nothing): no branch on the way to the messages
      Row::update(cur, sum, xn);
      const int local = t * groups + grp, row = sg.row0 + min(local, sg.rows - 1);
      if (weighted) {
        const T w = nw != nullptr ? __ldg(nw + row) : (wts != nullptr ? __ldg(wts + (code & 0x7fffu)) : omega);
        if (w != T(1)) {
          const unsigned own = W * __ldg(A.own + row);
#pragma unroll
          for (int j = 0; j < W; ++j) xn[j] = fma(T(1) - w, xs[own + j], w * xn[j]);
        }
        // every lane of a row has read its old value before one of them
        // sends the new one into the same slot
        __syncwarp();
      }
      send_row(to_x, xn, to_bar, cur.send != kNoSend);
      if (sg.schunks > 1)
        for (int q = 1; q < sg.schunks; ++q) {
          const unsigned to = __ldg(A.send + sg.sbase + (t * sg.schunks + q) * sg.stride + tid);
          send_row(remote(xs_addr + static_cast<unsigned>(W * sizeof(T)) * (to & 0xffffu), (to >> 16) & 15u), xn,
                   remote(bar_addr + 8 * p, (to >> 16) & 15u), to != kNoSend);
        }
      if (p >= keep && (tid & (G - 1)) == 0 && local < sg.rows)
#pragma unroll
        for (int j = 0; j < W; ++j) x[static_cast<size_t>(row) * W + j] = xn[j];
    }
    fresh = false;
    if (last_trip) {
      if (code & 0x8000u) {
        // every value of this sweep has arrived before the next one starts
        // (or before the CTAs leave)
        if (!dead) dead = !pass_wait(bar_addr + 8 * p, A.wait_clocks);
        if (next_code == 0xffffu) return true;
        if (A.relaxed) {
          __syncthreads();
          for (int k = tid; k < nslots * W; k += nthr) xp[k] = xs[k];
        }
        cluster_barrier();
        fresh = true;
      }
      ++p;
    }
    code = next_code;
    t = tn;
    sg = sn;
    return false;
  };
  for (;;) {
    if (step(unit0, unit1)) break;
    if (step(unit1, unit0)) break;
  }
  if (dead) drain_passes(bar_addr, npass, A.wait_clocks);
  cluster_barrier();
  if (dead) {
    *status.fault = kFaultCluster;
    *status.stop = 1;
  }
}

// Grid = one cluster of A.ncta CTAs. wts: per colour, nw: per node (or
// nullptr).
template <typename Row>
__global__ void __launch_bounds__(Row::kThreads, 1)
    cluster_gs_kernel(ClusterView<typename Row::V> A, ClusterPasses P, const typename Row::B *__restrict__ b,
                      typename Row::V *__restrict__ x, int zero, const typename Row::V *__restrict__ wts,
                      const typename Row::V *__restrict__ nw, typename Row::V omega, CgState *st) {
  cluster_steps<Row>(A, P, b, x, zero, wts, nw, omega, ClusterStatus{&st->done, &st->sync_fault});
}

// One cluster per system of a batch level: views[i] belongs to system
// systems[i], whose rows start at its row0 in b and x.
template <typename Row>
__global__ void __launch_bounds__(Row::kThreads, 1)
    cluster_gs_batch_kernel(const ClusterView<typename Row::V> *__restrict__ views, const int *__restrict__ systems,
                            int ncta, ClusterPasses P, const typename Row::B *__restrict__ b,
                            typename Row::V *__restrict__ x, int zero, typename Row::V omega, int *sys_done,
                            int *fault) {
  const int i = blockIdx.x / ncta;
  const ClusterView<typename Row::V> A = views[i];
  P.ncolors = A.ncolors;
  const size_t at = static_cast<size_t>(A.row0) * Row::kW;
  cluster_steps<Row>(A, P, b + at, x + at, zero, nullptr, nullptr, omega, ClusterStatus{sys_done + systems[i], fault});
}

}  // namespace gsb
