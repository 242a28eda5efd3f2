// Host construction of the cluster-resident smoothing layout (cluster.cuh):
// which CTA owns which rows, the slots of x each CTA keeps, the matrix in the
// order its threads read it, and where every updated row is sent.
#pragma once

#include <algorithm>
#include <cstring>
#include <mutex>
#include <type_traits>
#include <unordered_map>
#include <utility>
#include <vector>

#include "cluster.cuh"
#include "formats.cuh"
#include "solver.h"

namespace gsb {

// Where the layout has the off-diagonal entries of its matrix: what a refresh
// of the values needs.
struct ClusterEntries {
  std::vector<unsigned> at;          // entry e (scalar levels: rows in order; else blocks): its place in val
  std::vector<unsigned short> step;  // 3x3 levels: distance of the block's components
  BlockRows blocks;                  // 3x3 levels
};

template <typename T>
struct HostCluster {
  int ncta = 0, ncolors = 0, g = 0, threads = 0, max_slots = 0, relaxed = 0;
  long long wait_clocks = kClusterWaitClocks;
  std::vector<ClusterSeg> seg;
  std::vector<unsigned> expect;
  std::vector<int> slot_ptr, slot_row;
  std::vector<T> val;                // two per pair, or nine per block slot
  std::vector<unsigned short> col;   // two per pair, or one per block slot
  std::vector<unsigned> send;
  std::vector<unsigned short> own;
  std::vector<T> diag;               // scalar levels: {d, 1 / d} per row
  ClusterEntries entries;
};

// Rows [lo, hi) of colour piece q of ncta over [r0, r1).
inline int cluster_cut(int r0, int r1, int q, int ncta) {
  return r0 + static_cast<int>(static_cast<long long>(r1 - r0) * q / ncta);
}

// Layout of a level with n rows (or 3x3 nodes) in colour-contiguous order,
// colour c = rows [first[c], first[c + 1]), whose off-diagonal pattern is
// (rp, ci), columns ascending, for ncta CTAs of `threads` threads and g lanes
// per row: the k-th entry of a row goes to lane k % g, as the CSR-vector
// kernels read it, as that lane's entry k / g; `per` entries share a slot word
// (2 on scalar levels, 1 on 3x3 ones). The values are left zero, their places
// in h.entries. False when the level does not qualify: a CTA needs more than `slot_limit` slots, a single colour,
// too many colours, or a row is read by a row that its own owner does not
// read (the pattern is not structurally symmetric; see the race argument in
// cluster.cuh).
template <typename T>
bool cluster_build(int n, const std::vector<int> &rp, const std::vector<int> &ci, const std::vector<int> &first, int per,
                   int g, int ncta, int threads, bool relaxed, int slot_limit, HostCluster<T> &h) {
  const int nc = static_cast<int>(first.size()) - 1, values = per == 2 ? 2 : 9;  // values per slot word
  if (nc < 2 || nc > kClusterMaxColors || n < 1) return false;
  const int limit = std::min(slot_limit, kClusterMaxSlots);
  if (static_cast<long long>(n) > static_cast<long long>(limit) * ncta) return false;
  h.ncta = ncta, h.ncolors = nc, h.g = g, h.threads = threads, h.relaxed = relaxed ? 1 : 0;
  std::vector<unsigned char> owner(n);
  std::vector<int> colour(n);
  for (int c = 0; c < nc; ++c)
    for (int q = 0; q < ncta; ++q)
      for (int r = cluster_cut(first[c], first[c + 1], q, ncta); r < cluster_cut(first[c], first[c + 1], q + 1, ncta); ++r)
        owner[r] = static_cast<unsigned char>(q), colour[r] = c;
  // slots: the rows a CTA owns or reads, ascending
  std::vector<std::vector<int>> rows_of(ncta);
  std::vector<std::vector<unsigned short>> slot(ncta);
  const unsigned short none = 0xffff;
  std::vector<int> over(ncta, 0);
  parallel_for(ncta, [&](long long q0, long long q1) {
    for (long long q = q0; q < q1; ++q) {
      std::vector<unsigned char> need(n, 0);
      for (int c = 0; c < nc; ++c)
        for (int r = cluster_cut(first[c], first[c + 1], q, ncta); r < cluster_cut(first[c], first[c + 1], q + 1, ncta); ++r) {
          need[r] = 1;
          for (int k = rp[r]; k < rp[r + 1]; ++k) need[ci[k]] = 1;
        }
      slot[q].assign(n, none);
      for (int r = 0; r < n; ++r)
        if (need[r]) {
          if (static_cast<int>(rows_of[q].size()) >= limit) {
            over[q] = 1;
            break;
          }
          slot[q][r] = static_cast<unsigned short>(rows_of[q].size());
          rows_of[q].push_back(r);
        }
    }
  }, 1);
  for (int q = 0; q < ncta; ++q)
    if (over[q]) return false;
  h.max_slots = 0;
  h.slot_ptr.assign(1, 0);
  h.slot_row.clear();
  for (int q = 0; q < ncta; ++q) {
    h.max_slots = std::max(h.max_slots, static_cast<int>(rows_of[q].size()));
    h.slot_row.insert(h.slot_row.end(), rows_of[q].begin(), rows_of[q].end());
    h.slot_ptr.push_back(static_cast<int>(h.slot_row.size()));
  }
  const unsigned short zero_slot = static_cast<unsigned short>(h.max_slots);
  h.own.resize(n);
  for (int r = 0; r < n; ++r) h.own[r] = slot[owner[r]][r];
  // pieces: sizes and offsets
  const int groups = threads / g;
  h.seg.assign(static_cast<size_t>(ncta) * nc, ClusterSeg{});
  h.expect.assign(h.seg.size(), 0u);
  std::vector<unsigned> dests(n, 0);  // CTAs that keep row r
  for (int q = 0; q < ncta; ++q)
    for (int r : rows_of[q]) dests[r] |= 1u << q;
  long long words = 0, send_total = 0;
  std::vector<int> ok(ncta, 1);
  for (int q = 0; q < ncta; ++q)
    for (int c = 0; c < nc; ++c) {
      ClusterSeg &s = h.seg[static_cast<size_t>(q) * nc + c];
      s.row0 = cluster_cut(first[c], first[c + 1], q, ncta);
      s.rows = cluster_cut(first[c], first[c + 1], q + 1, ncta) - s.row0;
      int len = 0, deg = 1;
      for (int r = s.row0; r < s.row0 + s.rows; ++r) {
        len = std::max(len, rp[r + 1] - rp[r]);
        deg = std::max(deg, __builtin_popcount(dests[r]));
      }
      s.pairs = ((len + g - 1) / g + per - 1) / per;
      s.stride = std::min(threads, (s.rows * g + 31) / 32 * 32);
      s.schunks = (deg + g - 1) / g;
      const int trips = (s.rows + groups - 1) / groups;
      s.trips = std::max(1, trips);
      s.base = static_cast<int>(words);
      s.sbase = static_cast<int>(send_total);
      words += static_cast<long long>(trips) * s.pairs * s.stride;
      send_total += static_cast<long long>(trips) * s.schunks * s.stride;
      if (words * values > (1LL << 28) || send_total > (1LL << 28)) return false;  // 32-bit offsets in the kernel
      // rows of colour c among CTA q's slots
      const auto &rq = rows_of[q];
      h.expect[static_cast<size_t>(q) * nc + c] = static_cast<unsigned>(
          std::lower_bound(rq.begin(), rq.end(), first[c + 1]) - std::lower_bound(rq.begin(), rq.end(), first[c]));
    }
  if (cluster_message_withheld()) {  // tests: the wait for the first colour runs out
    ++h.expect[0];
    h.wait_clocks = 2000000;
  }
  h.val.assign(static_cast<size_t>(values) * words, T(0));
  h.entries.at.assign(ci.size(), 0u);
  if (per == 1) h.entries.step.assign(ci.size(), 0);
  h.col.assign(static_cast<size_t>(per) * words, zero_slot);
  h.send.assign(static_cast<size_t>(send_total), kNoSend);
  parallel_for(ncta, [&](long long q0, long long q1) {
    for (long long q = q0; q < q1; ++q)
      for (int c = 0; c < nc; ++c) {
        const ClusterSeg &s = h.seg[static_cast<size_t>(q) * nc + c];
        for (int i = 0; i < s.rows; ++i) {
          const int r = s.row0 + i, t = i / groups, lane0 = (i % groups) * g;
          for (int e = rp[r]; e < rp[r + 1]; ++e) {
            const int j = ci[e], k = e - rp[r], lane = lane0 + k % g, kk = k / g;
            unsigned short sl = slot[q][j];
            if (colour[j] == c) {
              if (!relaxed) ok[q] = 0;  // two coupled rows of one colour
              sl = static_cast<unsigned short>(sl + h.max_slots + 1);
            }
            if (slot[owner[j]][r] == none) ok[q] = 0;  // j's owner does not receive r
            const size_t word = static_cast<size_t>(t) * s.pairs + kk / per;  // of the lane, within the piece
            if (per == 2) {
              const size_t at = 2 * (s.base + word * s.stride + lane) + (kk & 1);
              h.col[at] = sl;
              h.entries.at[e] = static_cast<unsigned>(at);
            } else {
              h.col[s.base + word * s.stride + lane] = sl;
              h.entries.at[e] = static_cast<unsigned>(9 * static_cast<size_t>(s.base) + 9 * word * s.stride + lane);
              h.entries.step[e] = static_cast<unsigned short>(s.stride);
            }
          }
          int d = 0;
          for (int to = 0; to < ncta; ++to) {
            if ((dests[r] >> to & 1u) == 0) continue;
            h.send[s.sbase + (static_cast<size_t>(t) * s.schunks + d / g) * s.stride + lane0 + d % g] =
                static_cast<unsigned>(to) << 16 | slot[to][r];
            ++d;
          }
        }
      }
  }, 1);
  for (int q = 0; q < ncta; ++q)
    if (!ok[q]) return false;
  return true;
}

// First off-diagonal entry of each row.
inline std::vector<int> off_diagonal_rows(const Csr &a) {
  std::vector<int> rp(a.rows + 1, 0);
  parallel_for(a.rows, [&](long long r0, long long r1) {
    for (long long r = r0; r < r1; ++r)
      for (int k = a.rp[r]; k < a.rp[r + 1]; ++k) rp[r + 1] += a.ci[k] != r ? 1 : 0;
  }, row_grain(a.rows, a.nnz()));
  for (int r = 0; r < a.rows; ++r) rp[r + 1] += rp[r];
  return rp;
}

// The values of a scalar matrix in the layout, and {d, 1 / d} of every row; the
// reciprocal is 0 where d or 1 / d is too close to the ends of T's range for
// the kernel's quotient. False when the matrix is not the layout's.
template <typename T>
bool cluster_values(const Csr &a, const ClusterEntries &where, std::vector<T> &val, std::vector<T> &diag) {
  const std::vector<int> rp = off_diagonal_rows(a);
  if (static_cast<size_t>(rp[a.rows]) != where.at.size()) return false;
  const T big = sizeof(T) == 8 ? T(0x1p500) : T(0x1p60f);
  diag.assign(2 * static_cast<size_t>(a.rows), T(0));
  parallel_for(a.rows, [&](long long r0, long long r1) {
    for (long long r = r0; r < r1; ++r) {
      int e = rp[r];
      for (int k = a.rp[r]; k < a.rp[r + 1]; ++k) {
        if (a.ci[k] != r) {
          val[where.at[e++]] = T(a.v[k]);
          continue;
        }
        const T d = T(a.v[k]);
        diag[2 * r] = d;
        diag[2 * r + 1] = std::fabs(d) < big && std::fabs(d) > T(1) / big ? T(1) / d : T(0);
      }
    }
  }, row_grain(a.rows, a.nnz()));
  return true;
}

// The same for a 3x3-blocked matrix, whose inverse diagonal blocks are the
// level's own.
template <typename T>
bool cluster_block_values(const Csr &a, const ClusterEntries &where, std::vector<T> &val) {
  return for_block_entries(a, where.blocks,
                           [&](size_t e, int c, double v) { val[where.at[e] + static_cast<size_t>(c) * where.step[e]] = T(v); });
}

// The layout of a square scalar matrix (sorted columns).
template <typename T>
bool make_cluster(const Csr &a, const std::vector<int> &first, int g, int ncta, bool relaxed, int slot_limit,
                  HostCluster<T> &h) {
  const std::vector<int> rp = off_diagonal_rows(a);
  std::vector<int> ci(rp[a.rows]);
  parallel_for(a.rows, [&](long long r0, long long r1) {
    for (long long r = r0; r < r1; ++r) {
      int e = rp[r];
      for (int k = a.rp[r]; k < a.rp[r + 1]; ++k)
        if (a.ci[k] != r) ci[e++] = a.ci[k];
    }
  }, row_grain(a.rows, a.nnz()));
  return cluster_build<T>(a.rows, rp, ci, first, 2, g, ncta, kClusterThreads, relaxed, slot_limit, h) &&
         cluster_values<T>(a, h.entries, h.val, h.diag);
}

// The layout of a 3x3-blocked matrix, `first` in nodes; the inverse diagonal
// blocks stay where the level has them (upload_cluster).
template <typename T>
bool make_cluster_blocks(const Csr &a, const std::vector<int> &first, int g, int ncta, bool relaxed, int slot_limit,
                         HostCluster<T> &h) {
  h.entries.blocks = block_rows(a);
  return cluster_build<T>(a.rows / 3, h.entries.blocks.rp, h.entries.blocks.ci, first, 1, g, ncta, kClusterBlockThreads,
                          relaxed, slot_limit, h) &&
         cluster_block_values<T>(a, h.entries, h.val);
}

template <typename T>
struct DevCluster {
  int g = 0, ncta = 0, threads = 0, max_slots = 0;
  T *val = nullptr, *diag = nullptr;  // what a value refresh overwrites
  size_t values = 0;
  ClusterEntries entries;  // kept by levels whose values can be refreshed
  ClusterView<T> v{};
  // dynamic shared memory of a CTA, `width` values a slot
  size_t smem(int width) const {
    return (static_cast<size_t>(max_slots) + 1) * width * sizeof(T) * (v.relaxed ? 2 : 1);
  }
};

// `diag`: the level's inverse diagonal blocks (3x3 levels), else nullptr.
template <typename T>
DevCluster<T> upload_cluster(Arena &ar, const HostCluster<T> &h, const T *diag, int row0 = 0) {
  DevCluster<T> d;
  d.g = h.g, d.ncta = h.ncta, d.threads = h.threads, d.max_slots = h.max_slots;
  d.values = h.val.size();
  d.v.ncta = h.ncta, d.v.ncolors = h.ncolors, d.v.threads = h.threads, d.v.max_slots = h.max_slots;
  d.v.relaxed = h.relaxed;
  d.v.wait_clocks = h.wait_clocks;
  d.v.row0 = row0;
  // the values, and one allocation and one copy for the rest of the layout
  std::vector<unsigned char> pack;
  const auto put = [&](const auto &v) {
    const size_t at = (pack.size() + 255) / 256 * 256;
    pack.resize(at + sizeof(v[0]) * v.size());
    if (!v.empty()) std::memcpy(pack.data() + at, v.data(), sizeof(v[0]) * v.size());
    return at;
  };
  const size_t seg = put(h.seg), expect = put(h.expect), slot_ptr = put(h.slot_ptr), slot_row = put(h.slot_row),
               col = put(h.col), send = put(h.send), own = put(h.own), dd = put(h.diag);
  unsigned char *base = ar.upload(pack);
  d.v.seg = reinterpret_cast<const ClusterSeg *>(base + seg);
  d.v.expect = reinterpret_cast<const unsigned *>(base + expect);
  d.v.slot_ptr = reinterpret_cast<const int *>(base + slot_ptr);
  d.v.slot_row = reinterpret_cast<const int *>(base + slot_row);
  d.v.val = d.val = ar.upload(h.val);
  d.v.col = reinterpret_cast<const unsigned *>(base + col);
  d.v.send = reinterpret_cast<const unsigned *>(base + send);
  d.v.own = reinterpret_cast<const unsigned short *>(base + own);
  if (diag == nullptr) diag = d.diag = reinterpret_cast<T *>(base + dd);
  d.v.diag = diag;
  return d;
}

// Lanes per row: about five entries, or two 3x3 blocks, a lane (what a thread
// loads ahead). Fewer lanes leave the loaded-ahead slots (5,103 rows, 70
// entries a row: 111 us a step with 8 lanes, 71 with 16, 80 with 32).
inline int cluster_lanes(long long nnz, int rows, bool block) {
  const double len = static_cast<double>(nnz) / std::max(1, rows) / (block ? 3.0 : 1.0) - 1.0;
  int g = 4;
  while (g < 32 && g * (block ? 2.0 : 5.0) < len) g *= 2;
  return g;
}

// Lanes per row of the cluster layout's kernels.
template <typename F>
void with_lanes(int g, F &&f) {
  switch (g) {
    case 4: f(std::integral_constant<int, 4>()); break;
    case 8: f(std::integral_constant<int, 8>()); break;
    case 16: f(std::integral_constant<int, 16>()); break;
    default: f(std::integral_constant<int, 32>()); break;
  }
}

// Launch of clusters of ncta CTAs, with programmatic stream serialization
// when `overlap` (launch_pass).
struct ClusterLaunch {
  cudaLaunchAttribute attr[2];
  cudaLaunchConfig_t cfg = {};
  ClusterLaunch(int ncta, int clusters, int threads, size_t smem, bool overlap, cudaStream_t s) {
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ncta;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = dim3(static_cast<unsigned>(ncta * clusters));
    cfg.blockDim = dim3(static_cast<unsigned>(threads));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = overlap ? 2 : 1;
  }
  ClusterLaunch(const ClusterLaunch &) = delete;
};

// Shared memory that a CTA of the cluster kernels has for x.
inline int cluster_smem_bytes(int device) {
  int optin = 0;
  GSB_CK(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device));
  return optin - static_cast<int>(sizeof(ClusterSeg) * kClusterMaxColors + 8 * kClusterMaxPasses +
                                  2 * (kClusterMaxPasses + 8)) - 1024;
}

// Slots of `bytes` each that fit it.
inline int cluster_slots(int bytes, bool relaxed, int device) {
  return std::min(kClusterMaxSlots, cluster_smem_bytes(device) / (bytes * (relaxed ? 2 : 1)) - 1);
}

// Whether the device co-schedules clusters of 16 and of 8 CTAs of `kernel`
// with all the shared memory the CTAs may ask for (asked once per kernel and
// device). Raises the kernel's shared memory limit to what the device has (a
// limit only, the same for every solver of the process). Returns the largest
// size of at most `most`, or 0.
template <typename K>
int cluster_fit(K kernel, int threads, int most, int device) {
  static std::mutex mu;
  static std::unordered_map<const void *, std::vector<std::pair<int, int>>> cache;  // device, sizes (bit mask)
  std::lock_guard<std::mutex> lock(mu);
  auto &known = cache[reinterpret_cast<const void *>(kernel)];
  int sizes = -1;
  for (const auto &k : known)
    if (k.first == device) sizes = k.second;
  if (sizes < 0) {
    const int limit = cluster_smem_bytes(device);
    GSB_CK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, limit));
    GSB_CK(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    sizes = 0;
    for (int want : {16, 8}) {
      ClusterLaunch l(want, 1, threads, static_cast<size_t>(limit), false, nullptr);
      int n = 0;
      if (cudaOccupancyMaxActiveClusters(&n, kernel, &l.cfg) == cudaSuccess && n >= 1) sizes |= want;
      else cudaGetLastError();
    }
    known.emplace_back(device, sizes);
  }
  for (int want : {16, 8})
    if (want <= most && (sizes & want) != 0) return want;
  return 0;
}

}  // namespace gsb
