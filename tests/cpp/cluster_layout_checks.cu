// The cluster layout of small matrices (cluster_layout.h), checked on the host:
// prints "bad <n>" with the number of rules broken, and the layout's sizes.
#include <cstdio>
#include <vector>

#include "cluster_layout.h"

using namespace gsb;

// 9-point grid of nx x ny cells in four colours, rows in colour order.
static Csr grid(int nx, int ny, std::vector<int> &first) {
  std::vector<int> id(nx * ny), cell;
  first.assign(1, 0);
  for (int c = 0; c < 4; ++c) {
    for (int y = 0; y < ny; ++y)
      for (int x = 0; x < nx; ++x)
        if ((x & 1) + 2 * (y & 1) == c) id[y * nx + x] = static_cast<int>(cell.size()), cell.push_back(y * nx + x);
    first.push_back(static_cast<int>(cell.size()));
  }
  Csr a;
  a.rows = a.cols = nx * ny;
  a.rp.assign(1, 0);
  for (int r = 0; r < a.rows; ++r) {
    const int x0 = cell[r] % nx, y0 = cell[r] / nx;
    std::vector<int> cols;
    for (int y = std::max(0, y0 - 1); y <= std::min(ny - 1, y0 + 1); ++y)
      for (int x = std::max(0, x0 - 1); x <= std::min(nx - 1, x0 + 1); ++x) cols.push_back(id[y * nx + x]);
    std::sort(cols.begin(), cols.end());
    for (int c : cols) a.ci.push_back(c), a.v.push_back(c == r ? 9.0 : -1.0 - 0.01 * c);
    a.rp.push_back(static_cast<int>(a.ci.size()));
  }
  return a;
}

// Every message goes to a CTA and a slot that exist (also the address formed
// for a lane that sends nothing), and every CTA expects what it is sent.
template <typename T>
static int check(const HostCluster<T> &h) {
  int bad = 0;
  for (unsigned w : h.send) {
    const int cta = static_cast<int>((w >> 16) & 15u), slot = static_cast<int>(w & 0xffffu);
    if (cta >= h.ncta || slot >= std::max(1, h.max_slots)) ++bad;
  }
  for (int c = 0; c < h.ncolors; ++c) {
    std::vector<unsigned> got(h.ncta, 0);
    for (int q = 0; q < h.ncta; ++q) {
      const ClusterSeg &s = h.seg[static_cast<size_t>(q) * h.ncolors + c];
      const long long n = s.rows > 0 ? static_cast<long long>(s.trips) * s.schunks * s.stride : 0;
      for (long long i = 0; i < n; ++i)
        if (h.send[s.sbase + i] != kNoSend) ++got[(h.send[s.sbase + i] >> 16) & 15u];
    }
    for (int q = 0; q < h.ncta; ++q)
      if (got[q] != h.expect[static_cast<size_t>(q) * h.ncolors + c]) ++bad;
  }
  return bad;
}

// `a` with every entry replaced by a 3x3 block.
static Csr blocked(const Csr &a) {
  Csr m;
  m.rows = m.cols = 3 * a.rows;
  m.rp.assign(1, 0);
  for (int r = 0; r < m.rows; ++r) {
    for (int k = a.rp[r / 3]; k < a.rp[r / 3 + 1]; ++k)
      for (int c = 0; c < 3; ++c)
        if (a.ci[k] == r / 3 || c != r % 3 || (k & 1)) {  // blocks with holes
          m.ci.push_back(3 * a.ci[k] + c);
          m.v.push_back(a.v[k] + 0.001 * r + 0.01 * c);
        }
    m.rp.push_back(static_cast<int>(m.ci.size()));
  }
  return m;
}

// New values put into a kept layout against the layout built from them.
template <typename T>
static int refreshed(const Csr &a, const std::vector<int> &first, int g, int ncta, bool block) {
  HostCluster<T> h, fresh;
  Csr b = a;
  for (size_t k = 0; k < b.v.size(); ++k) b.v[k] = 1.0 / (3.0 + static_cast<double>(k % 1001));
  const auto make = [&](const Csr &m, HostCluster<T> &out) {
    return block ? make_cluster_blocks<T>(m, first, g, ncta, false, 20000, out) : make_cluster<T>(m, first, g, ncta, false, 20000, out);
  };
  if (!make(a, h) || !make(b, fresh)) return 1;
  std::vector<T> val(h.val.size(), T(0)), diag;
  if (!(block ? cluster_block_values<T>(b, h.entries, val) : cluster_values<T>(b, h.entries, val, diag))) return 1;
  int bad = val != fresh.val || (!block && diag != fresh.diag);
  // another pattern is refused
  const int u = block ? 3 : 1;
  Csr c = b;
  for (int r = 0; r < u; ++r) {
    const int at = c.rp[r + 1];
    c.ci.insert(c.ci.begin() + at, a.cols - 1);
    c.v.insert(c.v.begin() + at, 1.0);
    for (int q = r + 1; q <= c.rows; ++q) ++c.rp[q];
  }
  bad += block ? cluster_block_values<T>(c, h.entries, val) : cluster_values<T>(c, h.entries, val, diag);
  return bad;
}

int main() {
  int bad = 0, stale = 0;
  for (int ncta : {8, 16})
    for (int g : {4, 8, 16, 32})
      for (int side : {3, 17, 40}) {
        std::vector<int> first;
        const Csr a = grid(side, side + 2, first);
        HostCluster<double> h;
        if (!make_cluster<double>(a, first, g, ncta, false, 20000, h)) {
          ++bad;
          continue;
        }
        bad += check(h);
        stale += refreshed<double>(a, first, g, ncta, false) + refreshed<float>(a, first, g, ncta, false);
        const Csr b = blocked(a);
        stale += refreshed<double>(b, first, g, ncta, true) + refreshed<float>(b, first, g, ncta, true);
      }
  std::printf("bad %d\nstale %d\n", bad, stale);
  return 0;
}
