// pme_direct_plan.h -- host-side choices of the direct-space engine that need no device: the columns and
// x bins that the atoms are sorted into.  Plain C++, so that they can be checked without a GPU.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstddef>

namespace pme {
namespace direct {

constexpr int kCluster = 8;           // i atoms of a warp task: 4 lanes share one atom
constexpr int kMaxReach = 4;          // columns within the cutoff on each side, at most
constexpr int kMaxXBins = 1024;       // x look-up entries per column, at most
constexpr int kMaxColumns = 1 << 22;  // (y, z) columns, at most
constexpr double kMaxXEntries = 16.0e6;

struct Columns {
  int nc[3];   // x bins per column; columns along y and z
  int reach;   // columns within the cutoff on each side
  int count() const { return nc[1] * nc[2]; }
  size_t cells() const { return (size_t)count() * (nc[0] + 1); }   // per column: its x bins and its end
};

// Columns at least roff / reach wide along y and z, the width nearest to the edge of a cube of kCluster
// atoms at the system's density, so that a cluster is about as long as wide.  The margin is the rounding
// of a coordinate's column index in FP32.  Wider columns are as correct: where a cutoff far below the
// box would make more than kMaxColumns, both axes take fewer, in proportion.  x bins of about 1 A (a few
// atoms each), kMaxXEntries of them in all: at most 20.2e6 cells, 81 MB for each of the two tables.
inline Columns plan_columns(const double* box, double roff, int natom) {
  Columns c;
  const double edge = std::cbrt(box[0] * box[1] * box[2] * kCluster / std::max(natom, 1));
  c.reach = (int)std::max(1.0, std::min((double)kMaxReach, std::round(roff / edge)));
  double n[2];
  for (int d = 0; d < 2; d++) n[d] = std::max(1.0, std::floor(box[d + 1] * c.reach / (roff * (1.0 + 1e-5) + 1e-6 * box[d + 1])));
  if (n[0] * n[1] > kMaxColumns) {
    // not below 2 reach - 1 (what the shortest box, two cutoffs, has): an offset wraps around once only
    const int lo = n[0] <= n[1] ? 0 : 1;
    n[lo] = std::max(std::min(n[lo], 2.0 * c.reach - 1.0), std::floor(n[lo] * std::sqrt(kMaxColumns / (n[0] * n[1]))));
    n[1 - lo] = std::min(n[1 - lo], std::floor(kMaxColumns / n[lo]));
  }
  c.nc[1] = (int)n[0];
  c.nc[2] = (int)n[1];
  c.nc[0] = (int)std::max(1.0, std::min({box[0], (double)kMaxXBins, kMaxXEntries / (n[0] * n[1])}));
  return c;
}

// Clusters that n atoms make at most: every column rounds up once.
inline int most_clusters(int n, const Columns& c) { return n / kCluster + std::min(n, c.count()) + 1; }

// Columns of a box 5% longer along every edge at the same density: room for a box that breathes (constant
// pressure) without new work space at each new maximum, where a column more along an axis can be a
// quarter more cells.
inline Columns room_columns(const double* box, double roff, int natom) {
  const double f = 1.05, b[3] = {f * box[0], f * box[1], f * box[2]};
  return plan_columns(b, roff, (int)std::min(2147483647.0, std::ceil(f * f * f * natom)));
}

}  // namespace direct
}  // namespace pme
