// pme_direct_plan.h -- host-side choices and tables of the direct-space engine that need no device: the
// columns and x bins that the atoms are sorted into, the Ewald table.  Plain C++, so that they can be
// checked without a GPU.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstddef>
#include <vector>

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

constexpr int kWarps = 4;             // warps per CTA of the pair kernel
constexpr int kPairCtas = 5;          // its CTAs per SM
constexpr int kQueue = 72;            // queued candidates per i atom (at most 32 more at a time)
constexpr size_t kPairShared = kWarps * (kCluster * (kQueue + 1) * 8 + kCluster * 12);   // static, bytes

// Whether every CTA holds the vdW parameters as a square of types in shared memory, beside table_bytes of
// the Ewald table: while that costs none of the CTAs on an SM of sm_shared bytes (kPairCtas; fewer with
// energies beyond a cutoff of 29 A).  The packed triangle is else read through L1.  192,000 atoms at 9 A,
// us, square and packed: forces only 2 types 748 and 843, 40 (5 CTAs) 764 and 857, 48 (4) 868 and 863, 64
// (3) 1,050 and 868; with energies 32 (5) 1,036 and 1,091, 40 (4) 1,128 and 1,091, 64 (3) 1,336 and 1,098;
// 24,000 atoms at 32 A with energies, 2 types (4) 3,877 and 4,361.
inline bool square_types(int ntype, size_t table_bytes, size_t sm_shared) {
  const size_t without = kPairShared + table_bytes + 1024, with = without + 8 * (size_t)ntype * ntype;
  return with <= sm_shared && sm_shared / with >= std::min((size_t)kPairCtas, sm_shared / without);
}

// Ewald table: polynomials on the intervals of s = r^2 that share their leading float bits, kTabOctave
// per factor of two from s = 2 on, so that the interval is read off the bits.
constexpr int kTabOctave = 32, kTabTerms = 6, kTabMax = 16 * kTabOctave;

// Polynomial through f at the kTabTerms Chebyshev points of [mid - half, mid + half]: coefficients of
// 1, t, t^2, ..., t = s - mid (the Chebyshev series, written out in powers of t / half).
template <class F>
void chebyshev_powers(F f, double mid, double half, double* out) {
  const double pi = 3.14159265358979323846;
  double c[kTabTerms], prev[kTabTerms] = {1.0}, cur[kTabTerms] = {0.0, 1.0}, y[kTabTerms];
  for (int k = 0; k < kTabTerms; k++) y[k] = f(mid + half * std::cos(pi * (k + 0.5) / kTabTerms));
  for (int j = 0; j < kTabTerms; j++) {
    c[j] = 0.0;
    for (int k = 0; k < kTabTerms; k++) c[j] += (j == 0 ? 1.0 : 2.0) / kTabTerms * y[k] * std::cos(pi * j * (k + 0.5) / kTabTerms);
  }
  for (int i = 0; i < kTabTerms; i++) out[i] = c[0] * prev[i] + c[1] * cur[i];
  for (int j = 2; j < kTabTerms; j++) {   // T_j = 2 z T_{j-1} - T_{j-2}
    double next[kTabTerms];
    for (int i = 0; i < kTabTerms; i++) next[i] = (i > 0 ? 2.0 * cur[i - 1] : 0.0) - prev[i];
    for (int i = 0; i < kTabTerms; i++) {
      out[i] += c[j] * next[i];
      prev[i] = cur[i];
      cur[i] = next[i];
    }
  }
  double scale = 1.0;
  for (int i = 0; i < kTabTerms; i++, scale /= half) out[i] *= scale;
}

// Per interval from s = 2 to roff^2 the coefficients of F(s) = (r dE/dr) / s, then of E(s) = erfc(kappa r)
// / r.  Largest errors for r >= 1.5 A, kappa 0.32, cutoffs of 9 and 12 A: 3e-13 of F r, 5e-14 of E; rms over
// the pairs 1.4e-14 and 4e-15.  (Cubics on 64 intervals per factor of two, a third larger: 3e-10 and
// 6e-11, rms 1.5e-11 and 5e-12.  A cubic Hermite table of 4,096 even intervals, too large for shared
// memory: 4e-10 and 6e-11 at 9 A, rms 6e-12 and 1e-12.)
inline std::vector<double> ewald_table(double kappa, double roff) {
  const double c1 = 2.0 / std::sqrt(3.14159265358979323846) * kappa;
  auto E = [&](double s) { const double r = std::sqrt(s); return std::erfc(kappa * r) / r; };
  auto F = [&](double s) { return (-c1 * std::exp(-kappa * kappa * s) - E(s)) / s; };
  std::vector<double> t;
  for (int i = 0; i < kTabMax; i++) {
    const double w = std::ldexp(2.0, i / kTabOctave) / kTabOctave, a = (kTabOctave + i % kTabOctave) * w;
    if (a > roff * roff) break;
    t.resize(t.size() + 2 * kTabTerms);
    chebyshev_powers(F, a + 0.5 * w, 0.5 * w, t.data() + t.size() - 2 * kTabTerms);
    chebyshev_powers(E, a + 0.5 * w, 0.5 * w, t.data() + t.size() - kTabTerms);
  }
  return t;
}

}  // namespace direct
}  // namespace pme
