// Host-side choices, tables and sums of the direct-space engine, printed for tests/test_direct_plan.py (no GPU).
#include <cmath>
#include <cstdio>
#include <cstring>

#include "pme_direct_plan.h"
#include "pme_direct_math.h"

using namespace pme::direct;

// box and cutoff and atom count per line of stdin -> x bins, columns along y and z, reach, cells;
// cells and columns with room for a longer box
static int columns() {
  double b[3], roff;
  int n;
  while (std::scanf("%lf %lf %lf %lf %d", &b[0], &b[1], &b[2], &roff, &n) == 5) {
    const Columns c = plan_columns(b, roff, n), m = room_columns(b, roff, n);
    std::printf("%d %d %d %d %zu %zu %d\n", c.nc[0], c.nc[1], c.nc[2], c.reach, c.cells(), m.cells(), m.count());
  }
  return 0;
}

// terms per line of stdin -> their sum at 2^40 by RoundedSum after every one; terms of 2^10 and more go
// the way of the kernel's large ones
static int sums() {
  double v;
  RoundedSum a;
  int terms = 0;
  while (std::scanf("%lf", &v) == 1) {
    if (std::fabs(v) < 1024.0) {
      a.add_rounded(std::fma(v, 1099511627776.0, kRoundMagic));
      terms++;
    } else {
      a.add(std::llrint(v * 1099511627776.0));
    }
    std::printf("%lld\n", (long long)a.total(terms));
  }
  return 0;
}

// kappa and cutoff per line of stdin -> the Ewald table, an interval's coefficients per line
static int ewald() {
  double kappa, roff;
  while (std::scanf("%lf %lf", &kappa, &roff) == 2) {
    const std::vector<double> t = ewald_table(kappa, roff);
    for (size_t i = 0; i < t.size(); i++) std::printf(i % (2 * kTabTerms) == 2 * kTabTerms - 1 ? "%.17g\n" : "%.17g ", t[i]);
  }
  return 0;
}

// Ewald table bytes and shared memory per SM per line of stdin -> types up to which the square is held
static int types() {
  long long bytes, shared;
  while (std::scanf("%lld %lld", &bytes, &shared) == 2) {
    int n = 0;
    while (square_types(n + 1, (size_t)bytes, (size_t)shared)) n++;
    std::printf("%d\n", n);
  }
  return 0;
}

int main(int argc, char** argv) {
  if (argc == 2 && !std::strcmp(argv[1], "columns")) return columns();
  if (argc == 2 && !std::strcmp(argv[1], "sums")) return sums();
  if (argc == 2 && !std::strcmp(argv[1], "ewald")) return ewald();
  if (argc == 2 && !std::strcmp(argv[1], "types")) return types();
  return 1;
}
