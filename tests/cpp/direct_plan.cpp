// Host-side choices of the direct-space engine, printed for tests/test_direct_plan.py (no GPU).
#include <cstdio>
#include <cstring>

#include "pme_direct_plan.h"

using namespace pme::direct;

// box and cutoff and atom count per line of stdin -> x bins, columns along y and z, reach, cells
static int columns() {
  double b[3], roff;
  int n;
  while (std::scanf("%lf %lf %lf %lf %d", &b[0], &b[1], &b[2], &roff, &n) == 5) {
    const Columns c = plan_columns(b, roff, n);
    std::printf("%d %d %d %d %zu\n", c.nc[0], c.nc[1], c.nc[2], c.reach, c.cells());
  }
  return 0;
}

int main(int argc, char** argv) {
  if (argc == 2 && !std::strcmp(argv[1], "columns")) return columns();
  return 1;
}
