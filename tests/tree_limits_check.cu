// Host check of the elimination tree's estimates and sizes (tree_host.h), for instances read from standard
// input.  Built and run by tests/test_tree_limits.py.
//
// Arguments: walk-bytes limit node-bytes.
// Input: instances; per instance kind (InstDev's) E edge_reps.
// Output per instance: multiply-adds as estimated and as a walk in levels of walk-bytes adds them up
// (0: not walked); whether its levels fit the limit, and their bytes.
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "../thewalrus_gb300/csrc/tree_host.h"

using namespace wg;

static int rd() {
  int x;
  if (std::scanf("%d", &x) != 1) std::exit(2);
  return x;
}

int main(int, char** argv) {
  const double walk = std::atof(argv[1]), limit = std::atof(argv[2]);
  const int sb = std::atoi(argv[3]);
  for (int k = rd(); k > 0; --k) {
    InstDev d;
    memset(&d, 0, sizeof(d));
    d.kind = rd();
    d.glynn = d.nout = 1;
    for (int e = rd(); e > 0; --e) d.reps[d.E++] = rd();
    d.n = 2 * d.E;
    d.lda = d.n + 1;
    TreeInst T;
    if (!tree_build(d, T)) return 3;
    double sum = 0;
    if (walk > 0) {
      TreeLevels g;
      tree_levels(T, 16, walk, g);
      auto add = [&](int phase, int q, int, int np, int) { sum += tree_macs(T, phase, q, np); };
      tree_walk(T, g, 0, 1, add);
    }
    TreeLevels g;
    const bool fits = tree_levels_within(T, sb, limit, g);
    std::printf("%.17g %.17g %d %.17g\n", tree_work(T), sum, fits, (double)g.bytes);
  }
  return 0;
}
