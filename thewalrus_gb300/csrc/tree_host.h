// Host side of the elimination tree: an instance's edge order and positions, the sizes and costs
// of its levels, and how its tree is cut into tasks or launches.
#pragma once
#include <algorithm>
#include <cstring>
#include <vector>

#include "host_common.h"
#include "tree_kernel.cuh"

namespace wg {

// The tree of a prepared instance (whole sum, finite-difference signs); false when it does not
// take one: more than TREE_MAX_K photons pairs, or inclusion/exclusion signs.
static inline bool tree_build(const InstDev& d, TreeInst& T) {
  memset(&T, 0, sizeof(T));
  const bool batch = d.kind >= KIND_BATCH_EVEN;
  const int nbe = d.kind == KIND_BATCH_EVEN ? 1 : (d.kind == KIND_BATCH_ODD ? 2 : 0);
  if (!d.glynn || d.n <= 0) return false;
  T.lda = d.lda;
  T.nout = d.nout;
  T.pL = T.pO = T.pB = -1;
  T.a_off = d.a_off;
  auto extra = [&](int row, int col) {
    T.row[T.X] = (short)row;
    T.col[T.X] = (short)col;
    return T.X++;
  };
  if (d.kind != KIND_PLAIN) T.pL = extra(d.n, d.n);
  if (d.kind == KIND_LOOP_ODD) {
    T.pO = extra(d.n + 1, -1);
    T.oddloop = d.oddloop;
  }
  if (d.kind == KIND_BATCH_ODD) T.pO = extra(1, 1);
  if (batch) T.pB = extra(0, 0);
  // elimination order: one simple edge (it takes half of its signs at the root), the multiple
  // edges by multiplicity, the other simple edges (cheapest per child, so at the wide bottom)
  std::vector<int> simple, multi, order;
  for (int e = nbe; e < d.E; ++e) {
    if (d.reps[e] == 1) simple.push_back(e);
    else if (d.reps[e] > 1) multi.push_back(e);
    T.K += d.reps[e];
  }
  if (T.K > TREE_MAX_K) return false;
  std::stable_sort(multi.begin(), multi.end(), [&](int a, int b) { return d.reps[a] < d.reps[b]; });
  size_t s0 = 0;
  if (!simple.empty()) order.push_back(simple[s0++]);
  else
    for (size_t k = 0; k < multi.size(); ++k)  // an odd multiplicity halves exactly
      if (d.reps[multi[k]] & 1) { std::rotate(multi.begin(), multi.begin() + k, multi.begin() + k + 1); break; }
  order.insert(order.end(), multi.begin(), multi.end());
  order.insert(order.end(), simple.begin() + s0, simple.end());
  T.E = (int)order.size();
  // closed forms of the last simple edges (the root edge is eliminated when it is the only one)
  int rem = 0;
  if (!batch)
    while (rem < (T.pL < 0 ? 2 : 1) && rem < T.E && d.reps[order[T.E - 1 - rem]] == 1) ++rem;
  T.steps = T.E - rem;
  T.diag = batch || !multi.empty();
  T.dpos = TREE_MAX_POS;
  for (int q = 0; q < T.E; ++q) {
    const int e = order[q], i = T.X + 2 * (T.E - 1 - q);
    T.row[i] = T.col[i] = (short)e;
    T.row[i + 1] = T.col[i + 1] = (short)(d.E + e);
    T.reps[q] = (unsigned char)d.reps[e];
    T.radix[q] = (unsigned char)(d.reps[e] + 1);
    if (q == 0) T.radix[q] = (unsigned char)((d.reps[e] + 1 + (d.reps[e] % 2 == 0)) / 2);
    if (d.reps[e] > 1) T.dpos = i;
    T.deg[q + 1] = (unsigned char)(T.deg[q] + d.reps[e]);
  }
  return true;
}

// binary exponent of the outputs' scale: 2^-r of every eliminated edge, twice the half of the first
static inline int tree_scale_exp(const TreeInst& T) { return T.deg[T.steps] - (T.steps > 0 ? 1 : 0); }

struct TreeSizes {
  double nodes[MAX_EDGES + 2];  // of the whole tree, after q steps
  double cost[MAX_EDGES + 2];   // multiply-adds of step q per parent with all children; [steps]: the leaf's
  double one[MAX_EDGES + 2];    // of step q per parent with one child
  double total = 0;
};

static inline void tree_sizes(const TreeInst& T, TreeSizes& z) {
  z.nodes[0] = 1;
  z.total = 0;
  for (int q = 0; q < T.steps; ++q) {
    const double L = T.deg[q] + 1, Lc = T.deg[q + 1] + 1, W = tree_width(T.X, T.E, q + 1);
    const double ne = tree_entries((int)W, T.diag), R = T.radix[q];
    if (T.reps[q] == 1) {
      z.one[q] = z.cost[q] = (ne * 2 + (T.pL >= 0)) * L * (L + 1) / 2;
    } else {
      z.one[q] = (ne * 2 + 4 * W + 45) * Lc * (Lc + 1) / 2;
      z.cost[q] = R * z.one[q];
    }
    z.nodes[q + 1] = z.nodes[q] * R;
    z.total += z.nodes[q] * z.cost[q];
  }
  const double L = T.deg[T.steps] + 1;
  z.cost[T.steps] = (T.pB >= 0 ? 12.0 * T.nout : 4.0) * L * (L + 1) / 2;
  z.total += z.nodes[T.steps] * z.cost[T.steps];
}

// elements of a node, and of the scratch of step q (np parents, nd children each)
static inline long long tree_node_elems(const TreeInst& T, int q) {
  return (long long)tree_entries(tree_width(T.X, T.E, q), T.diag) * (T.deg[q] + 1);
}
static inline long long tree_scratch_elems(const TreeInst& T, int q, long long np, int nd) {
  if (q == T.steps) return T.pO >= 0 && T.steps < T.E ? np * (T.deg[q] + 1) : 0;
  if (T.reps[q] == 1) return T.pL >= 0 ? np * (T.deg[q] + 1) : 0;
  return np * nd * (T.deg[q + 1] + 1) * (6 + 2ll * tree_width(T.X, T.E, q + 1));
}

// CTA kernel: elements of the two node buffers and the scratch when q edges are on the path
static inline void tree_cta_elems(const TreeInst& T, int q, long long out[3]) {
  out[0] = out[1] = out[2] = 0;
  long long np = 1;
  for (int s = 0; s <= T.steps; ++s) {
    out[s & 1] = std::max(out[s & 1], np * tree_node_elems(T, s));
    const int nd = s < T.steps ? (s < q ? 1 : T.radix[s]) : 1;
    out[2] = std::max(out[2], tree_scratch_elems(T, s, np, nd));
    if (s < T.steps) np *= nd;
  }
}

// Grid mode: one buffer per level, as many nodes as the level has or its byte budget allows (the
// levels below are then walked in blocks of parents, depth first), and the scratch of a step.
struct TreeGridPlan {
  long long cap[MAX_EDGES + 2] = {0};    // nodes of level q's buffer
  long long chunk[MAX_EDGES + 2] = {0};  // parents of step q per block
  long long off[MAX_EDGES + 2] = {0};    // byte offsets
  long long scr_off = 0, bytes = 0;
  long long launches = 0, leaves = 0;    // of one execution
};

template <class F>
static void tree_walk(const TreeInst& T, const TreeGridPlan& g, int q, int np, F& launch) {
  if (q == T.steps) {
    if (T.pO >= 0 && T.steps < T.E) launch(TP_M, q, 0, np, np, 0, 0);
    launch(TP_LEAF, q, 0, np, np, 0, 0);
    return;
  }
  const int R = T.radix[q], blocks = (int)((np + g.chunk[q] - 1) / g.chunk[q]), per = (np + blocks - 1) / blocks;
  for (int p0 = 0; p0 < np; p0 += per) {
    const int c = std::min(per, np - p0);
    if (T.reps[q] == 1) {
      if (T.pL >= 0) launch(TP_M, q, p0, c, np, 0, R);
      launch(TP_UNIT, q, p0, c, np, 0, R);
    } else {
      launch(TP_PREP, q, p0, c, np, 0, R);
      if (tree_width(T.X, T.E, q + 1) > 0) {
        launch(TP_Y, q, p0, c, np, 0, R);
        launch(TP_MULTI, q, p0, c, np, 0, R);
        if (T.pL >= 0) launch(TP_GLOOP, q, p0, c, np, 0, R);
      }
    }
    tree_walk(T, g, q + 1, c * R, launch);
  }
}

static inline void tree_grid_plan(const TreeInst& T, int sb, double budget, TreeGridPlan& g) {
  double nodes = 1;
  long long off = 0, scr = 0;
  auto al = [](long long x) { return (x + 255) & ~255ll; };
  for (int q = 0; q <= T.steps; ++q) {
    const long long nb = tree_node_elems(T, q) * sb;
    const int R = q ? T.radix[q - 1] : 1;
    long long cap = std::max<long long>((long long)(budget / (double)nb), std::max(R, 64));
    if (q) {  // a block's children and its scratch
      const long long se = std::max<long long>(tree_scratch_elems(T, q - 1, 1, R) * sb, 1);
      g.chunk[q - 1] = std::min(std::max<long long>(cap / R, 1), std::max<long long>((long long)(budget / (double)se), 1));
      g.chunk[q - 1] = std::min(g.chunk[q - 1], g.cap[q - 1]);
      cap = g.chunk[q - 1] * R;
      scr = std::max(scr, tree_scratch_elems(T, q - 1, g.chunk[q - 1], R) * sb);
    }
    if (nodes < (double)cap) cap = (long long)nodes;
    g.cap[q] = cap;
    g.off[q] = off;
    off += al(cap * nb);
    if (q < T.steps) nodes *= T.radix[q];
  }
  scr = std::max(scr, tree_scratch_elems(T, T.steps, g.cap[T.steps], 1) * sb);
  g.scr_off = off;
  g.bytes = off + al(std::max<long long>(scr, 16));
  g.launches = 1;  // the root
  g.leaves = 0;
  auto count = [&](int phase, int, int, int, int, int, int) {
    ++g.launches;
    g.leaves += phase == TP_LEAF;
  };
  tree_walk(T, g, 0, 1, count);
}

// shared memory of the leaf and of the block sums
static inline int tree_smem(const TreeInst& T, int sb) {
  const int nw = TREE_THREADS / 32;
  return nw * (T.pB >= 0 ? 5 * (T.deg[T.steps] + 1) + 32 : 1) * sb;
}

// Where the path of a CTA's task ends: the split that minimises the whole work, each path
// recomputed by every task below it, over the chip's SMs plus one task's time as the tail
// (weighted by the instance's share of the launch's work).  Returns that time in multiply-adds
// of one SM; the workspace bound keeps a subtree's widest levels within max_elems.
static inline double tree_split(const TreeInst& T, const TreeSizes& z, int sms, double share, long long max_elems,
                                int& q_best) {
  double best = -1, path = 0;
  q_best = 0;
  for (int q = 0; q <= T.steps; ++q) {
    double sub = 0;
    for (int s = q; s <= T.steps; ++s) sub += z.nodes[s] / z.nodes[q] * z.cost[s];
    const double tasks = z.nodes[q], task = path + sub, f = tasks * task / sms + share * task;
    long long el[3];
    tree_cta_elems(T, q, el);
    const bool fits = el[0] + el[1] + el[2] <= max_elems && tasks <= 65536.0;
    if (fits && (best < 0 || f < best)) {
      best = f;
      q_best = q;
    }
    if (q < T.steps) path += z.one[q];
  }
  return best;
}

}  // namespace wg
