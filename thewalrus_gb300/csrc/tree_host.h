// Host side of the elimination tree: an instance's edge order and positions, the sizes of its levels,
// and the program (rounds of segments) that a launch of the tree kernel runs.
#pragma once
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "host_common.h"
#include "tree_kernel.cuh"

namespace wg {

constexpr long long TREE_SMEM_BYTES = 200 << 10;  // dynamic shared memory of a CTA, at most

// The tree of a prepared instance (whole sum, finite-difference signs); false when it does not
// take one: more than TREE_MAX_K photon pairs, or inclusion/exclusion signs.  `simple_only`: an edge of
// multiplicity r as r simple edges on copies of its vertices (the same sum: r signs add up to each
// delta binomially often), for at most MAX_EDGES pairs.
static inline bool tree_build(const InstDev& d, TreeInst& T, bool simple_only = false) {
  memset(&T, 0, sizeof(T));
  const bool batch = d.kind >= KIND_BATCH_EVEN;
  const int nbe = d.kind == KIND_BATCH_EVEN ? 1 : (d.kind == KIND_BATCH_ODD ? 2 : 0);
  if (!d.glynn || d.n <= 0) return false;
  T.lda = d.lda;
  T.nout = d.nout;
  T.pL = T.pO = T.pB = -1;
  T.a_off = d.a_off;
  auto extra = [&](int row, int col) {
    T.row[T.X] = (signed char)row;
    T.col[T.X] = (signed char)col;
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
    if (d.reps[e] == 1 || simple_only) simple.insert(simple.end(), d.reps[e], e);
    else if (d.reps[e] > 1) multi.push_back(e);
    T.K += d.reps[e];
  }
  if (T.K > (simple_only ? MAX_EDGES : TREE_MAX_K)) return false;
  std::stable_sort(multi.begin(), multi.end(), [&](int a, int b) { return d.reps[a] < d.reps[b]; });
  size_t s0 = 0;
  if (!simple.empty()) order.push_back(simple[s0++]);
  else
    for (size_t k = 0; k < multi.size(); ++k)  // an odd multiplicity halves exactly
      if (d.reps[multi[k]] & 1) { std::rotate(multi.begin(), multi.begin() + k, multi.begin() + k + 1); break; }
  order.insert(order.end(), multi.begin(), multi.end());
  order.insert(order.end(), simple.begin() + s0, simple.end());
  T.E = (int)order.size();
  // closed forms of the last simple edges
  int rem = 0;
  if (!batch)
    while (rem < (T.pL < 0 ? 2 : 1) && rem < T.E && (simple_only || d.reps[order[T.E - 1 - rem]] == 1)) ++rem;
  T.steps = T.E - rem;
  T.diag = batch || !multi.empty();
  T.dpos = TREE_MAX_POS;
  for (int q = 0; q < T.E; ++q) {
    const int e = order[q], i = T.X + 2 * (T.E - 1 - q), r = simple_only ? 1 : d.reps[e];
    T.row[i] = T.col[i] = (signed char)e;
    T.row[i + 1] = T.col[i + 1] = (signed char)(d.E + e);
    T.reps[q] = (unsigned char)r;
    T.radix[q] = (unsigned char)(r + 1);
    if (q == 0) T.radix[q] = (unsigned char)((r + 1 + (r % 2 == 0)) / 2);
    if (r > 1) T.dpos = i;
    T.deg[q + 1] = (unsigned char)(T.deg[q] + r);
  }
  return true;
}

// binary exponent of the outputs' scale: 2^-r of every eliminated edge, twice the half of the first
static inline int tree_scale_exp(const TreeInst& T) { return T.deg[T.steps] - (T.steps > 0 ? 1 : 0); }

// bytes of a node element
static inline int tree_bytes(int ttype) {
  switch (ttype) {
    case ST_CPLX64: return (int)sizeof(TreeScalar<c64>::T);
    case ST_CPLXDF: return (int)sizeof(TreeScalar<cdf>::T);
    case ST_CPLXDD: return (int)sizeof(TreeScalar<cdd>::T);
    default: return (int)stype_bytes(tree_stype(ttype));
  }
}

// elements of a node, of m in step q (np parents), and of its other scratch
static inline long long tree_node_elems(const TreeInst& T, int q) {
  return (long long)tree_entries(tree_width(T.X, T.E, q), T.diag) * (T.deg[q] + 1);
}
static inline long long tree_m_elems(const TreeInst& T, int q, long long np) {
  const bool has = q == T.steps ? T.pO >= 0 && T.steps < T.E : T.reps[q] == 1 && T.pL >= 0;
  return has ? np * (T.deg[q] + 1) : 0;
}
static inline long long tree_scratch_elems(const TreeInst& T, int q, long long np) {
  if (q == T.steps || T.reps[q] == 1) return 0;
  if (T.reps[q] == 2) return np * (T.deg[q] + 1) * (8 + 2ll * tree_width(T.X, T.E, q + 1));
  return np * T.radix[q] * (T.deg[q + 1] + 1) * (6 + 2ll * tree_width(T.X, T.E, q + 1));
}

// Levels of one instance in the workspace: one buffer per level, as many nodes as the level has or a
// byte budget allows (the levels below are then walked in blocks of parents, depth first).
struct TreeLevels {
  long long cap[MAX_EDGES + 2] = {0};    // nodes of level q's buffer
  long long chunk[MAX_EDGES + 2] = {0};  // parents of step q per block
  long long off[MAX_EDGES + 2] = {0};    // byte offsets
  long long scr_off = 0, m_elems = 0, bytes = 0;  // m_elems: of one step
  double phases = 0;                     // about, of one execution
};

static inline void tree_levels(const TreeInst& T, int sb, double budget, TreeLevels& g) {
  double nodes = 1, walks = 1;
  long long off = 0, scr = 0;
  auto al = [](long long x) { return (x + 255) & ~255ll; };
  g.phases = 1;
  for (int q = 0; q <= T.steps; ++q) {
    const long long nb = tree_node_elems(T, q) * sb;
    const int R = q ? T.radix[q - 1] : 1;
    long long cap = std::max<long long>((long long)(budget / (double)nb), std::max(R, 64));
    if (q) {  // a block's children and its scratch
      const long long se =
          std::max<long long>((tree_scratch_elems(T, q - 1, 1) + 2 * tree_m_elems(T, q - 1, 1)) * sb, 1);
      long long c = std::min(std::max<long long>(cap / R, 1), std::max<long long>((long long)(budget / (double)se), 1));
      c = std::min(c, g.cap[q - 1]);
      g.chunk[q - 1] = c;
      cap = c * R;
      scr = std::max(scr, tree_scratch_elems(T, q - 1, c) * sb);
      g.m_elems = std::max(g.m_elems, tree_m_elems(T, q - 1, c));
      walks *= (double)((g.cap[q - 1] + c - 1) / c);
      g.phases += walks * (T.reps[q - 1] == 1 ? 1 : (T.reps[q - 1] == 2 ? 2 : 4));
    }
    if (nodes < (double)cap) cap = (long long)nodes;
    g.cap[q] = cap;
    g.off[q] = off;
    off += al(cap * nb);
    if (q < T.steps) nodes *= T.radix[q];
  }
  g.phases += walks * (T.pL >= 0 ? 2 : 1);
  g.m_elems = std::max(g.m_elems, tree_m_elems(T, T.steps, g.cap[T.steps]));
  scr = std::max(scr, 2 * g.m_elems * sb);  // multiple edges come first: their scratch is free by then
  g.scr_off = off;
  g.bytes = off + al(std::max<long long>(scr, 16));
}

// A level's byte budget: larger levels are walked in blocks.  n = 40: 5,409 us with 64 MB, 4,851 with 200.
constexpr double TREE_LEVEL_BYTES = 200e6;

// The levels within `limit` bytes: blocks as large as TREE_LEVEL_BYTES and the limit allow.  False when
// even small blocks (a 256th of the default, whose rounds no longer fill the chip) take more.
static inline bool tree_levels_within(const TreeInst& T, int sb, double limit, TreeLevels& g) {
  for (double budget = TREE_LEVEL_BYTES; budget >= TREE_LEVEL_BYTES / 256; budget *= 0.7) {
    g = TreeLevels();
    tree_levels(T, sb, budget, g);
    if ((double)g.bytes <= limit) return true;
  }
  return false;
}

// Whether a phase stands in the round of the one before it: a double edge's g beside its rows; of a
// loop kind's simple edge the g of the step before, m and the other entries.
static inline bool tree_same_round(int before, int phase) {
  return (before == TP_W2 && phase == TP_G2) || (before == TP_G && phase == TP_M) || (before == TP_M && phase == TP_UNIT);
}

// The phases of step q (the last: of the leaves) in order: f(phase).  A loop kind's TP_G is not among
// them, see tree_walk.
template <class F>
static void tree_step(const TreeInst& T, int q, F f) {
  if (q == T.steps) {
    if (T.pO >= 0 && T.steps < T.E) f(TP_M);
    f(TP_LEAF);
  } else if (T.reps[q] == 1) {
    if (T.pL >= 0) f(TP_M);
    f(TP_UNIT);
  } else if (T.reps[q] == 2) {
    const bool rows = tree_width(T.X, T.E, q + 1) > 0;
    if (rows) f(TP_W2);
    f(TP_G2);  // beside TP_W2, in the same round
    if (rows) f(TP_MULTI2);
  } else {
    f(TP_PREP);
    if (tree_width(T.X, T.E, q + 1) > 0) {
      f(TP_Y);
      f(TP_MULTI);
      if (T.pL >= 0) f(TP_GLOOP);
    }
  }
}

// The phases of an instance in order, each once for every block: f(phase, q, p0, np, level's nodes).
// `late`, a parents' block [late0, late0 + late) of a level of `lateps` nodes: step q - 1's TP_G, due in
// this step's first round.
template <class F>
static void tree_walk(const TreeInst& T, const TreeLevels& g, int q, int np, F& f, int late0 = 0, int late = 0,
                      int lateps = 0) {
  if (late) f(TP_G, q - 1, late0, late, lateps);
  if (q == T.steps) {
    tree_step(T, q, [&](int phase) { f(phase, q, 0, np, np); });
    return;
  }
  const int R = T.radix[q], blocks = (int)((np + g.chunk[q] - 1) / g.chunk[q]), per = (np + blocks - 1) / blocks;
  const bool loop = T.reps[q] == 1 && T.pL >= 0;
  for (int p0 = 0; p0 < np; p0 += per) {
    const int c = std::min(per, np - p0);
    tree_step(T, q, [&](int phase) { f(phase, q, p0, c, np); });
    if (loop) tree_walk(T, g, q + 1, c * R, f, p0, c, np);
    else tree_walk(T, g, q + 1, c * R, f);
  }
}

// threads of a phase with `tile` coefficients a thread (0: four threads a coefficient), and its
// multiply-adds
static inline double tree_items(const TreeInst& T, int phase, int q, double np, int tile) {
  if (tile == TREE_PAIRS) return 2 * tree_items(T, phase, q, np, 1);
  if (tile == 0) {
    const bool whole = phase == TP_ROOT || phase == TP_FIRST || phase == TP_PREP || phase == TP_GLOOP || phase == TP_G2 ||
                       (phase == TP_LEAF && (T.pB >= 0 || T.steps == T.E));
    return tree_items(T, phase, q, np, 1) * (whole ? 1 : 4);
  }
  const int Lp = T.deg[q] + 1, Lc = q < T.steps ? T.deg[q + 1] + 1 : Lp, W = tree_width(T.X, T.E, q + 1);
  const double nc = q < T.steps ? np * T.radix[q] : np;
  switch (phase) {
    case TP_ROOT: return tree_entries(tree_width(T.X, T.E, 0), T.diag);
    case TP_FIRST: return tree_entries(W, T.diag);
    case TP_M: case TP_G: return np * tree_tiles(Lp, tile);
    case TP_UNIT: return np * tree_tiles(Lp, tile) * (tree_entries(W, T.diag) - (T.pL >= 0));
    case TP_PREP: case TP_GLOOP: return 32 * nc;
    case TP_G2: return 32 * np;
    case TP_W2: return np * 2 * W * tree_tiles(Lp, tile);
    case TP_MULTI2: return np * (tree_entries(W, T.diag) - 1) * tree_tiles(Lp + 1, tile);
    case TP_Y: return nc * 2 * W * tree_tiles(Lc, tile);
    case TP_MULTI: return nc * (tree_entries(W, T.diag) - 1) * tree_tiles(Lc, tile);
    default: return T.pB >= 0 ? 32 * np : np * (T.steps < T.E ? tree_tiles(Lp, tile) : 1);
  }
}
static inline double tree_macs(const TreeInst& T, int phase, int q, double np) {
  const double Lp = T.deg[q] + 1, Lc = q < T.steps ? T.deg[q + 1] + 1 : Lp, W = tree_width(T.X, T.E, q + 1);
  const double nc = q < T.steps ? np * T.radix[q] : np, tp = Lp * (Lp + 1) / 2, tc = Lc * (Lc + 1) / 2;
  switch (phase) {
    case TP_ROOT: return 0;
    case TP_FIRST: return 2 * tree_entries((int)W, T.diag);
    case TP_M: case TP_G: return np * tp;
    case TP_UNIT: return np * tp * (2 * tree_entries((int)W, T.diag) - (T.pL >= 0 ? 2 : 1));
    case TP_PREP: return nc * 12 * tc * std::max(1.0, 32 / Lc);
    case TP_GLOOP: return nc * 5 * tc * std::max(1.0, 32 / Lc);
    case TP_G2: return np * 8 * tp * std::max(1.0, 10 / Lp);
    case TP_W2: return np * 4 * W * tp;
    case TP_MULTI2: return np * 4 * (tree_entries((int)W, T.diag) - 1) * tp;
    case TP_Y: return nc * 4 * W * tc;
    case TP_MULTI: return nc * 2 * (tree_entries((int)W, T.diag) - 1) * tc;
    default: return np * (T.pB >= 0 ? 3.0 * T.nout : 3.0) * tp;
  }
}

// elements of a warp's shared memory: the output sums, a batch's work series (with copies of two of
// the node's), a multiple edge's; `most` when those would take too much (the phases then work in L2,
// a batch without the copies)
static inline int tree_smem(const TreeInst& T, int most) {
  const int L = T.deg[T.steps] + 1;
  int need = 1, lc = 0;
  for (int q = 0; q < T.steps; ++q)
    if (T.reps[q] > 1) lc = std::max(lc, T.deg[q + 1] + 1);  // 8 series of a double edge, 9 of the others
  if (9 * lc <= most) need = std::max(need, 9 * lc);
  const int all = 32 + (T.nout + 4) * L;
  if (T.pB >= 0) need = std::max(need, all <= most ? all : 5 * L + 32);
  return need;
}

// elements of a warp's shared memory in a launch of node elements of `sb` bytes, and whether a CTA has
// that much: not for double-double batches of more than ~45 photon pairs, which have no tree
static inline int tree_warp_elems(const TreeInst& T, int sb) {
  return tree_smem(T, (64 << 10) / (TREE_THREADS / 32) / sb);
}
static inline bool tree_fits(const TreeInst& T, int sb) {
  return (long long)tree_warp_elems(T, sb) * (TREE_THREADS / 32) * sb <= TREE_SMEM_BYTES;
}

// The program of one launch over `insts` (their levels placed one after another in the workspace):
// round r holds phase r of every instance, so that the narrow levels of one run beside others'.
// `nparts` advances by the leaves' partial slots; part_base[i] and part_count[i] are instance i's.
struct TreeProgram {
  std::vector<TreeInst> insts;
  std::vector<TreeRound> rounds;
  std::vector<TreeSeg> segs;
  long long ws_bytes = 0;
  int smem = 1;  // elements of a warp's shared memory
};

static inline void tree_program(std::vector<TreeInst>& insts, const std::vector<TreeLevels>& levels, int sb, int tile,
                                int chip_threads, int& nparts, std::vector<int>& part_base,
                                std::vector<int>& part_count, TreeProgram& P) {
  std::vector<std::vector<TreeSeg>> rounds;
  part_base.assign(insts.size(), 0);
  part_count.assign(insts.size(), 0);
  for (size_t k = 0; k < insts.size(); ++k) {
    TreeInst& T = insts[k];
    const TreeLevels& g = levels[k];
    T.scr_off = P.ws_bytes + g.scr_off;
    T.m_odd = (int)g.m_elems;
    P.smem = std::max(P.smem, tree_warp_elems(T, sb));
    size_t r = 0;
    int last = -1;
    auto add = [&](int phase, int q, int p0, int np, int ps) {
      TreeSeg s;
      memset(&s, 0, sizeof(s));
      s.par = P.ws_bytes + g.off[q];
      s.chi = phase == TP_ROOT ? s.par : P.ws_bytes + g.off[std::min(q + 1, T.steps)];
      s.inst = (int)k;
      s.np = np;
      s.p0 = p0;
      s.pstride = ps;
      s.phase = (unsigned char)phase;
      s.q = (unsigned char)q;
      if (tree_same_round(last, phase)) --r;
      last = phase;
      if (rounds.size() <= r) {
        rounds.emplace_back();
        rounds.back().reserve(insts.size());
      }
      rounds[r++].push_back(s);
    };
    if (T.steps > 0 && T.reps[0] == 1) {
      add(TP_FIRST, 0, 0, 1, 1);
      tree_walk(T, g, 1, 1, add);
    } else {
      add(TP_ROOT, 0, 0, 1, 1);
      tree_walk(T, g, 0, 1, add);
    }
    P.ws_bytes += g.bytes;
  }
  const bool dd = !insts.empty() && insts[0].comp_off > 0;
  std::vector<unsigned char> key;
  std::vector<int> order;
  size_t nsegs = 0;
  for (const auto& R : rounds) nsegs += R.size();
  P.segs.reserve(nsegs);
  // partial slots instance by instance, so that an instance's are contiguous
  for (auto& R : rounds) {
    // whole tiles when those fill the chip, else one coefficient a thread, else four threads each, or two
    // (a step's entries, when four would be more than a warp a sub-partition: fewer warps pay the sum over
    // the threads and the children's; double-double n = 24 305 -> 265 us, FP64 n = 24 84 -> 81, others within
    // 1 %; from a quarter of the chip on FP64 n = 22 72 -> 75)
    double whole = 0, split = 0;
    for (const TreeSeg& s : R) {
      whole += tree_items(insts[s.inst], s.phase, s.q, s.np, tile);
      split += tree_items(insts[s.inst], s.phase, s.q, s.np, 0);
    }
    // (half of it but for double-double, whose tiles are the longest chains: 64 photon patterns 518 ->
    // 498 us; double-double n = 28 630 -> 652)
    const int use = whole >= (dd ? 1.0 : 0.5) * chip_threads ? tile : (split > chip_threads ? 1 : 0);
    TreeRound rr;
    memset(&rr, 0, sizeof(rr));
    rr.seg0 = (int)P.segs.size();
    rr.nseg = (int)R.size();
    // the costly segments' warps first, by the exponent of their multiply-adds
    key.resize(R.size());
    order.resize(R.size());
    int at[64] = {0};
    for (size_t i = 0; i < R.size(); ++i) {
      const TreeSeg& s = R[i];
      ++at[key[i] = (unsigned char)(63 - std::min(std::ilogb(tree_macs(insts[s.inst], s.phase, s.q, s.np) + 1), 63))];
    }
    for (int b = 0, sum = 0; b < 64; ++b) {
      const int c = at[b];
      at[b] = sum;
      sum += c;
    }
    for (size_t i = 0; i < R.size(); ++i) order[at[key[i]]++] = (int)i;
    for (int i : order) {
      TreeSeg& s = R[i];
      const TreeInst& T = insts[s.inst];
      s.tile = (unsigned char)use;
      if (use == 1 && (s.phase == TP_W2 || s.phase == TP_MULTI2)) s.tile = (unsigned char)tile;
      if (use == 0 && s.phase == TP_UNIT && split > 0.35 * chip_threads) s.tile = TREE_PAIRS;
      long long warps = (long long)((tree_items(T, s.phase, s.q, s.np, s.tile) + 31) / 32);
      // leaves: at most the chip's warps, each with a partial for the reduction; the CTAs of a
      // single instance keep their sums over all leaf rounds and leave one partial each
      if (s.phase == TP_LEAF) {
        warps = std::max<long long>(std::min<long long>(warps, chip_threads / 32), 1);
        s.part = insts.size() > 1 ? part_count[s.inst] : 0;
        part_count[s.inst] = insts.size() > 1 ? part_count[s.inst] + (int)warps : chip_threads / TREE_THREADS;
      }
      s.warp0 = rr.nwarps;
      rr.nwarps += (int)std::max<long long>(warps, 1);
      P.segs.push_back(s);
    }
    P.rounds.push_back(rr);
  }
  for (size_t k = 0; k < insts.size(); ++k) {
    part_base[k] = nparts;
    nparts += part_count[k] * insts[k].pstride;
  }
  for (TreeSeg& s : P.segs)
    if (s.phase == TP_LEAF) s.part = part_base[s.inst] + s.part * insts[s.inst].pstride;
  P.insts = insts;
}

// Latency of a tree's rounds in edges of the per-term evaluation (8.4 us for plain FP64): a simple edge's
// one round, a double edge's two, the four of more photons with their root and exponential recurrences,
// chains of FP64 latencies.
static inline double tree_latency(const TreeInst& T) {
  double lat = 0;
  for (int q = 0; q < T.E; ++q) lat += T.reps[q] == 1 ? 0.7 : (T.reps[q] == 2 ? 2.0 : 4.0);
  return lat;
}
// a tree's multiply-adds, level by level (the blocks that large levels are walked in add up to the same;
// a level may have more nodes than an int holds)
static inline double tree_work(const TreeInst& T) {
  double macs = 0, nodes = 1;
  for (int q = 0; q <= T.steps; ++q) {
    tree_step(T, q, [&](int phase) { macs += tree_macs(T, phase, q, nodes); });
    if (q == T.steps) break;
    if (T.reps[q] == 1 && T.pL >= 0) macs += tree_macs(T, TP_G, q, nodes);
    nodes *= T.radix[q];
  }
  return macs;
}

// Whether one CTA does a launch's work sooner than the whole chip: the multiply-adds against the
// rounds, whose grid barrier and L2 latencies cost ~8000 clocks and one CTA's ~2500.
static inline bool tree_one_cta(const std::vector<TreeInst>& insts, const std::vector<TreeLevels>& levels, double clk,
                                int sms) {
  double macs = 0, rounds = 0;
  for (size_t k = 0; k < insts.size(); ++k) {
    const TreeInst& T = insts[k];
    double n = 0;
    int last = -1;
    auto add = [&](int phase, int q, int, int np, int) {
      macs += tree_macs(T, phase, q, np);
      n += !tree_same_round(last, phase);
      last = phase;
    };
    if (levels[k].phases > 200) return false;
    tree_walk(T, levels[k], 0, 1, add);
    rounds = std::max(rounds, n);
  }
  return 1.5 * macs * clk + 2500.0 * rounds <= macs * clk / sms + 8000.0 * rounds;
}

}  // namespace wg
