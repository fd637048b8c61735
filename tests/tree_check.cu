// Host check of the elimination tree (tree_kernel.cuh, tree_host.h): the node functions compiled
// for the host over a scalar type whose loads and stores are checked against the levels they belong
// to, run through the program that a launch of the kernel follows, for instances read from standard
// input.  Built and run by tests/test_tree_host.py; prints the outputs, or names the first access
// out of range.
//
// Input: instances level-budget-bytes tile chip-threads; per instance kind n E batch_max cutoff
// has_odd; edge_reps; A (n x n, re im); D (n); oddV (n); oddloop.  kind as in walrus_gb300.h (0 plain,
// 1 loop, 3 / 4 batch even / odd).
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <vector>

#include "../thewalrus_gb300/csrc/sieve_kernel.cuh"

namespace wg {

struct hc {
  double re, im;
};

template <>
struct Ar<hc> {
  using S = hc;
  static constexpr bool cplx = true, fp64 = true, modular = false, dd = false;
  using Comp = double;  // the device's warp reductions, compiled but not used here
  static constexpr int NC = 0;
  __device__ static Comp comp(const S& a, int) { return a.re; }
  __device__ static void set_comp(S&, int, Comp) {}
  __device__ static Comp cadd(Comp a, Comp b) { return a + b; }
  __device__ static Comp shfl_xor(Comp v, int) { return v; }
  __host__ __device__ static S zero() { return {0, 0}; }
  __host__ __device__ static S one() { return {1, 0}; }
  __host__ __device__ static S add(S a, S b) { return {a.re + b.re, a.im + b.im}; }
  __host__ __device__ static S sub(S a, S b) { return {a.re - b.re, a.im - b.im}; }
  __host__ __device__ static S neg(S a) { return {-a.re, -a.im}; }
  __host__ __device__ static S mul(S a, S b) { return {a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re}; }
  __host__ __device__ static S fma(S a, S b, S c) { return add(c, mul(a, b)); }
  __host__ __device__ static S scale(S a, double s) { return {a.re * s, a.im * s}; }
  __host__ __device__ static S scale_f(S a, float s) { return scale(a, s); }
  __host__ __device__ static S div_int(S a, int k) { return scale(a, 1.0 / k); }
  __host__ __device__ static S from_c64(c64 v) { return {v.re, v.im}; }
};

}  // namespace wg

#include "../thewalrus_gb300/csrc/tree_host.h"

using namespace wg;

static std::map<const hc*, size_t> g_bufs;  // start -> elements

static void check(const hc* p, const char* what) {
  auto it = g_bufs.upper_bound(p);
  if (it != g_bufs.begin()) {
    --it;
    if (p < it->first + it->second) return;
  }
  std::printf("FAIL %s out of range\n", what);
  std::exit(1);
}

namespace wg {
template <>
__host__ __device__ __forceinline__ hc tld<hc>(const hc* p) {
#ifndef __CUDA_ARCH__
  check(p, "load");
  if (std::isnan(p->re)) {
    std::printf("FAIL load of an element that was never stored\n");
    std::exit(1);
  }
#endif
  return *p;
}
template <>
__host__ __device__ __forceinline__ void tst<hc>(hc* p, hc v) {
#ifndef __CUDA_ARCH__
  check(p, "store");
#endif
  *p = v;
}
}  // namespace wg

static double rd() {
  double x;
  if (std::scanf("%lf", &x) != 1) std::exit(2);
  return x;
}

template <int TL>
static void phase(const TreeInst& T, const TreeSeg& G, const unsigned char* pool, const hc* par, hc* chi, hc* scr,
                  hc* sm, int smn, int tid, int nthr, hc* out) {
  hc* y = G.q < T.steps ? scr + 6ll * (T.deg[G.q + 1] + 1) * G.np * T.radix[G.q] : nullptr;
  switch (G.phase) {
    case TP_ROOT: tree_root<hc>(T, pool, chi, tid, nthr); break;
    case TP_FIRST: tree_first<hc>(T, pool, chi, tid, nthr); break;
    case TP_M: tree_m<hc, TL>(T, G.q, par, G.pstride, G.np, tree_m_of(T, scr, G.q), tid, nthr); break;
    case TP_UNIT: tree_unit<hc, TL>(T, G.q, par, G.pstride, G.np, chi, tid, nthr); break;
    case TP_G: tree_g<hc, TL>(T, G.q, par, G.pstride, G.np, tree_m_of(T, scr, G.q), chi, tid, nthr); break;
    case TP_G2:
      tree_g2<hc>(T, G.q, par, G.pstride, G.np, scr + (2ll * tree_width(T.X, T.E, G.q + 1)) * (T.deg[G.q] + 1) * G.np, chi,
                  sm, smn, tid, nthr);
      break;
    case TP_W2: tree_w2<hc, TL>(T, G.q, par, G.pstride, G.np, scr, tid, nthr); break;
    case TP_MULTI2: tree_multi2<hc, TL>(T, G.q, par, G.pstride, G.np, scr, chi, tid, nthr); break;
    case TP_PREP: tree_prep<hc>(T, G.q, par, G.pstride, G.np, scr, chi, sm, smn, tid, nthr); break;
    case TP_Y: tree_y<hc, TL>(T, G.q, par, G.pstride, G.np, scr, y, tid, nthr); break;
    case TP_MULTI: tree_multi<hc, TL>(T, G.q, par, G.pstride, G.np, y, chi, tid, nthr); break;
    case TP_GLOOP: tree_gloop<hc>(T, G.q, par, G.pstride, G.np, scr, y, chi, sm, smn, tid, nthr); break;
    default: {
      const hc s = tree_leaf<hc, TL>(T, par, G.pstride, G.np, tree_m_of(T, scr, G.q), sm, smn, tid, nthr);
      if (T.pB < 0) out[0] = Ar<hc>::add(out[0], s);
      else
        for (int k = 0; k < T.nout; ++k) out[k] = Ar<hc>::add(out[k], sm[k]);
    }
  }
}

int main(int argc, char**) {  // with an argument: multiple edges as simple ones
  const int count = (int)rd();
  const double budget = rd();
  const int tile = (int)rd(), chip = (int)rd();  // as tree_program's
  std::vector<TreeInst> insts(count);
  std::vector<TreeLevels> levels(count);
  std::vector<std::vector<hc>> exts(count);
  for (int k = 0; k < count; ++k) {
    InstDev d;
    memset(&d, 0, sizeof(d));
    const int kind = (int)rd(), n = (int)rd(), E = (int)rd(), bm = (int)rd(), cut = (int)rd(), odd = (int)rd();
    d.kind = kind == 1 && odd ? KIND_LOOP_ODD : kind;
    d.n = n;
    d.lda = n + 1;
    d.glynn = 1;
    d.nout = 1;
    if (kind >= 3) {
      d.reps[d.E++] = bm;
      if (kind == 4) d.reps[d.E++] = 1;
      d.nout = 2 * bm + cut + (kind == 4 ? 2 : 1);
    }
    for (int e = 0; e < E; ++e) d.reps[d.E++] = (int)rd();
    exts[k].assign((size_t)(n + 3) * (n + 1), hc{0, 0});
    auto at = [&](int r, int c) -> hc& { return exts[k][(size_t)r * (n + 1) + c]; };
    for (int r = 0; r < n; ++r)
      for (int c = 0; c < n; ++c) { const double re = rd(); at(r, c) = {re, rd()}; }
    for (int i = 0; i < n; ++i) { const double re = rd(); at(i, n) = at(n, i) = {re, rd()}; }
    for (int i = 0; i < n; ++i) { const double re = rd(); at(n + 1, i) = {re, rd()}; }
    d.oddloop.re = rd();
    d.oddloop.im = rd();
    if (!(argc > 1 && tree_build(d, insts[k], true)) && !tree_build(d, insts[k])) { std::printf("FAIL no tree\n"); return 1; }
    insts[k].pstride = insts[k].nout;
    tree_levels(insts[k], sizeof(hc), budget, levels[k]);
  }
  TreeProgram P;
  std::vector<int> base, cnt;
  int nparts = 0;
  tree_program(insts, levels, sizeof(hc), tile, chip, nparts, base, cnt, P);
  std::vector<hc> ws((size_t)P.ws_bytes / sizeof(hc), hc{NAN, NAN}), sm(P.smem);
  std::vector<int> slots(nparts, 0);
  std::vector<std::vector<hc>> out(count);
  for (int k = 0; k < count; ++k) out[k].assign(P.insts[k].nout, hc{0, 0});
  unsigned char* w = reinterpret_cast<unsigned char*>(ws.data());
  for (const TreeRound& R : P.rounds)
    for (int k = 0; k < R.nseg; ++k) {
      // a round's segments run side by side: last to first here for one of the sizes
      const int g = chip == 64 ? R.seg0 + R.nseg - 1 - k : R.seg0 + k;
      const TreeSeg& G = P.segs[g];
      const TreeInst& T = P.insts[G.inst];
      const TreeLevels& L = levels[G.inst];
      const int end = g + 1 < R.seg0 + R.nseg ? P.segs[g + 1].warp0 : R.nwarps, warps = end - G.warp0;
      if (warps < 1) { std::printf("FAIL segment without warps\n"); return 1; }
      // what the segment may touch: its two levels, its scratch
      const long long l0 = T.scr_off - L.scr_off;
      auto range = [&](long long off, long long elems) { g_bufs[reinterpret_cast<hc*>(w + off)] = (size_t)elems; };
      g_bufs.clear();
      g_bufs[sm.data()] = sm.size();
      range(l0 + L.off[G.q], L.cap[G.q] * tree_node_elems(T, G.q));
      if (G.q < T.steps) range(l0 + L.off[G.q + 1], L.cap[G.q + 1] * tree_node_elems(T, G.q + 1));
      range(T.scr_off, (L.bytes - L.scr_off) / (long long)sizeof(hc));
      const hc* par = reinterpret_cast<const hc*>(w + G.par) + G.p0;
      hc *chi = reinterpret_cast<hc*>(w + G.chi), *scr = reinterpret_cast<hc*>(w + T.scr_off);
      const unsigned char* pool = reinterpret_cast<const unsigned char*>(exts[G.inst].data());
      // chip 32: the phases that do not stage their series in shared memory
      const int smn = chip > 32 ? P.smem : (T.pB >= 0 ? 5 * (T.deg[T.steps] + 1) + 32 : 0);
      // every lane of the segment's warps as one thread (warp-wide phases: a warp of one lane)
      const bool wide = G.phase == TP_PREP || G.phase == TP_GLOOP || G.phase == TP_G2 || (G.phase == TP_LEAF && T.pB >= 0);
      const int nthr = wide ? warps : warps * 32;
      for (int t = 0; t < nthr; ++t) {
        if (G.tile == 0 || G.tile == TREE_PAIRS) phase<0>(T, G, pool, par, chi, scr, sm.data(), smn, t, nthr, out[G.inst].data());
        else if (G.tile == 1) phase<1>(T, G, pool, par, chi, scr, sm.data(), smn, t, nthr, out[G.inst].data());
        else phase<4>(T, G, pool, par, chi, scr, sm.data(), smn, t, nthr, out[G.inst].data());
      }
      if (G.phase == TP_LEAF && count > 1)
        for (int x = 0; x < warps * T.pstride; ++x)
          if (slots.at(G.part + x)++) { std::printf("FAIL partial slot used twice\n"); return 1; }
    }
  for (int x : slots)
    if (!x && count > 1) { std::printf("FAIL partial slot never written\n"); return 1; }
  for (int k = 0; k < count; ++k) {
    const double scale = std::ldexp(1.0, -tree_scale_exp(P.insts[k]));
    for (const hc& z : out[k]) std::printf("%.17g %.17g\n", z.re * scale, z.im * scale);
  }
  return 0;
}
