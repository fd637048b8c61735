// Host check of the elimination tree (tree_kernel.cuh, tree_host.h): the node functions compiled
// for the host over a scalar type whose loads and stores are checked against their buffers, walked
// both ways the kernels are launched (a CTA's path and subtree for every task, and level by level in
// blocks), for one instance read from standard input.  Built and run by tests/test_tree_host.py;
// prints each output twice, or names the first access out of range.
//
// Input: kind n E batch_max cutoff has_odd K-budget-bytes task-split; edge_reps; A (n x n, re im);
// D (n); oddV (n); oddloop.  kind as in walrus_gb300.h (0 plain, 1 loop, 3 / 4 batch even / odd).
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

struct Buf {
  std::vector<hc> v;
  explicit Buf(size_t n) : v(n, hc{NAN, NAN}) { g_bufs[v.data()] = n; }
  ~Buf() { g_bufs.erase(v.data()); }
  hc* p() { return v.data(); }
};

static double rd() {
  double x;
  if (std::scanf("%lf", &x) != 1) std::exit(2);
  return x;
}

static void leaf(const TreeInst& T, hc* par, long long ps, int np, hc* m, std::vector<hc>& out) {
  Buf sm(5 * (T.deg[T.steps] + 1) + 32);
  const hc s = tree_leaf<hc>(T, par, ps, np, m, sm.p(), 0, 0, 1);
  if (T.pB < 0) out[0] = Ar<hc>::add(out[0], s);
  else
    for (int k = 0; k < T.nout; ++k) out[k] = Ar<hc>::add(out[k], sm.p()[5 * (T.deg[T.steps] + 1) + k]);
}

int main() {
  InstDev d;
  memset(&d, 0, sizeof(d));
  const int kind = (int)rd(), n = (int)rd(), E = (int)rd(), bm = (int)rd(), cut = (int)rd(), odd = (int)rd();
  const double budget = rd();
  const int split = (int)rd();
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
  Buf ext((size_t)(n + 3) * (n + 1));
  for (auto& x : ext.v) x = {0, 0};
  auto at = [&](int r, int c) -> hc& { return ext.v[(size_t)r * (n + 1) + c]; };
  for (int r = 0; r < n; ++r)
    for (int c = 0; c < n; ++c) { const double re = rd(); at(r, c) = {re, rd()}; }
  for (int i = 0; i < n; ++i) { const double re = rd(); at(i, n) = at(n, i) = {re, rd()}; }
  for (int i = 0; i < n; ++i) { const double re = rd(); at(n + 1, i) = {re, rd()}; }
  d.oddloop.re = rd();
  d.oddloop.im = rd();

  TreeInst T;
  if (!tree_build(d, T)) { std::printf("FAIL no tree\n"); return 1; }
  const unsigned char* pool = reinterpret_cast<const unsigned char*>(ext.p());
  const double scale = std::ldexp(1.0, -tree_scale_exp(T));
  std::vector<hc> a(T.nout, hc{0, 0}), b = a;

  // every task of the CTA kernel: its path, then its subtree
  T.q = std::min(split, T.steps);
  long long el[3], tasks = 1;
  for (int q = 0; q < T.q; ++q) tasks *= T.radix[q];
  tree_cta_elems(T, T.q, el);
  for (long long t = 0; t < tasks; ++t) {
    Buf b0(el[0]), b1(std::max<long long>(el[1], 1)), sc(std::max<long long>(el[2], 1));
    hc* buf[2] = {b0.p(), b1.p()};
    long long code = t;
    tree_root<hc>(T, pool, buf[0], 0, 1);
    int cur = 0, np = 1;
    for (int q = 0; q < T.steps; ++q) {
      const int R = T.radix[q];
      int d0 = 0, nd = R;
      if (q < T.q) { d0 = (int)(code % R); code /= R; nd = 1; }
      hc *par = buf[cur], *chi = buf[cur ^ 1];
      if (T.reps[q] == 1) {
        if (T.pL >= 0) tree_m<hc>(T, q, par, np, np, sc.p(), 0, 1);
        tree_unit<hc>(T, q, par, np, np, sc.p(), chi, d0, nd, 0, 1);
      } else {
        hc* y = sc.p() + 6ll * (T.deg[q + 1] + 1) * np * nd;
        tree_prep<hc>(T, q, par, np, np, sc.p(), chi, d0, nd, 0, 1);
        if (tree_width(T.X, T.E, q + 1) > 0) {
          tree_y<hc>(T, q, par, np, np, sc.p(), y, nd, 0, 1);
          tree_multi<hc>(T, q, par, np, np, y, chi, nd, 0, 1);
          if (T.pL >= 0) tree_gloop<hc>(T, q, par, np, np, sc.p(), y, chi, d0, nd, 0, 1);
        }
      }
      np *= nd;
      cur ^= 1;
    }
    if (T.steps < T.E && T.pO >= 0) tree_m<hc>(T, T.steps, buf[cur], np, np, sc.p(), 0, 1);
    leaf(T, buf[cur], np, np, sc.p(), a);
  }

  // level by level
  TreeGridPlan g;
  tree_grid_plan(T, sizeof(hc), budget, g);
  std::vector<Buf*> lev;
  for (int q = 0; q <= T.steps; ++q) lev.push_back(new Buf((size_t)(g.cap[q] * tree_node_elems(T, q))));
  Buf sc((size_t)(g.bytes - g.scr_off) / sizeof(hc));
  long long launches = 1;
  auto launch = [&](int phase, int q, int p0, int np, int ps, int d0, int nd) {
    ++launches;
    hc *par = lev[q]->p() + p0, *chi = q < T.steps ? lev[q + 1]->p() : nullptr;
    hc* y = q < T.steps ? sc.p() + 6ll * (T.deg[q] + 1 + T.reps[q]) * np * nd : nullptr;
    switch (phase) {
      case TP_M: tree_m<hc>(T, q, par, ps, np, sc.p(), 0, 1); break;
      case TP_UNIT: tree_unit<hc>(T, q, par, ps, np, sc.p(), chi, d0, nd, 0, 1); break;
      case TP_PREP: tree_prep<hc>(T, q, par, ps, np, sc.p(), chi, d0, nd, 0, 1); break;
      case TP_Y: tree_y<hc>(T, q, par, ps, np, sc.p(), y, nd, 0, 1); break;
      case TP_MULTI: tree_multi<hc>(T, q, par, ps, np, y, chi, nd, 0, 1); break;
      case TP_GLOOP: tree_gloop<hc>(T, q, par, ps, np, sc.p(), y, chi, d0, nd, 0, 1); break;
      default: leaf(T, par, ps, np, sc.p(), b);
    }
  };
  tree_root<hc>(T, pool, lev[0]->p(), 0, 1);
  tree_walk(T, g, 0, 1, launch);
  if (launches != g.launches) { std::printf("FAIL launch count\n"); return 1; }
  for (int k = 0; k < T.nout; ++k)
    std::printf("%.17g %.17g %.17g %.17g\n", a[k].re * scale, a[k].im * scale, b[k].re * scale, b[k].im * scale);
  for (auto* x : lev) delete x;
  return 0;
}
