// Device side of the elimination tree: the finite-difference sieve summed edge by edge.
//
// The sieve writes a hafnian as a sum over the edges' sign vectors delta of
//   prod_e w_e(delta_e) [eta^K] F(eta delta),   F = det(I - X C)^(-1/2) exp(v^T (X^-1 - C)^-1 v / 2),
// X the edges' pairing scaled by eta delta_e.  F is a Gaussian integral over the paired vertices, so
// it can be taken one edge at a time: eliminating edge e = (i, j) leaves a smaller problem of the
// same kind on the other vertices, whose matrix entries are power series in eta (one power per
// delta), and the sum over delta_1 .. delta_E is a tree whose nodes at depth q share everything
// that depends on the first q signs.  Almost all nodes are near the leaves, where the matrices
// are 4 x 4 and 6 x 6: one n = 40 complex term costs 57,690 multiply-adds by itself (a Hessenberg
// reduction per term) and 1,330 as its share of the tree.
//
// Simple edges (multiplicity 1) need F only to first order in delta_e: higher powers belong to
// terms that use an edge twice, and at total degree K some other edge is then not used at all and
// its signs cancel.  The step is
//   C_ab' = C_ab + delta eta (C_ia C_jb + C_ja C_ib),   g' = g (1 + delta eta (C_ij + v_i v_j)),
// with v as one more row of C (position pL), and both signs share the products.  No divisions and
// no pivots.  Double edges go to second order likewise (tree_w2); higher multiplicities take the
// whole 2 x 2 block, P = (X_e^-1 - C_ee)^-1:
//   C' = C + C_re P C_er,   g' = g det(I - X_e C_ee)^(-1/2) exp(v_e^T P v_e / 2).
// delta -> -delta leaves a term's share unchanged (degree K in the deltas, as the weights), so
// the first edge takes half of its signs.  The last simple edges close: two of them in the hafnian
// of the 4 vertices left (their four sign pairs' sum), with loop weights one in C_ij + v_i v_j.
//
// What bounds it: the FP64 pipe (2 multiply-adds per clock and SM), i.e. the number of FP64 warp
// instructions; loads are a few bytes per clock even from L2.  So lanes are nodes (p fastest: the
// same entry and coefficients of 32 nodes, no idle lanes below the top few levels) and every
// thread forms tree_tile() consecutive coefficients of one entry in registers.  The levels are rounds
// of one cooperative launch with a barrier after each (2,400 clocks): the narrow ones, a few thousand
// clocks of FP64 and L2 latency, bound trees of up to ~14 pairs, the FP64 pipe (77 % busy at n = 34)
// the larger ones.  Measured against the per-term kernel (us a call): complex n = 24 576 -> 96, n = 40
// 244,600 -> 4,840; real n = 44 (positive) 380,900 -> 7,980; loops n = 27 2,320 -> 145; 96 matrices of
// n = 8 .. 32 in a plan 61,850 -> 1,720; complex n = 28 in double-double 22,300 -> 716, n = 34 in
// double-float 12,380 -> 443; the exact count of a graph of 32 vertices 9,100 -> 338.
// (The reference's tree for unit edges is thewalrus/_hafnian.py recursive_hafnian's squeeze; this
// one sums the finite-difference signs of _calc_hafnian / _calc_loop_hafnian, :443-577, and of
// loop_hafnian_batch.py:50-208.)
#pragma once
#include "sieve_kernel.cuh"

namespace wg {

constexpr int TREE_MAX_K = 63;
constexpr int TREE_MAX_POS = 3 + 2 * MAX_EDGES;
constexpr int TREE_THREADS = 512;  // one CTA per SM

// The node functions also compile for the host, one thread as a warp of one lane: a CPU check runs
// them over a checked scalar type (tests/tree_check.cu).
#ifdef __CUDA_ARCH__
#define WG_TREE_LANES 32
#define WG_TREE_SPLIT 4
#define WG_TREE_SYNCWARP() __syncwarp()
#else
#define WG_TREE_LANES 1
#define WG_TREE_SPLIT 1
#define WG_TREE_SYNCWARP() ((void)0)
#endif

// Coefficients a thread forms in registers (TL below): more of them share a load, but a level with
// fewer tiles than threads leaves the chip idle, so narrower levels take one coefficient a thread and
// the narrowest four threads a coefficient (TL = 0), whose chain of loads and FP64 instructions is the
// level's time.  Residues, one register each, take four (n = 40 999 -> 878 us, n = 36 257 -> 244, n = 32 as with
// three); four or more cost the others: double-float n = 34 316 -> 331 us, real n = 32 144 -> 149 (five).
template <class S>
__host__ __device__ constexpr int tree_tile() { return Ar<S>::modular ? 4 : (Ar<S>::dd && Ar<S>::cplx ? 2 : 3); }
__host__ __device__ __forceinline__ int tree_tiles(int L, int TL) { return (L + TL - 1) / TL; }

// One instance's tree.  Positions 0 .. X-1 are the rows that are never eliminated (pL: the loop
// weights, pO: an unpaired vertex, pB: the batch mode), then the edges' vertices, the last edge
// first: step q eliminates positions X + 2 (E-1-q) and the next, the highest two left.
struct alignas(16) TreeInst {
  long long a_off;           // byte offset of the extended matrix in the pool
  long long scr_off;         // of the instance's scratch in the workspace
  int lda;
  int E, K, X;
  int pL, pO, pB;            // -1: none
  int diag;                  // entries include the diagonal (multiple edges, or a batch mode)
  int dpos;                  // diagonal entries of positions >= dpos are kept (pending multiple edges)
  int steps;                 // edges eliminated by steps: E, E - 1 or E - 2 (tree_leaf's closed forms)
  int nout;
  int pstride, comp_off;     // partial slots of a leaf warp (as InstDev's)
  int m_odd;                 // loop kinds: scratch element from which odd steps keep m (even ones: 0)
  c64 oddloop;               // entry (pO, pL) when the unpaired vertex is not a vertex of A
  signed char row[TREE_MAX_POS], col[TREE_MAX_POS];  // position -> row and column of the extended matrix
  unsigned char reps[MAX_EDGES], radix[MAX_EDGES];
  unsigned char deg[MAX_EDGES + 4];  // degree of the series after q steps
};

constexpr int TREE_PAIRS = 255;  // a segment's tile: two threads a coefficient (TP_UNIT)

// The program of a launch: rounds of segments, with a barrier of the whole launch after each round.
// A segment is one phase of one step of one instance over a block of parents [p0, p0 + np) of a
// level of pstride nodes, by the round's warps [warp0, next segment's warp0).
// A loop kind's simple edge needs m = C_ij + v_i v_j as a series (TP_M) before its children's g (TP_G),
// which nothing reads before the next step's TP_G: so that TP_M stands in the round of the other
// entries (TP_UNIT) and TP_G in the round after it, beside the next step.  (A round of its own for
// TP_M: loop n = 27 160 us, 131 so; n = 21 93 and 81.)
enum TreePhase : int { TP_ROOT = 0, TP_FIRST, TP_M, TP_UNIT, TP_G, TP_PREP, TP_Y, TP_MULTI, TP_GLOOP, TP_W2, TP_G2, TP_MULTI2, TP_LEAF };
struct alignas(16) TreeSeg {
  long long par, chi;        // workspace byte offsets of the parents' and the children's level
  int inst, warp0;
  int np, p0, pstride;
  int part;                  // leaf: the first warp's partial slot (one instance: the first CTA's)
  unsigned char phase, q, tile;  // tile: coefficients a thread, 0: four threads a coefficient
  unsigned char pad[5];
};
struct alignas(16) TreeRound {
  int seg0, nseg, nwarps, pad;
};

static_assert(sizeof(TreeInst) % 16 == 0 && sizeof(TreeSeg) % 16 == 0 && sizeof(TreeRound) % 16 == 0,
              "programs are copied in 16-byte words");

// the final reduction's arguments, when a plan's only launch does it (done != nullptr)
struct TreeFinish {
  const InstDev* inst;
  const double2* partials;
  const double* scales;
  double2* out;
  double* mags;
  int* err;
  unsigned int *done, *counters;
  int ninst, first_out, end_out, ncounters, wpo;  // wpo: warps per output
};

struct TreeParams {
  const TreeInst* inst;
  const TreeRound* rounds;
  const TreeSeg* segs;
  int ninst, nrounds, nsegs;
  int cached;                // instances, rounds and segments are copied to shared memory first
  int sm_warp, sm_cache;     // shared memory: elements of a warp's work, byte offset of the cache
  int sm_ws;                 // shared memory: offset of the workspace (one CTA; 0: ws)
  const unsigned char* pool;
  unsigned char* ws;
  double2* partials;
  unsigned int* bar;
  unsigned int polls;        // of a barrier before a CTA gives up
  int* err;
  TreeFinish fin;
};

// trees modulo several primes side by side in one launch, whose CTAs they share in equal parts
struct TreeMods {
  int n;
  int prime[MOD_N];  // indices
  TreeParams p[MOD_N];
};

__host__ __device__ __forceinline__ int tree_width(int X, int E, int q) { return X + 2 * (E - q); }
__host__ __device__ __forceinline__ int tree_entries(int W, int diag) {
  return 1 + (diag ? W * (W + 1) / 2 : W * (W - 1) / 2);
}
// entry 0 is g; (a, b) with a >= b (a > b without the diagonal) follows
__host__ __device__ __forceinline__ int tree_ent(int a, int b, int diag) {
  return 1 + (diag ? a * (a + 1) / 2 : a * (a - 1) / 2) + b;
}
__host__ __device__ __forceinline__ int tree_ent2(int a, int b, int diag) {
  return a > b ? tree_ent(a, b, diag) : tree_ent(b, a, diag);
}
// where step q keeps its m
template <class S>
__host__ __device__ __forceinline__ S* tree_m_of(const TreeInst& T, S* scr, int q) { return scr + (q & 1 ? T.m_odd : 0); }
__host__ __device__ __forceinline__ void tree_decode(int e, int diag, int& a, int& b) {
  const int x = e - 1;
  int r = (int)((sqrtf(8.0f * (float)x + 1.0f) - 1.0f) * 0.5f);
  while ((r + 1) * (r + 2) / 2 <= x) ++r;
  while (r * (r + 1) / 2 > x) --r;
  a = diag ? r : r + 1;
  b = x - r * (r + 1) / 2;
}

// The running sum of real products.  Double-float and double-double sums stay unnormalised until
// they are read: a product's error terms and the two-sum's join the low part, which takes 12
// instructions a product where the scalar types' fma, which renormalises every time, takes 15.
template <class R>
struct RealAcc {
  R v;
#pragma nv_exec_check_disable
  __host__ __device__ static __forceinline__ RealAcc of(R x) { return {x}; }
#pragma nv_exec_check_disable
  __host__ __device__ __forceinline__ void fma(R a, R b) { v = Ar<R>::fma(a, b, v); }
#pragma nv_exec_check_disable
  __host__ __device__ __forceinline__ R sum() const { return v; }
};
template <>
struct RealAcc<dfr> {
  float hi, lo;
  __device__ static __forceinline__ RealAcc of(dfr x) { return {x.hi, x.lo}; }
  __device__ __forceinline__ void fma(dfr a, dfr b) {
    const float p = a.hi * b.hi;
    float e = fmaf(a.hi, b.hi, -p);
    e = fmaf(a.hi, b.lo, e);
    e = fmaf(a.lo, b.hi, e);
    const dfr s = df_two_sum(hi, p);
    hi = s.hi;
    lo += s.lo + e;
  }
  __device__ __forceinline__ dfr sum() const { return df_two_sum(hi, lo); }
};
template <>
struct RealAcc<ddr> {
  double hi, lo;
  __device__ static __forceinline__ RealAcc of(ddr x) { return {x.hi, x.lo}; }
  __device__ __forceinline__ void fma(ddr a, ddr b) {
    const double p = a.hi * b.hi;
    double e = ::fma(a.hi, b.hi, -p);
    e = ::fma(a.hi, b.lo, e);
    e = ::fma(a.lo, b.hi, e);
    const ddr s = dd_two_sum(hi, p);
    hi = s.hi;
    lo += s.lo + e;
  }
  __device__ __forceinline__ ddr sum() const { return dd_two_sum(hi, lo); }
};
// Complex nodes as the matrix's own scalar: four real products a term, each part rounded relative to
// its own terms.
template <class R, class C>
struct RealAccParts {
  RealAcc<R> re, im;
  __device__ __forceinline__ void fma(C a, C b) {
    re.fma(a.re, b.re);
    re.fma(Ar<R>::neg(a.im), b.im);
    im.fma(a.re, b.im);
    im.fma(a.im, b.re);
  }
  __device__ __forceinline__ C sum() const { return {re.sum(), im.sum()}; }
};
template <>
struct RealAcc<cdf> : RealAccParts<dfr, cdf> {
  __device__ static __forceinline__ RealAcc of(cdf x) { return {{RealAcc<dfr>::of(x.re), RealAcc<dfr>::of(x.im)}}; }
};
template <>
struct RealAcc<cdd> : RealAccParts<ddr, cdd> {
  __device__ static __forceinline__ RealAcc of(cdd x) { return {{RealAcc<ddr>::of(x.re), RealAcc<ddr>::of(x.im)}}; }
};
// Or with re + im beside the parts, so that a product of series takes three real products a term
// instead of four (re = P1 - P2, im = P3 - P1 - P2 with P1 = sum re re, P2 = sum im im, P3 = sum
// (re + im)(re + im)).  Its rounding is relative to |a| |b|: each part keeps its accuracy only where the
// parts are of like size, so that the host takes it for matrices whose rows say so (mixed_rows,
// sieve.cu) and the four products for the others.  C: the matrix scalar, R: its real one.  FP64 n = 40:
// 5,836 -> 5,405 us, n = 36: 1,212 -> 1,147 us.
template <class R, class C>
struct c3 {
  R re, im, s;
};
template <class R, class C>
struct Ar<c3<R, C>> {
  using S = c3<R, C>;
  using B = Ar<R>;
  using Comp = typename Ar<C>::Comp;
  static constexpr int NC = 2;
  static constexpr bool cplx = true, fp64 = B::fp64, modular = false, dd = B::dd;
  __device__ static __forceinline__ S of(R re, R im) { return {re, im, B::add(re, im)}; }
  __device__ static __forceinline__ S of(C z) { return of(z.re, z.im); }
  __device__ static __forceinline__ C to(S a) { return {a.re, a.im}; }
  __device__ static __forceinline__ S zero() { return {B::zero(), B::zero(), B::zero()}; }
  __device__ static __forceinline__ S one() { return {B::one(), B::zero(), B::one()}; }
  __device__ static __forceinline__ S add(S a, S b) { return of(B::add(a.re, b.re), B::add(a.im, b.im)); }
  __device__ static __forceinline__ S sub(S a, S b) { return of(B::sub(a.re, b.re), B::sub(a.im, b.im)); }
  __device__ static __forceinline__ S neg(S a) { return {B::neg(a.re), B::neg(a.im), B::neg(a.s)}; }
  __device__ static __forceinline__ S mul(S a, S b) { return of(Ar<C>::mul(to(a), to(b))); }
  __device__ static __forceinline__ S fma(S a, S b, S c) { return of(Ar<C>::fma(to(a), to(b), to(c))); }
  __device__ static __forceinline__ S scale(S a, double s) { return of(B::scale(a.re, s), B::scale(a.im, s)); }
  __device__ static __forceinline__ S scale_f(S a, float s) { return of(B::scale_f(a.re, s), B::scale_f(a.im, s)); }
  __device__ static __forceinline__ S div_int(S a, int k) { return of(B::div_int(a.re, k), B::div_int(a.im, k)); }
  __device__ static __forceinline__ S from_c64(c64 v) { return of(Ar<C>::from_c64(v)); }
  __device__ static __forceinline__ c64 to_c64(S a) { return Ar<C>::to_c64(to(a)); }
  __device__ static __forceinline__ c64 lo_c64(S a) { return Ar<C>::lo_c64(to(a)); }
  __device__ static __forceinline__ Comp comp(const S& a, int i) { return i ? a.im : a.re; }
  __device__ static __forceinline__ void set_comp(S& a, int i, Comp v) {  // parts in order
    if (i) a = of(a.re, v); else a.re = v;
  }
  __device__ static __forceinline__ Comp cadd(Comp a, Comp b) { return Ar<C>::cadd(a, b); }
  __device__ static __forceinline__ Comp shfl_xor(Comp v, int m) { return Ar<C>::shfl_xor(v, m); }
};
// the node scalar of a matrix scalar, and back
template <class M>
struct TreeScalar {
  using T = M;
};
template <>
struct TreeScalar<c64> {
  using T = c3<double, c64>;
};
template <>
struct TreeScalar<cdf> {
  using T = c3<dfr, cdf>;
};
template <>
struct TreeScalar<cdd> {
  using T = c3<ddr, cdd>;
};
template <class S>
struct TreeMatrix {
  using T = S;
  __host__ __device__ static __forceinline__ S load(const S* p) { return *p; }
};
template <class R, class C>
struct TreeMatrix<c3<R, C>> {
  using T = C;
  __device__ static __forceinline__ c3<R, C> load(const C* p) { return Ar<c3<R, C>>::of(*p); }
};

// the running sum of a series product
template <class S>
struct ConvAcc : RealAcc<S> {
  using U = S;  // the sum as an addend
#pragma nv_exec_check_disable
  __host__ __device__ static __forceinline__ ConvAcc of(S x) { return {RealAcc<S>::of(x)}; }
#pragma nv_exec_check_disable
  __host__ __device__ __forceinline__ U parts() const { return this->sum(); }
#pragma nv_exec_check_disable
  __host__ __device__ static __forceinline__ S plus(S c, U u) { return Ar<S>::add(c, u); }
};
template <class R, class C>
struct ConvAcc<c3<R, C>> {
  RealAcc<R> p1, p2, p3;
  __device__ static __forceinline__ ConvAcc of(c3<R, C> x) {
    return {RealAcc<R>::of(x.re), RealAcc<R>::of(Ar<R>::zero()), RealAcc<R>::of(x.s)};
  }
  __device__ __forceinline__ void fma(c3<R, C> a, c3<R, C> b) {
    p1.fma(a.re, b.re);
    p2.fma(a.im, b.im);
    p3.fma(a.s, b.s);
  }
  using U = C;  // without re + im, which an addend does not need (an FP64 instruction a sum)
  __device__ __forceinline__ U parts() const {
    const R x = p1.sum(), y = p2.sum();
    return {Ar<R>::sub(x, y), Ar<R>::sub(Ar<R>::sub(p3.sum(), x), y)};
  }
  __device__ __forceinline__ c3<R, C> sum() const { return Ar<c3<R, C>>::of(parts()); }
  __device__ static __forceinline__ c3<R, C> plus(c3<R, C> c, U u) {
    return Ar<c3<R, C>>::of(Ar<R>::add(c.re, u.re), Ar<R>::add(c.im, u.im));
  }
};

// Sums over leaves.  Within a phase a thread adds its few (a level's 200 MB over the chip's threads: at
// most 20) in the node's scalar, as a term's coefficients are.  Beyond it FP64 and double-float leaves are
// added in FP64, a warp's phases with Neumaier's compensation, as the per-term kernel adds its terms;
// double-double and residue sums stay in their own scalar.  V: what is added up and stored.
template <class S>
struct Leaf {
  using V = S;
  static constexpr bool compensated = false;
  __device__ static __forceinline__ V of(S x) { return x; }
};
template <class S, class Val>
struct LeafFp {
  using V = Val;
  static constexpr bool compensated = true;
  __device__ static __forceinline__ V of(S x) {
    if constexpr (Ar<S>::cplx) return Ar<S>::to_c64(x);
    else return Ar<S>::to_c64(x).re;
  }
};
template <> struct Leaf<double> : LeafFp<double, double> {};
template <> struct Leaf<dfr> : LeafFp<dfr, double> {};
template <> struct Leaf<c64> : LeafFp<c64, c64> {};
template <> struct Leaf<cdf> : LeafFp<cdf, c64> {};
template <> struct Leaf<c3<double, c64>> : LeafFp<c3<double, c64>, c64> {};
template <> struct Leaf<c3<dfr, cdf>> : LeafFp<c3<dfr, cdf>, c64> {};

// The sums of a single instance's leaves, output k of a warp at [warp][k], in shared memory: they are
// touched once a leaf phase, and registers kept for them through all the others cost spills.
template <class S>
struct LeafSums {
  using V = typename Leaf<S>::V;
  V s[TREE_THREADS / 32][32], c[Leaf<S>::compensated ? TREE_THREADS / 32 : 1][32];
  __device__ __forceinline__ void begin(int w, int k, V x) {
    s[w][k] = x;
    if constexpr (Leaf<S>::compensated) c[w][k] = Ar<V>::zero();
  }
  __device__ __forceinline__ void add(int w, int k, V x) {
    if constexpr (!Leaf<S>::compensated) {
      s[w][k] = Ar<V>::add(s[w][k], x);
    } else if constexpr (Ar<V>::cplx) {
      neumaier(s[w][k].re, c[w][k].re, x.re);
      neumaier(s[w][k].im, c[w][k].im, x.im);
    } else {
      neumaier(s[w][k], c[w][k], x);
    }
  }
  __device__ __forceinline__ V value(int w, int k) const {
    if constexpr (Leaf<S>::compensated) return Ar<V>::add(s[w][k], c[w][k]);
    else return s[w][k];
  }
};

// loads and stores of node elements (the host check counts them)
template <class S>
__host__ __device__ __forceinline__ S tld(const S* p) { return *p; }
template <class S>
__host__ __device__ __forceinline__ void tst(S* p, S v) { *p = v; }

// acc[k] += sum_s a_s b_(t0+k-s), k < T, s < la: coefficients t0 .. t0+T-1 of a product of two
// series (element stride sa, sb).  A window of T coefficients of b slides through registers, so a
// step is one load of each series and T multiply-adds; the last T-1 steps are the triangle where b
// runs out.  t0 < 0: only the coefficients t0 + k >= 0.  b has lb coefficients.
#pragma nv_exec_check_disable
template <class S, int T>
__host__ __device__ __forceinline__ void conv_tile(ConvAcc<S> (&acc)[T], const S* a, long long sa, int la, const S* b,
                                          long long sb, int t0, int lb = 1 << 30) {
  if (t0 < 0) {
#pragma unroll
    for (int k = 1; k < T; ++k) {
      const int t = t0 + k;
      if (t >= 0)
        for (int s = t < lb ? 0 : t - lb + 1; s <= t && s < la; ++s) acc[k].fma(tld(a + s * sa), tld(b + (t - s) * sb));
    }
    return;
  }
  S w[T];
#pragma unroll
  for (int k = 0; k < T; ++k) w[k] = t0 + k < lb ? tld(b + (t0 + k) * sb) : Ar<S>::zero();
  const int n = t0 < la ? t0 : la;  // steps that slide the window
  const S* pa = a;
  const S* pb = b + (t0 - 1) * sb;
#pragma unroll 4
  for (int s = 0; s < n; ++s) {
    const S x = tld(pa), y = tld(pb);
    pa += sa;
    pb -= sb;
#pragma unroll
    for (int k = 0; k < T; ++k) acc[k].fma(x, w[k]);
#pragma unroll
    for (int k = T - 1; k > 0; --k) w[k] = w[k - 1];
    w[0] = y;
  }
  // s = t0 + kk: w[k] = b_k here
#pragma unroll
  for (int kk = 0; kk < T; ++kk) {
    if (t0 + kk < la) {
      const S x = tld(pa);
      pa += sa;
#pragma unroll
      for (int k = kk; k < T; ++k) acc[k].fma(x, w[k - kk]);
    }
  }
}

// x / k for a small integer k >= 1, x / 2, k x
#pragma nv_exec_check_disable
template <class S>
__host__ __device__ __forceinline__ S tree_div(S x, int k) {
  using A = Ar<S>;
  if constexpr (A::modular) return A::mul(x, inv_of<S>(k));
#ifdef __CUDA_ARCH__
  else if constexpr (A::fp64 && !A::dd) return A::scale(x, inv_int(k));
#endif
  else return A::div_int(x, k);
}
#pragma nv_exec_check_disable
template <class S>
__host__ __device__ __forceinline__ S tree_half(S x) {
  using A = Ar<S>;
  if constexpr (A::modular) return A::mul(x, A::half());
  else return A::scale_f(x, 0.5f);
}
#pragma nv_exec_check_disable
template <class S>
__host__ __device__ __forceinline__ S tree_times(S x, int k) {
  using A = Ar<S>;
  if constexpr (A::modular) return A::mul(x, A::of_int(k));
  else return A::scale_f(x, (float)k);
}

// sum_s a_s b_(t-s), s < la, by one thread
#pragma nv_exec_check_disable
template <class S>
__host__ __device__ __forceinline__ S conv_one(const S* a, long long sa, int la, const S* b, long long sb, int lb, int t) {
  using A = Ar<S>;
  ConvAcc<S> r = ConvAcc<S>::of(Ar<S>::zero());
  const int s0 = t - lb + 1 > 0 ? t - lb + 1 : 0;
  const int n = t < la - 1 ? t : la - 1;
#pragma unroll 4
  for (int s = s0; s <= n; ++s) r.fma(tld(a + s * sa), tld(b + (t - s) * sb));
  return r.sum();
}

// the terms s = sub, sub + SP, ... of coefficient t of a product
#pragma nv_exec_check_disable
template <int SP = WG_TREE_SPLIT, class S>
__host__ __device__ __forceinline__ void conv_part(ConvAcc<S>& acc, const S* a, long long sa, int la, const S* b, long long sb,
                                                   int t, int sub) {
  const int n = t < la - 1 ? t : la - 1;
#pragma unroll 4
  for (int s = sub; s <= n; s += SP) acc.fma(tld(a + s * sa), tld(b + (t - s) * sb));
}
// the same of two products at once: their loads overlap
#pragma nv_exec_check_disable
template <int SP = WG_TREE_SPLIT, class S>
__host__ __device__ __forceinline__ void conv_part2(ConvAcc<S>& acc, const S* a, const S* b, const S* c, const S* d, long long sa,
                                                    int la, long long sb, int t, int sub) {
  const int n = t < la - 1 ? t : la - 1;
#pragma unroll 2
  for (int s = sub; s <= n; s += SP) {
    const S x = tld(a + s * sa), y = tld(b + (t - s) * sb), z = tld(c + s * sa), w = tld(d + (t - s) * sb);
    acc.fma(x, y);
    acc.fma(z, w);
  }
}
// the sum over the SP threads of a coefficient, in each of them
#pragma nv_exec_check_disable
template <int SP = WG_TREE_SPLIT, class S>
__host__ __device__ __forceinline__ S split_sum(S v) {
#ifdef __CUDA_ARCH__
  using A = Ar<S>;
#pragma unroll
  for (int off = 1; off < SP; off *= 2) {
#pragma unroll
    for (int c = 0; c < A::NC; ++c) {
      const typename A::Comp x = A::comp(v, c);
      A::set_comp(v, c, A::cadd(x, A::shfl_xor(x, off)));
    }
  }
#endif
  return v;
}

__host__ __device__ __forceinline__ bool tree_need(const TreeInst& T, int a, int b) {
  return a != b || a == T.pB || a >= T.dpos;
}

// entry (a, b) of the root: the mean of the matrix's two triangles (equal to either when they
// agree); the unpaired vertex of an odd loop hafnian has a row only, and its loop weight apart
#pragma nv_exec_check_disable
template <class S>
__host__ __device__ __forceinline__ S tree_root_entry(const TreeInst& T, const typename TreeMatrix<S>::T* ext, int a,
                                                           int b) {
  using A = Ar<S>;
  using M = TreeMatrix<S>;
  const int ca = T.col[a], cb = T.col[b];
  if (ca < 0 || cb < 0) {
    const int o = ca < 0 ? a : b, x = ca < 0 ? b : a;
    return x == o ? A::zero() : (x == T.pL ? A::from_c64(T.oddloop) : M::load(ext + (size_t)T.row[o] * T.lda + T.col[x]));
  }
  const S x = M::load(ext + (size_t)T.row[a] * T.lda + cb), y = M::load(ext + (size_t)T.row[b] * T.lda + ca);
  return A::add(x, tree_half(A::sub(y, x)));
}

// ---- root: one node, one coefficient per entry
#pragma nv_exec_check_disable
template <class S>
__host__ __device__ void tree_root(const TreeInst& T, const unsigned char* __restrict__ pool, S* out, int tid, int nthr) {
  using M = typename TreeMatrix<S>::T;
  const M* __restrict__ ext = reinterpret_cast<const M*>(pool + T.a_off);
  const int ne = tree_entries(tree_width(T.X, T.E, 0), T.diag);
  for (int e = tid; e < ne; e += nthr) {
    int a = 0, b = 0;
    if (e) tree_decode(e, T.diag, a, b);
    tst(out + e, e ? tree_root_entry<S>(T, ext, a, b) : Ar<S>::one());
  }
}

// ---- the root and its simple edge in one: the +1 child, two coefficients an entry
#pragma nv_exec_check_disable
template <class S>
__host__ __device__ void tree_first(const TreeInst& T, const unsigned char* __restrict__ pool, S* chi, int tid,
                                    int nthr) {
  using A = Ar<S>;
  using M = typename TreeMatrix<S>::T;
  const M* __restrict__ ext = reinterpret_cast<const M*>(pool + T.a_off);
  const int i = T.X + 2 * (T.E - 1), j = i + 1, ne = tree_entries(i, T.diag);
  for (int e = tid; e < ne; e += nthr) {
    int a = 0, b = 0;
    S c = A::one(), u;
    if (e) {
      tree_decode(e, T.diag, a, b);
      if (!tree_need(T, a, b)) continue;
      c = tree_root_entry<S>(T, ext, a, b);
      u = A::fma(tree_root_entry<S>(T, ext, i, a), tree_root_entry<S>(T, ext, j, b),
                 A::mul(tree_root_entry<S>(T, ext, j, a), tree_root_entry<S>(T, ext, i, b)));
    } else {
      u = tree_root_entry<S>(T, ext, j, i);
      if (T.pL >= 0) u = A::fma(tree_root_entry<S>(T, ext, i, T.pL), tree_root_entry<S>(T, ext, j, T.pL), u);
    }
    tst(chi + 2 * e, c);
    tst(chi + 2 * e + 1, u);
  }
}

// ---- m = C_ij + v_i v_j of the edge of step q (loop kinds): scr[t np + p]
#pragma nv_exec_check_disable
template <class S, int TL>
__host__ __device__ void tree_m(const TreeInst& T, int q, const S* par, long long ps, int np, S* scr,
                       int tid, int nthr) {
  using A = Ar<S>;
  const int i = T.X + 2 * (T.E - 1 - q), j = i + 1;
  const int Lp = T.deg[q] + 1;
  if constexpr (TL == 0) {
    const int total = Lp * np, sub = tid % WG_TREE_SPLIT, step = nthr / WG_TREE_SPLIT;
    for (int x0 = 0; x0 < total; x0 += step) {
      const int x = x0 + tid / WG_TREE_SPLIT, p = x % np, t = Lp - 1 - x / np;
      const long long st = (long long)Lp * ps;
      ConvAcc<S> acc = ConvAcc<S>::of(A::zero());
      if (x < total)
        conv_part(acc, par + tree_ent(i, T.pL, T.diag) * st + p, ps, Lp, par + tree_ent(j, T.pL, T.diag) * st + p, ps,
                  t, sub);
      const S v = split_sum(acc.sum());
      if (x < total && sub == 0)
        tst(scr + (long long)t * np + p, A::add(tld(par + tree_ent(j, i, T.diag) * st + t * ps + p), v));
    }
    return;
  }
  constexpr int TT = TL ? TL : 1;
  const int nt = (Lp + TT - 1) / TT;
  for (int x = tid; x < nt * np; x += nthr) {
    const int p = x % np, t0 = Lp - TT * (x / np + 1);
    ConvAcc<S> acc[TT];
#pragma unroll
    for (int k = 0; k < TT; ++k)
      acc[k] = ConvAcc<S>::of(
          t0 + k >= 0 ? tld(par + ((long long)tree_ent(j, i, T.diag) * Lp + t0 + k) * ps + p) : A::zero());
    conv_tile<S, TT>(acc, par + (long long)tree_ent(i, T.pL, T.diag) * Lp * ps + p, ps, Lp,
                     par + (long long)tree_ent(j, T.pL, T.diag) * Lp * ps + p, ps, t0);
#pragma unroll
    for (int k = 0; k < TT; ++k)
      if (t0 + k >= 0) tst(scr + (long long)(t0 + k) * np + p, acc[k].sum());
  }
}

// ---- a simple edge: children delta = +1 (nodes 0 .. np-1) and -1 (np .. 2 np - 1) from the same
// products.  The weight -1 of the second joins g (loop kinds: tree_g).
#pragma nv_exec_check_disable
template <class S, int TL>
__host__ __device__ void tree_unit(const TreeInst& T, int q, const S* par, long long ps, int np,
                          S* chi, int tid, int nthr) {
  using A = Ar<S>;
  const int i = T.X + 2 * (T.E - 1 - q), j = i + 1, dg = T.diag;
  const int e0 = T.pL >= 0, ne = tree_entries(i, dg) - e0, Lp = T.deg[q] + 1, Lc = Lp + 1;
  const int nd = T.radix[q];  // 1: the root, which takes +1 only
  const long long cs = (long long)np * nd;
  if constexpr (TL <= 0) {  // TL < 0: two threads a coefficient
    constexpr int SP = TL < 0 ? (WG_TREE_SPLIT + 1) / 2 : WG_TREE_SPLIT;
    const unsigned total = (unsigned)Lp * ne * np, step = nthr / SP;
    const int sub = tid % SP;
    for (unsigned x0 = 0; x0 < total; x0 += step) {
      const unsigned x = x0 + tid / SP, r = x / np;
      const int p = x - r * np, e = e0 + r % ne, t = Lp - 1 - (int)(r / ne);
      int a = 0, b = 0;
      if (e) tree_decode(e, dg, a, b);
      const bool live = x < total && (e == 0 || tree_need(T, a, b));
      const S* pp = par + p;
      const long long st = (long long)Lp * ps;
      const S* base = pp + e * st;
      ConvAcc<S> acc = ConvAcc<S>::of(A::zero());
      S c = A::zero(), c0 = A::zero();
      if (live) {
        if (sub < 2 && t + 1 < Lp) c = tld(base + (t + 1) * ps);
        if (sub < 2 && t == 0) c0 = tld(base);
        if (e) {
          conv_part2<SP>(acc, pp + tree_ent(i, a, dg) * st, pp + tree_ent(j, b, dg) * st, pp + tree_ent(j, a, dg) * st,
                     pp + tree_ent(i, b, dg) * st, ps, Lp, ps, t, sub);
        } else {
          conv_part<SP>(acc, pp, ps, Lp, pp + tree_ent(j, i, dg) * st, ps, t, sub);
        }
      }
      using CA = ConvAcc<S>;
      const typename CA::U u = split_sum<SP>(acc.parts());
      if (live && sub < 2) {  // thread 0 stores the +1 child, thread 1 the -1 child, in the same instructions
        S* o = chi + (long long)e * Lc * cs + p;
        for (int h = sub; h < (SP > 1 ? sub + 1 : 2) && h < nd; ++h) {
          const S v = CA::plus(c, h ? Ar<typename CA::U>::neg(u) : u);
          const bool flip = h == 1 && e == 0;
          tst(o + h * np + (t + 1) * cs, flip ? A::neg(v) : v);
          if (t == 0) tst(o + h * np, flip ? A::neg(c0) : c0);
        }
      }
    }
    return;
  }
  constexpr int TT = TL > 0 ? TL : 1;
  const int nt = (Lp + TT - 1) / TT;
  const unsigned total = (unsigned)nt * ne * np;
  for (unsigned x = tid; x < total; x += nthr) {
    const unsigned r = x / np;
    const int p = x - r * np, e = e0 + r % ne, t0 = Lp - TT * ((int)(r / ne) + 1);
    const S* pp = par + p;
    ConvAcc<S> acc[TT];
#pragma unroll
    for (int k = 0; k < TT; ++k) acc[k] = ConvAcc<S>::of(A::zero());
    if (e == 0) {
      conv_tile<S, TT>(acc, pp, ps, Lp, pp + (long long)tree_ent(j, i, dg) * Lp * ps, ps, t0);
    } else {
      int a, b;
      tree_decode(e, dg, a, b);
      if (!tree_need(T, a, b)) continue;
      const long long st = (long long)Lp * ps;
      conv_tile<S, TT>(acc, pp + tree_ent(i, a, dg) * st, ps, Lp, pp + tree_ent(j, b, dg) * st, ps, t0);
      conv_tile<S, TT>(acc, pp + tree_ent(j, a, dg) * st, ps, Lp, pp + tree_ent(i, b, dg) * st, ps, t0);
    }
    const S* base = pp + (long long)e * Lp * ps;
    S* o = chi + (long long)e * Lc * cs + p;
#pragma unroll
    for (int k = -1; k < TT; ++k) {  // coefficient t + 1 of the children; k = -1: coefficient 0
      const int t = t0 + k;
      if (k < 0 ? t0 <= 0 : t >= 0) {
        const int tc = k < 0 ? 0 : t + 1;
        const S c = tc < Lp ? tld(base + tc * ps) : A::zero();
        S* w = o + tc * cs;
        if (k < 0) {
          tst(w, c);
          if (nd > 1) tst(w + np, e == 0 ? A::neg(c) : c);
        } else {
          const typename ConvAcc<S>::U u = acc[k < 0 ? 0 : k].parts();
          tst(w, ConvAcc<S>::plus(c, u));
          if (nd > 1) {
            const S v = ConvAcc<S>::plus(c, Ar<typename ConvAcc<S>::U>::neg(u));
            tst(w + np, e == 0 ? A::neg(v) : v);
          }
        }
      }
    }
  }
}

// ---- a loop kind's simple edge: the children's g = g (1 + delta eta m), of delta = -1 negative
#pragma nv_exec_check_disable
template <class S, int TL>
__host__ __device__ void tree_g(const TreeInst& T, int q, const S* par, long long ps, int np, const S* m, S* chi, int tid,
                                int nthr) {
  using A = Ar<S>;
  const int Lp = T.deg[q] + 1;
  const long long cs = 2ll * np;
  if constexpr (TL == 0) {
    const int total = Lp * np, sub = tid % WG_TREE_SPLIT, step = nthr / WG_TREE_SPLIT;
    for (int x0 = 0; x0 < total; x0 += step) {
      const int x = x0 + tid / WG_TREE_SPLIT, p = x % np, t = Lp - 1 - x / np;
      ConvAcc<S> acc = ConvAcc<S>::of(A::zero());
      if (x < total) conv_part(acc, par + p, ps, Lp, m + p, (long long)np, t, sub);
      const S u = split_sum(acc.sum());
      if (x < total && sub == 0) {
        const S c = t + 1 < Lp ? tld(par + p + (t + 1) * ps) : A::zero();
        S* o = chi + p + (t + 1) * cs;
        tst(o, A::add(c, u));
        tst(o + np, A::sub(u, c));
        if (t == 0) {
          tst(chi + p, tld(par + p));
          tst(chi + p + np, A::neg(tld(par + p)));
        }
      }
    }
    return;
  }
  constexpr int TT = TL ? TL : 1;
  const int nt = (Lp + TT - 1) / TT;
  for (int x = tid; x < nt * np; x += nthr) {
    const int p = x % np, t0 = Lp - TT * (x / np + 1);
    ConvAcc<S> acc[TT];
#pragma unroll
    for (int k = 0; k < TT; ++k) acc[k] = ConvAcc<S>::of(A::zero());
    conv_tile<S, TT>(acc, par + p, ps, Lp, m + p, (long long)np, t0);
#pragma unroll
    for (int k = 0; k < TT; ++k) {
      const int t = t0 + k;
      if (t < 0) continue;
      const S c = t + 1 < Lp ? tld(par + p + (t + 1) * ps) : A::zero(), u = acc[k].sum();
      tst(chi + p + (t + 1) * cs, A::add(c, u));
      tst(chi + p + np + (t + 1) * cs, A::sub(u, c));
    }
    if (t0 <= 0) {
      tst(chi + p, tld(par + p));
      tst(chi + p + np, A::neg(tld(par + p)));
    }
  }
}

// ---- a multiple edge of multiplicity r: child (digit d, parent p) = node d np + p, delta = r - 2 d
__host__ __device__ __forceinline__ double tree_weight(const TreeInst& T, int q, int d) {
  const int r = T.reps[q];
#ifdef __CUDA_ARCH__
  double w = c_binom[r][d];
#else
  double w = 1.0;
  for (int k = 0; k < d; ++k) w = w * (r - k) / (k + 1);
#endif
  if (d & 1) w = -w;
  if (T.radix[q] != r + 1 && 2 * d == r) w *= 0.5;  // the halved edge's delta = 0
  return w;
}

// A series in memory: elements `st` apart.
template <class S>
struct TreeSer {
  S* p;
  long long st;
  __host__ __device__ __forceinline__ S& operator[](int t) const { return p[t * st]; }
};
#pragma nv_exec_check_disable
template <class S>
__host__ __device__ __forceinline__ S conv_ser(TreeSer<S> a, int la, TreeSer<S> b, int lb, int t) {
  return conv_one((const S*)a.p, a.st, la, (const S*)b.p, b.st, lb, t);
}
// a copy of n elements of src (in global memory) into the warp's shared memory at dst
#pragma nv_exec_check_disable
template <class S>
__host__ __device__ __forceinline__ TreeSer<S> ser_stage(const S* src, long long st, int n, S* dst, int lane) {
  for (int t = lane; t < n; t += WG_TREE_LANES) dst[t] = tld(src + t * st);
  return {dst, 1};
}

// Series of the edge's 2 x 2 block, one warp per child: scr[(f Lc + t) nc + x], f = 0..2 the entries
// P_ii, P_ij, P_jj, f = 3 the factor h = Delta^(-1/2) (Delta = (1 - z c)^2 - z^2 a b, z = delta eta,
// a, b, c = C_ii, C_jj, C_ij), f = 4.. work; without loop weights also the child's g = w g h.  The
// recurrences are chains of short steps, so they run on copies in the warp's shared memory (smn
// elements at sm) when those fit: a step costs 30 clocks of latency there and 700 in L2.
#pragma nv_exec_check_disable
template <class S>
__host__ __device__ void tree_prep(const TreeInst& T, int q, const S* par, long long ps, int np, S* scr,
                          S* chi, S* sm, int smn, int tid, int nthr) {
  using A = Ar<S>;
  const int i = T.X + 2 * (T.E - 1 - q), j = i + 1, r = T.reps[q];
  const int Lp = T.deg[q] + 1, Lc = Lp + r, nc = np * T.radix[q];
  const int lane = tid & (WG_TREE_LANES - 1);
  const bool staged = smn >= 7 * Lc;
  for (int x = tid / WG_TREE_LANES; x < nc; x += nthr / WG_TREE_LANES) {
    const int p = x % np, d = x / np;
    const double z = (double)(r - 2 * d);
    const S* pp = par + p;
    const long long st = (long long)Lp * ps;
    auto work = [&](int f) -> TreeSer<S> { return {scr + (long long)f * Lc * nc + x, nc}; };
    const TreeSer<S> P0 = work(0), P1 = work(1), P2 = work(2), H = work(3);
    TreeSer<S> ca = {const_cast<S*>(pp + tree_ent(i, i, 1) * st), ps}, cb = {const_cast<S*>(pp + tree_ent(j, j, 1) * st), ps};
    TreeSer<S> cc = {const_cast<S*>(pp + tree_ent(j, i, 1) * st), ps}, g = {const_cast<S*>(pp), ps};
    TreeSer<S> h = H, dl = work(4), hh = work(5);
    if (staged) {
      ca = ser_stage<S>(ca.p, ps, Lp, sm, lane);
      cb = ser_stage<S>(cb.p, ps, Lp, sm + Lc, lane);
      cc = ser_stage<S>(cc.p, ps, Lp, sm + 2 * Lc, lane);
      g = ser_stage<S>(g.p, ps, Lp, sm + 3 * Lc, lane);
      h = {sm + 4 * Lc, 1};
      dl = {sm + 5 * Lc, 1};
      hh = {sm + 6 * Lc, 1};
      WG_TREE_SYNCWARP();
    }
    // Delta = 1 - 2 z c + z^2 (c c - a b)
    for (int t = lane; t < Lc; t += WG_TREE_LANES) {
      S v = t == 0 ? A::one() : A::zero();
      if (t >= 1 && t - 1 < Lp) v = A::sub(v, A::scale(cc[t - 1], 2.0 * z));
      if (t >= 2) {
        const S k = A::sub(conv_ser(cc, Lp, cc, Lp, t - 2), conv_ser(ca, Lp, cb, Lp, t - 2));
        v = A::add(v, A::scale(k, z * z));
      }
      dl[t] = v;
      h[t] = t == 0 ? A::one() : A::zero();
    }
    WG_TREE_SYNCWARP();
    // h = Delta^(-1/2), right-looking as in inv_sqrt_series
    for (int k = 0; k + 1 < Lc; ++k) {
      const S gk = h[k];
      for (int t = k + 1 + lane; t < Lc; t += WG_TREE_LANES) {
        S acc;
        if constexpr (A::modular) acc = A::fma(dl[t - k], A::mul(gk, A::mul(A::of_int(t + k), A::half())), h[t]);
        else acc = A::fma(dl[t - k], A::scale_f(gk, 0.5f * (float)(t + k)), h[t]);
        if (t == k + 1) acc = A::neg(tree_div(acc, t));
        h[t] = acc;
      }
      WG_TREE_SYNCWARP();
    }
    // 1 / Delta
    for (int t = lane; t < Lc; t += WG_TREE_LANES) hh[t] = conv_ser(h, Lc, h, Lc, t);
    WG_TREE_SYNCWARP();
    // P = z / Delta [[z b, 1 - z c], [1 - z c, z a]]
    for (int t = lane; t < Lc; t += WG_TREE_LANES) {
      S pi = A::zero(), pj = A::zero(), pc = A::zero();
      if (t >= 1) pc = A::scale(hh[t - 1], z);
      if (t >= 2) {
        pi = A::scale(conv_ser(hh, Lc, cb, Lp, t - 2), z * z);
        pj = A::scale(conv_ser(hh, Lc, ca, Lp, t - 2), z * z);
        pc = A::sub(pc, A::scale(conv_ser(hh, Lc, cc, Lp, t - 2), z * z));
      }
      tst(&P0[t], pi);
      tst(&P1[t], pc);
      tst(&P2[t], pj);
      if (staged && T.pL >= 0) tst(&H[t], h[t]);  // for tree_gloop
    }
    if (T.pL < 0) {
      const double w = tree_weight(T, q, d);
      for (int t = lane; t < Lc; t += WG_TREE_LANES)
        tst(chi + (long long)t * nc + x, A::scale(conv_ser(h, Lc, g, Lp, t), w));
    }
    WG_TREE_SYNCWARP();
  }
}

// Y = P C_e,b for every remaining row b: scr_y[((2 b + s) Lc + t) nc + x]
#pragma nv_exec_check_disable
template <class S, int TL>
__host__ __device__ void tree_y(const TreeInst& T, int q, const S* par, long long ps, int np,
                       const S* scr, S* y, int tid, int nthr) {
  using A = Ar<S>;
  const int i = T.X + 2 * (T.E - 1 - q), j = i + 1, W = i;
  const int Lp = T.deg[q] + 1, Lc = Lp + T.reps[q], nc = np * T.radix[q];
  const long long fs = (long long)Lc * nc;
  if constexpr (TL == 0) {
    const int total = Lc * 2 * W * nc, sub = tid % WG_TREE_SPLIT, step = nthr / WG_TREE_SPLIT;
    for (int x0 = 0; x0 < total; x0 += step) {
      const int x = x0 + tid / WG_TREE_SPLIT, r = x / nc, c = x - r * nc, bs = r % (2 * W), t = Lc - 1 - r / (2 * W);
      const int b = bs >> 1, s = bs & 1, p = c % np;
      ConvAcc<S> acc = ConvAcc<S>::of(A::zero());
      if (x < total) {
        conv_part2(acc, par + (long long)tree_ent(i, b, T.diag) * Lp * ps + p, scr + s * fs + c,
                   par + (long long)tree_ent(j, b, T.diag) * Lp * ps + p, scr + (s + 1) * fs + c, ps, Lp, (long long)nc,
                   t, sub);
      }
      const S v = split_sum(acc.sum());
      if (x < total && sub == 0) tst(y + (long long)bs * fs + (long long)t * nc + c, v);
    }
    return;
  }
  constexpr int TT = TL ? TL : 1;
  const int nt = (Lc + TT - 1) / TT;
  for (int x = tid; x < nt * 2 * W * nc; x += nthr) {
    const int r = x / nc, c = x - r * nc, bs = r % (2 * W), t0 = Lc - TT * (r / (2 * W) + 1);
    const int b = bs >> 1, s = bs & 1, p = c % np;
    ConvAcc<S> acc[TT];
#pragma unroll
    for (int k = 0; k < TT; ++k) acc[k] = ConvAcc<S>::of(A::zero());
    conv_tile<S, TT>(acc, par + (long long)tree_ent(i, b, T.diag) * Lp * ps + p, ps, Lp, scr + s * fs + c, nc, t0);
    conv_tile<S, TT>(acc, par + (long long)tree_ent(j, b, T.diag) * Lp * ps + p, ps, Lp, scr + (s + 1) * fs + c, nc,
                     t0);
#pragma unroll
    for (int k = 0; k < TT; ++k)
      if (t0 + k >= 0) tst(y + (long long)bs * fs + (long long)(t0 + k) * nc + c, acc[k].sum());
  }
}

// C' = C + C_ae Y(b)
#pragma nv_exec_check_disable
template <class S, int TL>
__host__ __device__ void tree_multi(const TreeInst& T, int q, const S* par, long long ps, int np,
                           const S* y, S* chi, int tid, int nthr) {
  using A = Ar<S>;
  const int i = T.X + 2 * (T.E - 1 - q), j = i + 1, dg = T.diag;
  const int ne = tree_entries(i, dg) - 1;
  const int Lp = T.deg[q] + 1, Lc = Lp + T.reps[q], nc = np * T.radix[q];
  const long long fs = (long long)Lc * nc, st = (long long)Lp * ps;
  if constexpr (TL == 0) {
    const unsigned total = (unsigned)Lc * ne * nc, step = nthr / WG_TREE_SPLIT;
    const int sub = tid % WG_TREE_SPLIT;
    for (unsigned x0 = 0; x0 < total; x0 += step) {
      const unsigned x = x0 + tid / WG_TREE_SPLIT, r = x / nc;
      const int c = x - r * nc, e = 1 + r % ne, t = Lc - 1 - (int)(r / ne), p = c % np;
      int a, b;
      tree_decode(e, dg, a, b);
      const bool live = x < total && tree_need(T, a, b);
      ConvAcc<S> acc = ConvAcc<S>::of(A::zero());
      if (live) {
        conv_part2(acc, par + p + tree_ent(i, a, dg) * st, y + (long long)(2 * b) * fs + c,
                   par + p + tree_ent(j, a, dg) * st, y + (long long)(2 * b + 1) * fs + c, ps, Lp, (long long)nc, t, sub);
      }
      S v = split_sum(acc.sum());
      if (live && sub == 0) {
        if (t < Lp) v = A::add(v, tld(par + p + e * st + t * ps));
        tst(chi + (long long)e * fs + (long long)t * nc + c, v);
      }
    }
    return;
  }
  constexpr int TT = TL ? TL : 1;
  const int nt = (Lc + TT - 1) / TT;
  const unsigned total = (unsigned)nt * ne * nc;
  for (unsigned x = tid; x < total; x += nthr) {
    const unsigned r = x / nc;
    const int c = x - r * nc, e = 1 + r % ne, t0 = Lc - TT * ((int)(r / ne) + 1), p = c % np;
    int a, b;
    tree_decode(e, dg, a, b);
    if (!tree_need(T, a, b)) continue;
    const S* base = par + p + (long long)e * st;
    ConvAcc<S> acc[TT];
#pragma unroll
    for (int k = 0; k < TT; ++k) {
      const int t = t0 + k;
      acc[k] = ConvAcc<S>::of(t >= 0 && t < Lp ? tld(base + t * ps) : A::zero());
    }
    conv_tile<S, TT>(acc, par + p + tree_ent(i, a, dg) * st, ps, Lp, y + (long long)(2 * b) * fs + c, nc, t0);
    conv_tile<S, TT>(acc, par + p + tree_ent(j, a, dg) * st, ps, Lp, y + (long long)(2 * b + 1) * fs + c, nc, t0);
#pragma unroll
    for (int k = 0; k < TT; ++k)
      if (t0 + k >= 0) tst(chi + (long long)e * fs + (long long)(t0 + k) * nc + c, acc[k].sum());
  }
}

// ---- a double edge.  To second order in z = delta eta (higher orders use the edge three times),
//   C' = C + z (c_i c_j^T + c_j c_i^T) + z^2 (c_i w_i^T + c_j w_j^T),  w_i = C_jj c_i + C_ij c_j,  w_j = C_ij c_i + C_ii c_j,
//   g' = g (1 + z M + z^2 (M^2 - w^2 + A B / 2)),  w = v_i v_j, M = C_ij + w, A = C_ii + v_i^2, B = C_jj + v_j^2,
// for z = 2, 0, -2 times eta: no recurrences, and the products serve all three children.
// w_i, w_j of every remaining row: y[((2 b + s) Lp + t) np + p]
#pragma nv_exec_check_disable
template <class S, int TL>
__host__ __device__ void tree_w2(const TreeInst& T, int q, const S* par, long long ps, int np, S* y, int tid, int nthr) {
  using A = Ar<S>;
  const int i = T.X + 2 * (T.E - 1 - q), j = i + 1, W = i, Lp = T.deg[q] + 1;
  const long long st = (long long)Lp * ps;
  constexpr int TT = TL ? TL : 1, SP = TL ? 1 : WG_TREE_SPLIT;
  const int nt = (Lp + TT - 1) / TT, total = nt * 2 * W * np, sub = tid % SP;
  for (int x0 = 0; x0 < total; x0 += nthr / SP) {
    const int x = x0 + tid / SP, r = x / np, p = x - r * np, bs = r % (2 * W), t0 = Lp - TT * (r / (2 * W) + 1);
    const int b = bs >> 1, s = bs & 1;
    const S* pp = par + p;
    const S *ci = pp + tree_ent(i, b, T.diag) * st, *cj = pp + tree_ent(j, b, T.diag) * st;
    const S *m0 = pp + (s ? tree_ent(j, i, 1) : tree_ent(j, j, 1)) * st;
    const S *m1 = pp + (s ? tree_ent(i, i, 1) : tree_ent(j, i, 1)) * st;
    ConvAcc<S> acc[TT];
#pragma unroll
    for (int k = 0; k < TT; ++k) acc[k] = ConvAcc<S>::of(A::zero());
    if constexpr (TL == 0) {
      if (x < total) conv_part2(acc[0], ci, m0, cj, m1, ps, Lp, ps, t0, sub);
      const S v = split_sum(acc[0].sum());
      if (x < total && sub == 0) tst(y + ((long long)bs * Lp + t0) * np + p, v);
    } else if (x < total) {
      conv_tile<S, TT>(acc, ci, ps, Lp, m0, ps, t0);
      conv_tile<S, TT>(acc, cj, ps, Lp, m1, ps, t0);
#pragma unroll
      for (int k = 0; k < TT; ++k)
        if (t0 + k >= 0) tst(y + ((long long)bs * Lp + t0 + k) * np + p, acc[k].sum());
    }
  }
}

// the children's entries: child coefficient t = U1_(t-1) z + U2_(t-2) z^2 + C_t, a tile over t - 1
#pragma nv_exec_check_disable
template <class S, int TL>
__host__ __device__ void tree_multi2(const TreeInst& T, int q, const S* par, long long ps, int np, const S* y, S* chi,
                                     int tid, int nthr) {
  using A = Ar<S>;
  using CA = ConvAcc<S>;
  const int i = T.X + 2 * (T.E - 1 - q), j = i + 1, dg = T.diag, nd = T.radix[q];
  const int ne = tree_entries(i, dg) - 1, Lp = T.deg[q] + 1, Lc = Lp + 2, Lt = Lp + 1;
  const long long st = (long long)Lp * ps, yt = (long long)Lp * np, cs = (long long)np * nd;
  constexpr int TT = TL ? TL : 1, SP = TL ? 1 : WG_TREE_SPLIT;
  const unsigned nt = (Lt + TT - 1) / TT, total = nt * ne * np;
  const int sub = tid % SP;
  for (unsigned x0 = 0; x0 < total; x0 += nthr / SP) {
    const unsigned x = x0 + tid / SP, r = x / np;
    const int p = x - r * np, e = 1 + r % ne, t0 = Lt - TT * ((int)(r / ne) + 1);
    int a, b;
    tree_decode(e, dg, a, b);
    const bool live = x < total && tree_need(T, a, b);
    const S* pp = par + p;
    const S *ia = pp + tree_ent(i, a, dg) * st, *ja = pp + tree_ent(j, a, dg) * st;
    const S *wi = y + 2 * b * yt + p, *wj = wi + yt;
    CA u1[TT], u2[TT];
#pragma unroll
    for (int k = 0; k < TT; ++k) u1[k] = u2[k] = CA::of(A::zero());
    if (live) {
      const S *ib = pp + tree_ent(i, b, dg) * st, *jb = pp + tree_ent(j, b, dg) * st;
      if constexpr (TL == 0) {
        if (t0 < Lp) conv_part2(u1[0], ia, jb, ja, ib, ps, Lp, ps, t0, sub);
        if (t0 > 0) conv_part2(u2[0], ia, wi, ja, wj, ps, Lp, (long long)np, t0 - 1, sub);
      } else {
        conv_tile<S, TT>(u1, ia, ps, Lp, jb, ps, t0, Lp);
        conv_tile<S, TT>(u1, ja, ps, Lp, ib, ps, t0, Lp);
        conv_tile<S, TT>(u2, ia, ps, Lp, wi, np, t0 - 1, Lp);
        conv_tile<S, TT>(u2, ja, ps, Lp, wj, np, t0 - 1, Lp);
      }
    }
    const S* base = pp + e * st;
    S* o = chi + (long long)e * Lc * cs + p;
#pragma unroll
    for (int k = -1; k < TT; ++k) {  // child coefficient t0 + k + 1; k = -1: coefficient 0
      const int t = t0 + k + 1;
      if (k < 0) {
        if (live && t0 <= 0 && sub == 0)
          for (int d = 0; d < nd; ++d) tst(o + d * np, tld(base));
        continue;
      }
      S v1 = u1[k < 0 ? 0 : k].sum(), v2 = u2[k < 0 ? 0 : k].sum();
      if constexpr (TL == 0) {
        v1 = split_sum(v1);
        v2 = split_sum(v2);
      }
      if (!live || t < 1 || sub != 0) continue;
      const S c = t < Lp ? tld(base + t * ps) : A::zero();
      const S even = A::add(c, tree_times(v2, 4)), odd = tree_times(v1, 2);
      S* w = o + t * cs;
      tst(w, A::add(even, odd));
      if (nd > 1) tst(w + np, c);
      if (nd > 2) tst(w + 2 * np, A::sub(even, odd));
    }
  }
}

// the children's g, one warp per parent; series in the warp's shared memory, or in `wk` (8 Lp np)
#pragma nv_exec_check_disable
template <class S>
__host__ __device__ void tree_g2(const TreeInst& T, int q, const S* par, long long ps, int np, S* wk, S* chi, S* sm,
                                 int smn, int tid, int nthr) {
  using A = Ar<S>;
  const int i = T.X + 2 * (T.E - 1 - q), j = i + 1, nd = T.radix[q], Lp = T.deg[q] + 1;
  const long long st = (long long)Lp * ps, cs = (long long)np * nd;
  const int lane = tid & (WG_TREE_LANES - 1);
  const bool loops = T.pL >= 0;
  for (int p = tid / WG_TREE_LANES; p < np; p += nthr / WG_TREE_LANES) {
    S* w0 = smn >= 8 * Lp ? sm : wk + 8ll * Lp * p;
    auto ser = [&](int f, int t) -> S& { return w0[f * Lp + t]; };  // g, M, A, B, w, v_i, v_j, second order
    const S* pp = par + p;
    for (int t = lane; t < Lp; t += WG_TREE_LANES) {
      ser(0, t) = tld(pp + t * ps);
      ser(1, t) = tld(pp + tree_ent(j, i, 1) * st + t * ps);
      ser(2, t) = tld(pp + tree_ent(i, i, 1) * st + t * ps);
      ser(3, t) = tld(pp + tree_ent(j, j, 1) * st + t * ps);
      if (loops) {
        ser(5, t) = tld(pp + tree_ent(i, T.pL, 1) * st + t * ps);
        ser(6, t) = tld(pp + tree_ent(j, T.pL, 1) * st + t * ps);
      }
    }
    WG_TREE_SYNCWARP();
    if (loops) {  // w, v_i^2, v_j^2 side by side over the lanes
      for (int x = lane; x < 3 * Lp; x += WG_TREE_LANES) {
        const int f = x / Lp, t = x - f * Lp;
        const S *u = w0 + (f == 2 ? 6 : 5) * Lp, *v = w0 + (f == 1 ? 5 : 6) * Lp;
        const S r = conv_one(u, 1, Lp, v, 1, Lp, t);
        if (f == 0) {
          ser(4, t) = r;
          ser(1, t) = A::add(ser(1, t), r);
        } else {
          ser(f + 1, t) = A::add(ser(f + 1, t), r);
        }
      }
      WG_TREE_SYNCWARP();
    }
    for (int t = lane; t < Lp; t += WG_TREE_LANES) {
      ConvAcc<S> x = ConvAcc<S>::of(A::zero()), y = x, z = x;
      for (int s = 0; s <= t; ++s) {
        x.fma(ser(1, s), ser(1, t - s));
        y.fma(ser(2, s), ser(3, t - s));
        if (loops) z.fma(ser(4, s), ser(4, t - s));
      }
      S r = A::add(x.sum(), tree_half(y.sum()));
      if (loops) r = A::sub(r, z.sum());
      ser(7, t) = r;
    }
    WG_TREE_SYNCWARP();
    for (int x = lane; x < 2 * Lp; x += WG_TREE_LANES) {  // g M and g times the second order
      const int f = x / Lp, t = x - f * Lp;
      ser(5 + f, t) = conv_one((const S*)w0, 1, Lp, (const S*)(w0 + (f ? 7 : 1) * Lp), 1, Lp, t);
    }
    WG_TREE_SYNCWARP();
    for (int x = lane; x < nd * (Lp + 2); x += WG_TREE_LANES) {
      const int d = x / (Lp + 2), t = x - d * (Lp + 2);
      S r = t < Lp ? ser(0, t) : A::zero();
      if (d != 1) {
        if (t >= 1 && t - 1 < Lp) r = A::add(r, tree_times(ser(5, t - 1), 2 - 2 * d));
        if (t >= 2) r = A::add(r, tree_times(ser(6, t - 2), 4));
      }
      tst(chi + t * cs + d * np + p, A::scale(r, tree_weight(T, q, d)));
    }
    WG_TREE_SYNCWARP();
  }
}

// loop kinds: g' = w g h exp(v_e Y(L) / 2), one warp per child; shared memory as in tree_prep
#pragma nv_exec_check_disable
template <class S>
__host__ __device__ void tree_gloop(const TreeInst& T, int q, const S* par, long long ps, int np, S* scr,
                           const S* y, S* chi, S* sm, int smn, int tid, int nthr) {
  using A = Ar<S>;
  const int i = T.X + 2 * (T.E - 1 - q), j = i + 1;
  const int Lp = T.deg[q] + 1, Lc = Lp + T.reps[q], nc = np * T.radix[q];
  const long long fs = (long long)Lc * nc, st = (long long)Lp * ps;
  const int lane = tid & (WG_TREE_LANES - 1);
  const bool staged = smn >= 9 * Lc;
  for (int x = tid / WG_TREE_LANES; x < nc; x += nthr / WG_TREE_LANES) {
    const int p = x % np, d = x / np;
    TreeSer<S> vi = {const_cast<S*>(par + p + tree_ent(i, T.pL, T.diag) * st), ps};
    TreeSer<S> vj = {const_cast<S*>(par + p + tree_ent(j, T.pL, T.diag) * st), ps};
    TreeSer<S> g = {const_cast<S*>(par + p), ps}, h = {scr + 3 * fs + x, nc};
    TreeSer<S> yi = {const_cast<S*>(y + (long long)(2 * T.pL) * fs + x), nc}, yj = {yi.p + fs, nc};
    TreeSer<S> u = {scr + 4 * fs + x, nc}, ex = {scr + 5 * fs + x, nc}, gh = {scr + x, nc};  // P is not needed any more
    if (staged) {
      vi = ser_stage<S>(vi.p, ps, Lp, sm, lane);
      vj = ser_stage<S>(vj.p, ps, Lp, sm + Lc, lane);
      g = ser_stage<S>(g.p, ps, Lp, sm + 2 * Lc, lane);
      yi = ser_stage<S>(yi.p, nc, Lc, sm + 3 * Lc, lane);
      yj = ser_stage<S>(yj.p, nc, Lc, sm + 4 * Lc, lane);
      h = ser_stage<S>(h.p, nc, Lc, sm + 5 * Lc, lane);
      u = {sm + 6 * Lc, 1};
      ex = {sm + 7 * Lc, 1};
      gh = {sm + 8 * Lc, 1};
      WG_TREE_SYNCWARP();
    }
    for (int t = lane; t < Lc; t += WG_TREE_LANES) {
      u[t] = tree_half(A::add(conv_ser(vi, Lp, yi, Lc, t), conv_ser(vj, Lp, yj, Lc, t)));
      ex[t] = t == 0 ? A::one() : A::zero();
      gh[t] = conv_ser(h, Lc, g, Lp, t);
    }
    WG_TREE_SYNCWARP();
    for (int k = 0; k + 1 < Lc; ++k) {  // exp, right-looking as in exp_series
      const S ek = ex[k];
      for (int t = k + 1 + lane; t < Lc; t += WG_TREE_LANES) {
        S acc;
        if constexpr (A::modular) acc = A::fma(A::mul(u[t - k], A::of_int(t - k)), ek, ex[t]);
        else acc = A::fma(A::scale_f(u[t - k], (float)(t - k)), ek, ex[t]);
        if (t == k + 1) acc = tree_div(acc, t);
        ex[t] = acc;
      }
      WG_TREE_SYNCWARP();
    }
    const double w = tree_weight(T, q, d);
    for (int t = lane; t < Lc; t += WG_TREE_LANES)
      tst(chi + (long long)t * nc + x, A::scale(conv_ser(ex, Lc, gh, Lc, t), w));
    WG_TREE_SYNCWARP();
  }
}

// ---- leaves without a batch mode: this thread's share of the output over nodes [0, np) of a buffer of stride ps
#pragma nv_exec_check_disable
template <class S, int TL>
__host__ __device__ S tree_leaf_sum(const TreeInst& T, const S* par, long long ps, int np, const S* m, int tid, int nthr) {
  using A = Ar<S>;
  const int L = T.deg[T.steps] + 1, D = L - 1, dg = T.diag;
  const long long st = (long long)L * ps;
  S sum = A::zero();
  if (T.steps < T.E) {
    // simple edges left: the coefficient of their deltas at once, [eta^D] g h, one thread per node
    // and tile of h.  Two edges on X .. X+3 (no loop weights): h = haf(4 x 4).  One edge on X, X+1:
    // h = C_ij + v_i v_j; with an unpaired vertex o, h = v_o (C_ij + v_i v_j) + C_io v_j + C_jo v_i
    // (m = C_ij + v_i v_j from tree_m).
    constexpr int TT = TL ? TL : 1;
    const int nt = TL ? (L + TT - 1) / TT : L * WG_TREE_SPLIT, X = T.X;
    const bool two = T.E - T.steps == 2;
    for (int x = tid; x < nt * np; x += nthr) {
      // four threads a coefficient: neighbours share the node and coefficient, and split its products
      const int sub = TL ? 0 : x % WG_TREE_SPLIT, xx = TL ? x : x / WG_TREE_SPLIT;
      const int p = xx % np, t0 = L - TT * (xx / np + 1);
      const S* pp = par + p;
      ConvAcc<S> acc[TT];
#pragma unroll
      for (int k = 0; k < TT; ++k) acc[k] = ConvAcc<S>::of(A::zero());
      if (!two && T.pO < 0 && sub == 0) {
#pragma unroll
        for (int k = 0; k < TT; ++k)
          if (t0 + k >= 0) acc[k] = ConvAcc<S>::of(tld(pp + tree_ent(X + 1, X, dg) * st + (t0 + k) * ps));
      }
      const int nw = two ? 3 : (T.pO >= 0 ? 3 : (T.pL >= 0 ? 1 : 0));
#pragma unroll 1
      for (int w = 0; w < nw; ++w) {
        const S *u, *v;
        long long su = ps;
        if (two) {  // pairings (01)(23), (02)(13), (12)(03)
          u = pp + st * (w == 0 ? tree_ent(X + 1, X, dg) : tree_ent(X + 2, w == 1 ? X : X + 1, dg));
          v = pp + st * (w == 0 ? tree_ent(X + 3, X + 2, dg) : tree_ent(X + 3, w == 1 ? X + 1 : X, dg));
        } else if (T.pO < 0) {
          u = pp + st * tree_ent(X, T.pL, dg);
          v = pp + st * tree_ent(X + 1, T.pL, dg);
        } else if (w == 2) {
          u = m + p;
          su = np;
          v = pp + st * tree_ent2(T.pO, T.pL, dg);
        } else {
          u = pp + st * tree_ent(X + w, T.pO, dg);
          v = pp + st * tree_ent(X + 1 - w, T.pL, dg);
        }
        if constexpr (TL == 0) conv_part(acc[0], u, su, L, v, ps, t0, sub);
        else conv_tile<S, TT>(acc, u, su, L, v, ps, t0);
      }
#pragma unroll
      for (int k = 0; k < TT; ++k)
        if (t0 + k >= 0) sum = A::fma(tld(pp + (D - t0 - k) * ps), acc[k].sum(), sum);
    }
  } else {
    for (int p = tid; p < np; p += nthr) {
      if (T.pO < 0) {
        sum = A::add(sum, tld(par + D * ps + p));
      } else {
        const S* vo = par + p + (long long)tree_ent2(T.pO, T.pL, dg) * st;
        for (int s = 0; s <= D; ++s) sum = A::fma(tld(par + p + (D - s) * ps), tld(vo + s * ps), sum);
      }
    }
  }
  return sum;
}

// ---- leaves with a batch mode: the sums of the warp's nodes, left in sm
#pragma nv_exec_check_disable
template <class S>
__host__ __device__ void tree_leaf_batch(const TreeInst& T, const S* par, long long ps, int np, S* sm, int smn, int tid,
                                         int nthr) {
  using A = Ar<S>;
  const int L = T.deg[T.steps] + 1, D = L - 1, dg = T.diag;
  const long long st = (long long)L * ps;
  // batch mode b with loop series v and pair series c: k photons give H_k = v H_(k-1) +
  // (k-1) c H_(k-2); with an unpaired vertex o: v_o H_k + k c_ob H_(k-1).  One warp per node, the
  // series and the output sums in its shared memory.  An FP64 instruction takes its 64 clocks
  // however few lanes it has, so the lanes split: four to a coefficient, then four to an output
  // (12 modes, cutoff 6: 53,000 clocks with a lane per coefficient and a warp sum per output).
  const int lane = tid & (WG_TREE_LANES - 1), nw = nthr / WG_TREE_LANES;
  const int sub = lane % WG_TREE_SPLIT, grp = lane / WG_TREE_SPLIT;
  constexpr int NG = WG_TREE_LANES / WG_TREE_SPLIT;
  const bool staged = smn >= 32 + (T.nout + 4) * L;  // every H_k kept, and copies of v and c
  const int rows = staged ? T.nout : 3;
  S *const o = sm, *const h = sm + 32, *gv = h + rows * L, *gc = gv + L;
  for (int k = lane; k < T.nout; k += WG_TREE_LANES) o[k] = A::zero();
  WG_TREE_SYNCWARP();
  for (int p = tid / WG_TREE_LANES; p < np; p += nw) {
    const S* pp = par + p;
    TreeSer<S> v = {const_cast<S*>(pp + (long long)tree_ent2(T.pB, T.pL, dg) * st), ps};
    TreeSer<S> c = {const_cast<S*>(pp + (long long)tree_ent(T.pB, T.pB, 1) * st), ps};
    if (staged) {
      v = ser_stage<S>(v.p, ps, L, gc + L, lane);
      c = ser_stage<S>(c.p, ps, L, gc + 2 * L, lane);
    }
    for (int t = lane; t < L; t += WG_TREE_LANES) {
      h[t] = t == 0 ? A::one() : A::zero();
      if (T.pO >= 0) {
        gv[t] = conv_one(pp, ps, L, pp + (long long)tree_ent2(T.pO, T.pL, dg) * st, ps, L, t);
        gc[t] = conv_one(pp, ps, L, pp + (long long)tree_ent2(T.pO, T.pB, dg) * st, ps, L, t);
      } else {
        gv[t] = tld(pp + t * ps);
      }
    }
    WG_TREE_SYNCWARP();
    // the dots of outputs k0 .. k1 - 1
    auto dots = [&](int k0, int k1) {
      for (int kb = k0; kb < k1; kb += NG) {
        const int k = kb + grp;
        ConvAcc<S> x = ConvAcc<S>::of(A::zero()), y = x;
        if (k < k1) {
          const S *hk = h + (k % rows) * L, *hl = h + ((k + rows - 1) % rows) * L;
          for (int t = sub; t < L; t += WG_TREE_SPLIT) {
            x.fma(gv[D - t], hk[t]);
            if (k && T.pO >= 0) y.fma(gc[D - t], hl[t]);
          }
        }
        S r = x.sum();
        if (T.pO >= 0) r = A::add(r, tree_times(y.sum(), k));
        r = split_sum(r);
        if (k < k1 && sub == 0) o[k] = A::add(o[k], r);
      }
      WG_TREE_SYNCWARP();
    };
    for (int k = 1; k < T.nout; ++k) {
      S* hn = h + (k % rows) * L;
      const S *h1 = h + ((k - 1) % rows) * L, *h2 = h + ((k + rows - 2) % rows) * L;
      if (!staged) dots(k - 1, k);
      for (int tb = 0; tb < L; tb += NG) {
        const int t = tb + grp;
        ConvAcc<S> x = ConvAcc<S>::of(A::zero()), y = x;
        if (t < L) {
          conv_part(x, (const S*)v.p, v.st, L, h1, 1ll, t, sub);
          if (k > 1) conv_part(y, (const S*)c.p, c.st, L, h2, 1ll, t, sub);
        }
        S n = x.sum();
        if (k > 1) n = A::add(n, tree_times(y.sum(), k - 1));
        n = split_sum(n);
        if (t < L && sub == 0) hn[t] = n;
      }
      WG_TREE_SYNCWARP();
    }
    dots(staged ? 0 : T.nout - 1, T.nout);
  }
}

// either
#pragma nv_exec_check_disable
template <class S, int TL>
__host__ __device__ S tree_leaf(const TreeInst& T, const S* par, long long ps, int np, const S* m, S* sm, int smn,
                                int tid, int nthr) {
  if (T.pB < 0) return tree_leaf_sum<S, TL>(T, par, ps, np, m, tid, nthr);
  tree_leaf_batch<S>(T, par, ps, np, sm, smn, tid, nthr);
  return Ar<S>::zero();
}

template <class S>
__device__ __forceinline__ void tree_store(const TreeInst& T, S sum, long long slot, double2* partials) {
  using A = Ar<S>;
  const int lane = threadIdx.x & 31;
  if (lane < T.nout) {
    const c64 z = A::to_c64(sum);
    partials[slot + lane] = make_double2(z.re, z.im);
    if constexpr (A::dd) {
      const c64 zl = A::lo_c64(sum);
      partials[slot + T.comp_off + lane] = make_double2(zl.re, zl.im);
    }
  }
}

// Barrier of the `ctas` CTAs of a cooperative launch that share trees (one CTA: a block barrier).  The
// wait is bounded: after TREE_POLLS polls, about 3 s, a CTA gives up, its later barriers do not wait, and
// the error flag makes the outputs gave_up(), which the host reports and clears (read_outputs, sieve.cu).
constexpr unsigned int TREE_POLLS = 1u << 22;
struct TreeSync {
  unsigned int* bar;
  int* err;
  unsigned int ctas, polls;
  unsigned int target = 0;
  bool ok = true;  // thread 0's
  __device__ __forceinline__ void operator()() {
    __syncthreads();
    if (ctas == 1) return;
    target += ctas;
    if (threadIdx.x == 0) {
      __threadfence();
      atomicAdd(bar, 1u);
      if (ok) {
        unsigned int v, n = 0;
        do {
          asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
        } while (v < target && ++n < polls);
        ok = v >= target;
        if (!ok) atomicExch(err, 1);
      }
    }
    __syncthreads();  // orders every thread's reads after thread 0's acquire (a fence there too: n = 24 87 us, 84 without)
  }
};

// The plan's only launch also reduces: the CTA that finishes last sums the partials of every
// output, as reduce_kernel does, and re-arms the counters.
__device__ __forceinline__ void tree_finish(const TreeFinish& F, unsigned int ctas) {
  if (!F.done) return;
  __shared__ int s_last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    s_last = ctas == 1 || atomicAdd(F.done, 1u) == ctas - 1;
    __threadfence();
  }
  __syncthreads();
  if (!s_last) return;
  const int nw = blockDim.x >> 5;
  reduce_block(F.inst, F.ninst, F.partials, F.scales, F.out, F.first_out, nw / F.wpo, F.end_out, F.wpo, F.mags, F.err);
  for (int i = threadIdx.x; i < F.ncounters; i += blockDim.x) F.counters[i] = 0u;
}

// ---- trees by the whole chip in one cooperative launch: every round over all warps, one barrier of
// the launch after it.  Consecutive warps of a round lie on different SMs, so that a narrow level
// still uses every FP64 pipe.  Levels live in the workspace (L2 resident; a single CTA's in shared
// memory).
// `cta` of the `ctas` CTAs that share P's trees.
template <class S>
__device__ __forceinline__ void tree_body(const TreeParams& P, const int cta, const int ctas) {
  extern __shared__ __align__(16) unsigned char smem[];
  using A = Ar<S>;
  constexpr int TL = tree_tile<S>();
  S* sm = reinterpret_cast<S*>(smem);
  S* smw = sm + (threadIdx.x >> 5) * P.sm_warp;
  using V = typename Leaf<S>::V;
  __shared__ LeafSums<S> sums;
  bool some = false;  // this warp has leaves in `sums`
  const TreeInst* insts = P.inst;
  const TreeRound* rounds = P.rounds;
  const TreeSeg* segs = P.segs;
  if (P.cached) {  // the host laid the three arrays out one after another
    const int words = (int)((P.ninst * sizeof(TreeInst) + P.nrounds * sizeof(TreeRound) + P.nsegs * sizeof(TreeSeg)) / 16);
    const int4* src = reinterpret_cast<const int4*>(P.inst);
    int4* dst = reinterpret_cast<int4*>(smem + P.sm_cache);
    for (int w = threadIdx.x; w < words; w += blockDim.x) dst[w] = src[w];
    insts = reinterpret_cast<const TreeInst*>(dst);
    rounds = reinterpret_cast<const TreeRound*>(insts + P.ninst);
    segs = reinterpret_cast<const TreeSeg*>(rounds + P.nrounds);
    __syncthreads();
  }
  unsigned char* ws = P.sm_ws ? smem + P.sm_ws : P.ws;
  const int lane = threadIdx.x & 31;
  const int gn = ctas * (blockDim.x >> 5);
  __shared__ int s_next[2];
  if (threadIdx.x == 0) s_next[0] = 0;
  __syncthreads();
  TreeSync sync{P.bar, P.err, (unsigned int)ctas, P.polls};
  for (int r = 0; r < P.nrounds; ++r) {
    const TreeRound R = rounds[r];
    // A round's warps go to the CTAs in turn.  Where that is more than one a warp, the CTA's warps take
    // its next one as they come free (from a counter in shared memory; one in global memory for all CTAs
    // measured 4 % slower at n = 40 than fixed turns).  Fixed turns otherwise, so that a single
    // instance's leaf sums, at most one a warp, add up in the same order every time.
    if (threadIdx.x == 0) s_next[(r + 1) & 1] = 0;
    const bool taken = R.nwarps > gn;
    for (int turn = threadIdx.x >> 5;; turn += blockDim.x >> 5) {
      if (taken) {
        if (lane == 0) turn = atomicAdd(&s_next[r & 1], 1);
        turn = __shfl_sync(0xffffffffu, turn, 0);
      }
      const int vw = turn * ctas + cta;
      if (vw >= R.nwarps) break;
      int lo = R.seg0, hi = R.seg0 + R.nseg - 1;
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (segs[mid].warp0 <= vw) lo = mid; else hi = mid - 1;
      }
      const TreeSeg G = segs[lo];
      const int end = lo + 1 < R.seg0 + R.nseg ? segs[lo + 1].warp0 : R.nwarps;
      const TreeInst& T = insts[G.inst];
      const int tid = (vw - G.warp0) * 32 + lane, nthr = (end - G.warp0) * 32;
      const S* par = reinterpret_cast<const S*>(ws + G.par) + G.p0;
      S* chi = reinterpret_cast<S*>(ws + G.chi);
      S* scr = reinterpret_cast<S*>(ws + T.scr_off);
      S* ms = tree_m_of(T, scr, G.q);
      switch (G.phase) {
        case TP_ROOT: tree_root<S>(T, P.pool, chi, tid, nthr); break;
        case TP_FIRST: tree_first<S>(T, P.pool, chi, tid, nthr); break;
        case TP_M:
          if (G.tile == 0) tree_m<S, 0>(T, G.q, par, G.pstride, G.np, ms, tid, nthr);
          else if (G.tile == 1) tree_m<S, 1>(T, G.q, par, G.pstride, G.np, ms, tid, nthr);
          else tree_m<S, TL>(T, G.q, par, G.pstride, G.np, ms, tid, nthr);
          break;
        case TP_UNIT:
          if (G.tile == 0) tree_unit<S, 0>(T, G.q, par, G.pstride, G.np, chi, tid, nthr);
          else if (G.tile == TREE_PAIRS) tree_unit<S, -1>(T, G.q, par, G.pstride, G.np, chi, tid, nthr);
          else if (G.tile == 1) tree_unit<S, 1>(T, G.q, par, G.pstride, G.np, chi, tid, nthr);
          else tree_unit<S, TL>(T, G.q, par, G.pstride, G.np, chi, tid, nthr);
          break;
        case TP_G:
          if (G.tile == 0) tree_g<S, 0>(T, G.q, par, G.pstride, G.np, ms, chi, tid, nthr);
          else if (G.tile == 1) tree_g<S, 1>(T, G.q, par, G.pstride, G.np, ms, chi, tid, nthr);
          else tree_g<S, TL>(T, G.q, par, G.pstride, G.np, ms, chi, tid, nthr);
          break;
        case TP_PREP: tree_prep<S>(T, G.q, par, G.pstride, G.np, scr, chi, smw, P.sm_warp, tid, nthr); break;
        case TP_LEAF: {
          V share;
          if (T.pB >= 0) {  // output k's to lane k
            tree_leaf_batch<S>(T, par, G.pstride, G.np, smw, P.sm_warp, tid, nthr);
            __syncwarp();
            share = Leaf<S>::of(lane < T.nout ? smw[lane] : A::zero());
            __syncwarp();
          } else {
            const S sum = G.tile == 0   ? tree_leaf_sum<S, 0>(T, par, G.pstride, G.np, ms, tid, nthr)
                          : G.tile == 1 ? tree_leaf_sum<S, 1>(T, par, G.pstride, G.np, ms, tid, nthr)
                                        : tree_leaf_sum<S, TL>(T, par, G.pstride, G.np, ms, tid, nthr);
            share = warp_sum(Leaf<S>::of(sum));
          }
          if (P.ninst > 1) {
            tree_store<V>(T, share, G.part + (long long)(vw - G.warp0) * T.pstride, P.partials);
          } else if (lane < T.nout) {  // all leaves are one instance's: one partial per CTA, below
            if (some) sums.add(threadIdx.x >> 5, lane, share);
            else sums.begin(threadIdx.x >> 5, lane, share);
          }
          some = true;
          break;
        }
        case TP_G2: {
          S* wk = scr + (2ll * tree_width(T.X, T.E, G.q + 1)) * (T.deg[G.q] + 1) * G.np;
          tree_g2<S>(T, G.q, par, G.pstride, G.np, wk, chi, smw, P.sm_warp, tid, nthr);
          break;
        }
        case TP_W2:
          if (G.tile == 0) tree_w2<S, 0>(T, G.q, par, G.pstride, G.np, scr, tid, nthr);
          else tree_w2<S, TL>(T, G.q, par, G.pstride, G.np, scr, tid, nthr);
          break;
        case TP_MULTI2:
          if (G.tile == 0) tree_multi2<S, 0>(T, G.q, par, G.pstride, G.np, scr, chi, tid, nthr);
          else tree_multi2<S, TL>(T, G.q, par, G.pstride, G.np, scr, chi, tid, nthr);
          break;
        default: {
          S* y = scr + 6ll * (T.deg[G.q + 1] + 1) * G.np * T.radix[G.q];
          if (G.phase == TP_GLOOP) {
            tree_gloop<S>(T, G.q, par, G.pstride, G.np, scr, y, chi, smw, P.sm_warp, tid, nthr);
          } else if (G.phase == TP_Y) {
            if (G.tile == 0) tree_y<S, 0>(T, G.q, par, G.pstride, G.np, scr, y, tid, nthr);
            else if (G.tile == 1) tree_y<S, 1>(T, G.q, par, G.pstride, G.np, scr, y, tid, nthr);
            else tree_y<S, TL>(T, G.q, par, G.pstride, G.np, scr, y, tid, nthr);
          } else {
            if (G.tile == 0) tree_multi<S, 0>(T, G.q, par, G.pstride, G.np, y, chi, tid, nthr);
            else if (G.tile == 1) tree_multi<S, 1>(T, G.q, par, G.pstride, G.np, y, chi, tid, nthr);
            else tree_multi<S, TL>(T, G.q, par, G.pstride, G.np, y, chi, tid, nthr);
          }
        }
      }
    }
    if (r + 1 < P.nrounds) sync();
  }
  if (P.ninst == 1) {
    const TreeInst& T = insts[0];
    if (!some && lane < T.nout) sums.begin(threadIdx.x >> 5, lane, Ar<V>::zero());
    __syncthreads();
    if (threadIdx.x < 32) {
      const int nw = blockDim.x >> 5;
      V v = Ar<V>::zero();
      if (T.nout == 1) v = warp_sum(lane < nw ? sums.value(lane, 0) : v);
      else if (lane < T.nout)
        for (int w = 0; w < nw; ++w) v = Ar<V>::add(v, sums.value(w, lane));
      tree_store<V>(T, v, segs[P.nsegs - 1].part + (long long)cta * T.pstride, P.partials);
    }
  }
  tree_finish(P.fin, ctas);
}

template <class S>
static __global__ void __launch_bounds__(TREE_THREADS, 1) tree_kernel(const TreeParams P) {
  tree_body<S>(P, blockIdx.x, gridDim.x);
}

}  // namespace wg
