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
// no pivots.  Multiple edges take the whole 2 x 2 block, P = (X_e^-1 - C_ee)^-1:
//   C' = C + C_re P C_er,   g' = g det(I - X_e C_ee)^(-1/2) exp(v_e^T P v_e / 2).
// delta -> -delta leaves a term's share unchanged (degree K in the deltas, as the weights), so
// the first edge takes half of its signs.  The last simple edges close: two of them in the hafnian
// of the 4 vertices left (their four sign pairs' sum), with loop weights one in C_ij + v_i v_j.
//
// What bounds it: the FP64 pipe (2 multiply-adds per clock and SM), i.e. the number of FP64 warp
// instructions; loads are a few bytes per clock even from L2.  So lanes are nodes (p fastest: the
// same entry and coefficients of 32 nodes, no idle lanes below the top few levels) and every
// thread forms tree_tile() consecutive coefficients of one entry in registers.  Measured against the
// per-term kernel (us a call): complex n = 24 568 -> 248, n = 40 244,700 -> 6,580; real n = 44
// (positive) 380,900 -> 9,010; 96 matrices of n = 8 .. 32 in a plan 61,850 -> 2,560; complex n = 28
// in double-double 22,330 -> 1,910, n = 34 in double-float 12,420 -> 520; a graph of 32 vertices
// modulo the primes of its exact count 9,090 -> 600.
// (The reference's tree for unit edges is thewalrus/_hafnian.py recursive_hafnian's squeeze; this
// one sums the finite-difference signs of _calc_hafnian / _calc_loop_hafnian, :443-577, and of
// loop_hafnian_batch.py:50-208.)
#pragma once
#include "sieve_kernel.cuh"

namespace wg {

constexpr int TREE_MAX_K = 63;
constexpr int TREE_MAX_POS = 3 + 2 * MAX_EDGES;
constexpr int TREE_THREADS = 256;

// The node functions also compile for the host, one thread as a warp of one lane: a CPU check runs
// them over a checked scalar type (tests/tree_check.cu).
#ifdef __CUDA_ARCH__
#define WG_TREE_LANES 32
#define WG_TREE_SYNCWARP() __syncwarp()
#else
#define WG_TREE_LANES 1
#define WG_TREE_SYNCWARP() ((void)0)
#endif

// coefficients a thread forms in registers
template <class S>
constexpr int tree_tile() { return Ar<S>::dd && Ar<S>::cplx ? 2 : 4; }

// One instance's tree.  Positions 0 .. X-1 are the rows that are never eliminated (pL: the loop
// weights, pO: an unpaired vertex, pB: the batch mode), then the edges' vertices, the last edge
// first: step q eliminates positions X + 2 (E-1-q) and the next, the highest two left.
struct TreeInst {
  long long a_off;           // byte offset of the extended matrix in the pool
  int lda;
  int E, K, X;
  int pL, pO, pB;            // -1: none
  int diag;                  // entries include the diagonal (multiple edges, or a batch mode)
  int dpos;                  // diagonal entries of positions >= dpos are kept (pending multiple edges)
  int steps;                 // edges eliminated by steps: E, E - 1 or E - 2 (tree_leaf's closed forms)
  int nout;
  int part_base, pstride, comp_off;  // partial slots of a task or leaf block (as InstDev's)
  int q;                     // CTA kernel: edges whose sign a task fixes
  int tasks, task_base;      // CTA kernel
  c64 oddloop;               // entry (pO, pL) when the unpaired vertex is not a vertex of A
  short row[TREE_MAX_POS], col[TREE_MAX_POS];  // position -> row and column of the extended matrix
  unsigned char reps[MAX_EDGES], radix[MAX_EDGES];
  unsigned char deg[MAX_EDGES + 4];  // degree of the series after q steps
};

struct TreeParams {
  const TreeInst* inst;
  int ninst, ntasks;
  const unsigned char* pool;
  unsigned char* ws;         // CTA kernel: per-CTA workspace
  long long ws_stride;
  long long off_b, off_s;    // second node buffer, scratch
  double2* partials;
  unsigned int* counter;
};

// grid mode: one launch per phase of a step
enum TreePhase : int { TP_ROOT = 0, TP_M, TP_UNIT, TP_PREP, TP_Y, TP_MULTI, TP_GLOOP, TP_LEAF };
struct TreeGrid {
  TreeParams P;
  int inst, phase, q;
  int np, p0, pstride;       // parents [p0, p0 + np) of a buffer of pstride nodes
  int d0, nd;                // digits d0 .. d0 + nd - 1
  long long part;            // leaf: first partial slot of the launch
  unsigned char *par, *chi, *scr;
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
__host__ __device__ __forceinline__ void tree_decode(int e, int diag, int& a, int& b) {
  const int x = e - 1;
  int r = (int)((sqrtf(8.0f * (float)x + 1.0f) - 1.0f) * 0.5f);
  while ((r + 1) * (r + 2) / 2 <= x) ++r;
  while (r * (r + 1) / 2 > x) --r;
  a = diag ? r : r + 1;
  b = x - r * (r + 1) / 2;
}

// one scalar in one access: the buffers are 16-byte aligned
#pragma nv_exec_check_disable
template <class S>
__host__ __device__ __forceinline__ S tld(const S* p) { return *p; }
template <>
__host__ __device__ __forceinline__ c64 tld<c64>(const c64* p) {
  const double2 v = *reinterpret_cast<const double2*>(p);
  return {v.x, v.y};
}
#pragma nv_exec_check_disable
template <class S>
__host__ __device__ __forceinline__ void tst(S* p, S v) { *p = v; }
template <>
__host__ __device__ __forceinline__ void tst<c64>(c64* p, c64 v) { *reinterpret_cast<double2*>(p) = make_double2(v.re, v.im); }

// acc[k] += sum_s a_s b_(t0+k-s), k < T, s < la: coefficients t0 .. t0+T-1 of a product of two
// series (element stride sa, sb).  A window of T coefficients of b slides through registers, so a
// step is one load of each series and T multiply-adds; the last T-1 steps are the triangle where b
// runs out.  t0 < 0: only the coefficients t0 + k >= 0.
#pragma nv_exec_check_disable
template <class S, int T>
__host__ __device__ __forceinline__ void conv_tile(S (&acc)[T], const S* a, long long sa, int la, const S* b,
                                          long long sb, int t0) {
  using A = Ar<S>;
  if (t0 < 0) {
#pragma unroll
    for (int k = 1; k < T; ++k) {
      const int t = t0 + k;
      if (t >= 0)
        for (int s = 0; s <= t && s < la; ++s) acc[k] = A::fma(tld(a + s * sa), tld(b + (t - s) * sb), acc[k]);
    }
    return;
  }
  S w[T];
#pragma unroll
  for (int k = 0; k < T; ++k) w[k] = tld(b + (t0 + k) * sb);
  const int sm = t0 < la - 1 ? t0 : la - 1;
  const S* pa = a;
  const S* pb = b + (t0 - 1) * sb;
#pragma unroll 4
  for (int s = 0; s <= sm; ++s) {
    const S x = tld(pa);
    pa += sa;
#pragma unroll
    for (int k = 0; k < T; ++k) acc[k] = A::fma(x, w[k], acc[k]);
#pragma unroll
    for (int k = T - 1; k > 0; --k) w[k] = w[k - 1];
    if (s < t0) w[0] = tld(pb);
    pb -= sb;
  }
  // s = t0 + kk: w[k] = b_(k-1) here
#pragma unroll
  for (int kk = 1; kk < T; ++kk) {
    if (t0 + kk < la) {
      const S x = tld(pa);
      pa += sa;
#pragma unroll
      for (int k = kk; k < T; ++k) acc[k] = A::fma(x, w[k - kk + 1], acc[k]);
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
  S r = A::zero();
  const int s0 = t - lb + 1 > 0 ? t - lb + 1 : 0;
  for (int s = s0; s <= t && s < la; ++s) r = A::fma(tld(a + s * sa), tld(b + (t - s) * sb), r);
  return r;
}

__host__ __device__ __forceinline__ bool tree_need(const TreeInst& T, int a, int b) {
  return a != b || a == T.pB || a >= T.dpos;
}

// ---- root: one node, one coefficient per entry
#pragma nv_exec_check_disable
template <class S>
__host__ __device__ void tree_root(const TreeInst& T, const unsigned char* __restrict__ pool, S* out, int tid,
                          int nthr) {
  using A = Ar<S>;
  const S* __restrict__ ext = reinterpret_cast<const S*>(pool + T.a_off);
  const int W = tree_width(T.X, T.E, 0), ne = tree_entries(W, T.diag);
  for (int e = tid; e < ne; e += nthr) {
    S v = A::one();
    if (e > 0) {
      int a, b;
      tree_decode(e, T.diag, a, b);
      const int ca = T.col[a], cb = T.col[b];
      if (ca < 0 || cb < 0) {  // the unpaired vertex has a row only, and its loop weight apart
        const int o = ca < 0 ? a : b, x = ca < 0 ? b : a;
        v = x == o ? A::zero() : (x == T.pL ? A::from_c64(T.oddloop) : ext[(size_t)T.row[o] * T.lda + T.col[x]]);
      } else {
        // the mean of the two triangles: equal to either when they agree
        const S x = ext[(size_t)T.row[a] * T.lda + cb], y = ext[(size_t)T.row[b] * T.lda + ca];
        v = A::add(x, tree_half(A::sub(y, x)));
      }
    }
    tst(out + e, v);
  }
}

// ---- m = C_ij + v_i v_j of the edge of step q (loop kinds): scr[t np + p]
#pragma nv_exec_check_disable
template <class S>
__host__ __device__ void tree_m(const TreeInst& T, int q, const S* par, long long ps, int np, S* scr,
                       int tid, int nthr) {
  using A = Ar<S>;
  constexpr int TL = tree_tile<S>();
  const int i = T.X + 2 * (T.E - 1 - q), j = i + 1;
  const int Lp = T.deg[q] + 1, nt = (Lp + TL - 1) / TL;
  for (int x = tid; x < nt * np; x += nthr) {
    const int p = x % np, t0 = Lp - TL * (x / np + 1);
    S acc[TL];
#pragma unroll
    for (int k = 0; k < TL; ++k)
      acc[k] = t0 + k >= 0 ? tld(par + ((long long)tree_ent(j, i, T.diag) * Lp + t0 + k) * ps + p) : A::zero();
    conv_tile<S, TL>(acc, par + (long long)tree_ent(i, T.pL, T.diag) * Lp * ps + p, ps, Lp,
                     par + (long long)tree_ent(j, T.pL, T.diag) * Lp * ps + p, ps, t0);
#pragma unroll
    for (int k = 0; k < TL; ++k)
      if (t0 + k >= 0) tst(scr + (long long)(t0 + k) * np + p, acc[k]);
  }
}

// ---- a simple edge: children delta = +1 (nodes 0 .. np-1) and -1 (np .. 2 np - 1) from the same
// products; digits d0 .. d0 + nd - 1 are made (0: +1, 1: -1).  The weight -1 of the second joins g.
#pragma nv_exec_check_disable
template <class S>
__host__ __device__ void tree_unit(const TreeInst& T, int q, const S* par, long long ps, int np,
                          const S* m, S* chi, int d0, int nd, int tid, int nthr) {
  using A = Ar<S>;
  constexpr int TL = tree_tile<S>();
  const int i = T.X + 2 * (T.E - 1 - q), j = i + 1, dg = T.diag;
  const int ne = tree_entries(i, dg), Lp = T.deg[q] + 1, Lc = Lp + 1, nt = (Lp + TL - 1) / TL;
  const long long cs = (long long)np * nd;
  const unsigned total = (unsigned)nt * ne * np;
  for (unsigned x = tid; x < total; x += nthr) {
    const unsigned r = x / np;
    const int p = x - r * np, e = r % ne, t0 = Lp - TL * ((int)(r / ne) + 1);
    const S* pp = par + p;
    S acc[TL];
#pragma unroll
    for (int k = 0; k < TL; ++k) acc[k] = A::zero();
    if (e == 0) {
      if (T.pL >= 0) conv_tile<S, TL>(acc, pp, ps, Lp, m + p, np, t0);
      else conv_tile<S, TL>(acc, pp, ps, Lp, pp + (long long)tree_ent(j, i, dg) * Lp * ps, ps, t0);
    } else {
      int a, b;
      tree_decode(e, dg, a, b);
      if (!tree_need(T, a, b)) continue;
      const long long st = (long long)Lp * ps;
      conv_tile<S, TL>(acc, pp + tree_ent(i, a, dg) * st, ps, Lp, pp + tree_ent(j, b, dg) * st, ps, t0);
      conv_tile<S, TL>(acc, pp + tree_ent(j, a, dg) * st, ps, Lp, pp + tree_ent(i, b, dg) * st, ps, t0);
    }
    const S* base = pp + (long long)e * Lp * ps;
    S* o = chi + (long long)e * Lc * cs + p;
#pragma unroll
    for (int k = -1; k < TL; ++k) {  // coefficient t + 1 of the children; k = -1: coefficient 0
      const int t = t0 + k;
      if (k < 0 ? t0 <= 0 : t >= 0) {
        const int tc = k < 0 ? 0 : t + 1;
        const S c = tc < Lp ? tld(base + tc * ps) : A::zero();
        const S u = k < 0 ? A::zero() : acc[k < 0 ? 0 : k];
        S* w = o + tc * cs;
        if (d0 == 0) {
          tst(w, A::add(c, u));
          w += np;
        }
        if (d0 + nd > 1) tst(w, e == 0 ? A::sub(u, c) : A::sub(c, u));
      }
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

// Series of the edge's 2 x 2 block, one warp per child: scr[(f Lc + t) nc + x], f = 0..2 the entries
// P_ii, P_ij, P_jj, f = 3 the factor h = Delta^(-1/2) (Delta = (1 - z c)^2 - z^2 a b, z = delta eta,
// a, b, c = C_ii, C_jj, C_ij), f = 4.. work; without loop weights also the child's g = w g h.
#pragma nv_exec_check_disable
template <class S>
__host__ __device__ void tree_prep(const TreeInst& T, int q, const S* par, long long ps, int np, S* scr,
                          S* chi, int d0, int nd, int tid, int nthr) {
  using A = Ar<S>;
  const int i = T.X + 2 * (T.E - 1 - q), j = i + 1, r = T.reps[q];
  const int Lp = T.deg[q] + 1, Lc = Lp + r, nc = np * nd;
  const int lane = tid & (WG_TREE_LANES - 1);
  for (int x = tid / WG_TREE_LANES; x < nc; x += nthr / WG_TREE_LANES) {
    const int p = x % np, d = d0 + x / np;
    const double z = (double)(r - 2 * d);
    const S* pp = par + p;
    const S* ca = pp + (long long)tree_ent(i, i, 1) * Lp * ps;
    const S* cb = pp + (long long)tree_ent(j, j, 1) * Lp * ps;
    const S* cc = pp + (long long)tree_ent(j, i, 1) * Lp * ps;
    auto at = [&](int f, int t) -> S& { return scr[((long long)f * Lc + t) * nc + x]; };
    const long long fs = (long long)Lc * nc;
    // Delta = 1 - 2 z c + z^2 (c c - a b), f = 4
    for (int t = lane; t < Lc; t += WG_TREE_LANES) {
      S v = t == 0 ? A::one() : A::zero();
      if (t >= 1 && t - 1 < Lp) v = A::sub(v, A::scale(tld(cc + (t - 1) * ps), 2.0 * z));
      if (t >= 2) {
        const S k = A::sub(conv_one(cc, ps, Lp, cc, ps, Lp, t - 2), conv_one(ca, ps, Lp, cb, ps, Lp, t - 2));
        v = A::add(v, A::scale(k, z * z));
      }
      at(4, t) = v;
      at(3, t) = t == 0 ? A::one() : A::zero();
    }
    WG_TREE_SYNCWARP();
    // h = Delta^(-1/2), right-looking as in inv_sqrt_series
    for (int k = 0; k + 1 < Lc; ++k) {
      const S gk = at(3, k);
      for (int t = k + 1 + lane; t < Lc; t += WG_TREE_LANES) {
        S acc;
        if constexpr (A::modular) {
          acc = A::fma(at(4, t - k), A::mul(gk, A::mul(A::of_int(t + k), A::half())), at(3, t));
          if (t == k + 1) acc = A::neg(tree_div(acc, t));
        } else {
          acc = A::fma(at(4, t - k), A::scale_f(gk, 0.5f * (float)(t + k)), at(3, t));
          if (t == k + 1) acc = A::neg(tree_div(acc, t));
        }
        at(3, t) = acc;
      }
      WG_TREE_SYNCWARP();
    }
    const S* h = scr + 3 * fs + x;
    S* hh = scr + 5 * fs + x;  // 1 / Delta
    for (int t = lane; t < Lc; t += WG_TREE_LANES) hh[(long long)t * nc] = conv_one(h, nc, Lc, h, nc, Lc, t);
    WG_TREE_SYNCWARP();
    // P = z / Delta [[z b, 1 - z c], [1 - z c, z a]]
    for (int t = lane; t < Lc; t += WG_TREE_LANES) {
      S pi = A::zero(), pj = A::zero(), pc = A::zero();
      if (t >= 1) pc = A::scale(hh[(long long)(t - 1) * nc], z);
      if (t >= 2) {
        pi = A::scale(conv_one((const S*)hh, nc, Lc, cb, ps, Lp, t - 2), z * z);
        pj = A::scale(conv_one((const S*)hh, nc, Lc, ca, ps, Lp, t - 2), z * z);
        pc = A::sub(pc, A::scale(conv_one((const S*)hh, nc, Lc, cc, ps, Lp, t - 2), z * z));
      }
      at(0, t) = pi;
      at(1, t) = pc;
      at(2, t) = pj;
    }
    if (T.pL < 0) {
      const double w = tree_weight(T, q, d);
      for (int t = lane; t < Lc; t += WG_TREE_LANES)
        tst(chi + (long long)t * nc + x, A::scale(conv_one(h, nc, Lc, pp, ps, Lp, t), w));
    }
    WG_TREE_SYNCWARP();
  }
}

// Y = P C_e,b for every remaining row b: scr_y[((2 b + s) Lc + t) nc + x]
#pragma nv_exec_check_disable
template <class S>
__host__ __device__ void tree_y(const TreeInst& T, int q, const S* par, long long ps, int np,
                       const S* scr, S* y, int nd, int tid, int nthr) {
  using A = Ar<S>;
  constexpr int TL = tree_tile<S>();
  const int i = T.X + 2 * (T.E - 1 - q), j = i + 1, W = i;
  const int Lp = T.deg[q] + 1, Lc = Lp + T.reps[q], nc = np * nd, nt = (Lc + TL - 1) / TL;
  const long long fs = (long long)Lc * nc;
  for (int x = tid; x < nt * 2 * W * nc; x += nthr) {
    const int r = x / nc, c = x - r * nc, bs = r % (2 * W), t0 = Lc - TL * (r / (2 * W) + 1);
    const int b = bs >> 1, s = bs & 1, p = c % np;
    S acc[TL];
#pragma unroll
    for (int k = 0; k < TL; ++k) acc[k] = A::zero();
    conv_tile<S, TL>(acc, par + (long long)tree_ent(i, b, T.diag) * Lp * ps + p, ps, Lp, scr + s * fs + c, nc, t0);
    conv_tile<S, TL>(acc, par + (long long)tree_ent(j, b, T.diag) * Lp * ps + p, ps, Lp, scr + (s + 1) * fs + c, nc,
                     t0);
#pragma unroll
    for (int k = 0; k < TL; ++k)
      if (t0 + k >= 0) tst(y + (long long)bs * fs + (long long)(t0 + k) * nc + c, acc[k]);
  }
}

// C' = C + C_ae Y(b)
#pragma nv_exec_check_disable
template <class S>
__host__ __device__ void tree_multi(const TreeInst& T, int q, const S* par, long long ps, int np,
                           const S* y, S* chi, int nd, int tid, int nthr) {
  using A = Ar<S>;
  constexpr int TL = tree_tile<S>();
  const int i = T.X + 2 * (T.E - 1 - q), j = i + 1, dg = T.diag;
  const int ne = tree_entries(i, dg) - 1;
  const int Lp = T.deg[q] + 1, Lc = Lp + T.reps[q], nc = np * nd, nt = (Lc + TL - 1) / TL;
  const long long fs = (long long)Lc * nc, st = (long long)Lp * ps;
  const unsigned total = (unsigned)nt * ne * nc;
  for (unsigned x = tid; x < total; x += nthr) {
    const unsigned r = x / nc;
    const int c = x - r * nc, e = 1 + r % ne, t0 = Lc - TL * ((int)(r / ne) + 1), p = c % np;
    int a, b;
    tree_decode(e, dg, a, b);
    if (!tree_need(T, a, b)) continue;
    const S* base = par + p + (long long)e * st;
    S acc[TL];
#pragma unroll
    for (int k = 0; k < TL; ++k) {
      const int t = t0 + k;
      acc[k] = t >= 0 && t < Lp ? tld(base + t * ps) : A::zero();
    }
    conv_tile<S, TL>(acc, par + p + tree_ent(i, a, dg) * st, ps, Lp, y + (long long)(2 * b) * fs + c, nc, t0);
    conv_tile<S, TL>(acc, par + p + tree_ent(j, a, dg) * st, ps, Lp, y + (long long)(2 * b + 1) * fs + c, nc, t0);
#pragma unroll
    for (int k = 0; k < TL; ++k)
      if (t0 + k >= 0) tst(chi + (long long)e * fs + (long long)(t0 + k) * nc + c, acc[k]);
  }
}

// loop kinds: g' = w g h exp(v_e Y(L) / 2), one warp per child
#pragma nv_exec_check_disable
template <class S>
__host__ __device__ void tree_gloop(const TreeInst& T, int q, const S* par, long long ps, int np, S* scr,
                           const S* y, S* chi, int d0, int nd, int tid, int nthr) {
  using A = Ar<S>;
  const int i = T.X + 2 * (T.E - 1 - q), j = i + 1;
  const int Lp = T.deg[q] + 1, Lc = Lp + T.reps[q], nc = np * nd;
  const long long fs = (long long)Lc * nc, st = (long long)Lp * ps;
  const int lane = tid & (WG_TREE_LANES - 1);
  for (int x = tid / WG_TREE_LANES; x < nc; x += nthr / WG_TREE_LANES) {
    const int p = x % np, d = d0 + x / np;
    const S* vi = par + p + tree_ent(i, T.pL, T.diag) * st;
    const S* vj = par + p + tree_ent(j, T.pL, T.diag) * st;
    const S* yi = y + (long long)(2 * T.pL) * fs + x;
    const S* yj = y + (long long)(2 * T.pL + 1) * fs + x;
    S* u = scr + 4 * fs + x;
    S* ex = scr + 5 * fs + x;
    S* gh = scr + x;  // P is no longer needed here
    for (int t = lane; t < Lc; t += WG_TREE_LANES) {
      u[(long long)t * nc] = tree_half(A::add(conv_one(vi, ps, Lp, yi, nc, Lc, t), conv_one(vj, ps, Lp, yj, nc, Lc, t)));
      ex[(long long)t * nc] = t == 0 ? A::one() : A::zero();
    }
    WG_TREE_SYNCWARP();
    for (int k = 0; k + 1 < Lc; ++k) {  // exp, right-looking as in exp_series
      const S ek = ex[(long long)k * nc];
      for (int t = k + 1 + lane; t < Lc; t += WG_TREE_LANES) {
        S acc;
        const S ut = u[(long long)(t - k) * nc];
        if constexpr (A::modular) {
          acc = A::fma(A::mul(ut, A::of_int(t - k)), ek, ex[(long long)t * nc]);
          if (t == k + 1) acc = tree_div(acc, t);
        } else {
          acc = A::fma(A::scale_f(ut, (float)(t - k)), ek, ex[(long long)t * nc]);
          if (t == k + 1) acc = tree_div(acc, t);
        }
        ex[(long long)t * nc] = acc;
      }
      WG_TREE_SYNCWARP();
    }
    const S* h = scr + 3 * fs + x;
    for (int t = lane; t < Lc; t += WG_TREE_LANES) gh[(long long)t * nc] = conv_one(h, nc, Lc, par + p, ps, Lp, t);
    WG_TREE_SYNCWARP();
    const double w = tree_weight(T, q, d);
    for (int t = lane; t < Lc; t += WG_TREE_LANES)
      tst(chi + (long long)t * nc + x, A::scale(conv_one((const S*)ex, nc, Lc, (const S*)gh, nc, Lc, t), w));
    WG_TREE_SYNCWARP();
  }
}

// ---- leaves: this thread's share of the output (batch: the sums of the warp, left in sm) over nodes [0, np) of a buffer of stride ps
#pragma nv_exec_check_disable
template <class S>
__host__ __device__ S tree_leaf(const TreeInst& T, const S* par, long long ps, int np, const S* m, S* sm, int wb,
                                int tid, int nthr) {
  using A = Ar<S>;
  constexpr int TL = tree_tile<S>();
  const int L = T.deg[T.steps] + 1, D = L - 1, dg = T.diag;
  const long long st = (long long)L * ps;
  S sum = A::zero();
  if (T.steps < T.E) {
    // simple edges left: the coefficient of their deltas at once, [eta^D] g h, one thread per node
    // and tile of h.  Two edges on X .. X+3 (no loop weights): h = haf(4 x 4).  One edge on X, X+1:
    // h = C_ij + v_i v_j; with an unpaired vertex o, h = v_o (C_ij + v_i v_j) + C_io v_j + C_jo v_i
    // (m = C_ij + v_i v_j from tree_m).
    const int nt = (L + TL - 1) / TL, X = T.X;
    const bool two = T.E - T.steps == 2;
    for (int x = tid; x < nt * np; x += nthr) {
      const int p = x % np, t0 = L - TL * (x / np + 1);
      const S* pp = par + p;
      S acc[TL];
#pragma unroll
      for (int k = 0; k < TL; ++k) acc[k] = A::zero();
      if (!two && T.pO < 0) {
#pragma unroll
        for (int k = 0; k < TL; ++k)
          if (t0 + k >= 0) acc[k] = tld(pp + tree_ent(X + 1, X, dg) * st + (t0 + k) * ps);
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
        conv_tile<S, TL>(acc, u, su, L, v, ps, t0);
      }
#pragma unroll
      for (int k = 0; k < TL; ++k)
        if (t0 + k >= 0) sum = A::fma(tld(pp + (D - t0 - k) * ps), acc[k], sum);
    }
  } else if (T.pB < 0) {
    for (int p = tid; p < np; p += nthr) {
      if (T.pO < 0) {
        sum = A::add(sum, tld(par + D * ps + p));
      } else {
        const S* vo = par + p + (long long)tree_ent2(T.pO, T.pL, dg) * st;
        for (int s = 0; s <= D; ++s) sum = A::fma(tld(par + p + (D - s) * ps), tld(vo + s * ps), sum);
      }
    }
  } else {
    // batch mode b with loop series v and pair series c: k photons give H_k = v H_(k-1) +
    // (k-1) c H_(k-2); with an unpaired vertex o: v_o H_k + k c_ob H_(k-1).  One warp per node, its
    // work series and the output sums in the warp's part of sm.
    const int lane = tid & (WG_TREE_LANES - 1), nw = nthr / WG_TREE_LANES;
    S* const base = sm + wb * (5 * L + 32);
    S *gv = base + 3 * L, *gc = base + 4 * L, *o = base + 5 * L;
    for (int k = lane; k < T.nout; k += WG_TREE_LANES) o[k] = A::zero();
    WG_TREE_SYNCWARP();
    for (int p = tid / WG_TREE_LANES; p < np; p += nw) {
      const S* pp = par + p;
      const S* v = pp + (long long)tree_ent2(T.pB, T.pL, dg) * st;
      const S* c = pp + (long long)tree_ent(T.pB, T.pB, 1) * st;
      S *h0 = base, *h1 = base + L, *h2 = base + 2 * L;
      for (int t = lane; t < L; t += WG_TREE_LANES) {
        h0[t] = A::zero();
        h1[t] = t == 0 ? A::one() : A::zero();
        if (T.pO >= 0) {
          gv[t] = conv_one(pp, ps, L, pp + (long long)tree_ent2(T.pO, T.pL, dg) * st, ps, L, t);
          gc[t] = conv_one(pp, ps, L, pp + (long long)tree_ent2(T.pO, T.pB, dg) * st, ps, L, t);
        } else {
          gv[t] = tld(pp + t * ps);
          gc[t] = A::zero();
        }
      }
      WG_TREE_SYNCWARP();
      for (int k = 0; k < T.nout; ++k) {  // h1 = H_k, h0 = H_(k-1)
        S part = A::zero();
        for (int t = lane; t < L; t += WG_TREE_LANES) {
          part = A::fma(gv[D - t], h1[t], part);
          if (k && T.pO >= 0) part = A::fma(tree_times(gc[D - t], k), h0[t], part);
          if (k + 1 < T.nout) {
            S n = conv_one(v, ps, L, (const S*)h1, 1, L, t);
            if (k) n = A::add(n, tree_times(conv_one(c, ps, L, (const S*)h0, 1, L, t), k));
            h2[t] = n;
          }
        }
#ifdef __CUDA_ARCH__
        part = warp_sum(part);
#endif
        if (lane == 0) o[k] = A::add(o[k], part);
        WG_TREE_SYNCWARP();
        S* u = h0;
        h0 = h1;
        h1 = h2;
        h2 = u;
      }
    }
  }
  return sum;
}

// block sum of the leaf shares in a fixed order, into the partial slots
template <class S>
__device__ void tree_store(const TreeInst& T, S sum, long long slot, double2* __restrict__ partials, S* red) {
  using A = Ar<S>;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const bool batch = T.pB >= 0;
  const int L = T.deg[T.steps] + 1;
  if (!batch) {
    sum = warp_sum(sum);
    if (lane == 0) red[warp] = sum;
  }
  __syncthreads();
  if (warp == 0 && lane < T.nout) {
    S s = A::zero();
    for (int w = 0; w < nw; ++w) s = A::add(s, batch ? red[w * (5 * L + 32) + 5 * L + lane] : red[w]);
    const c64 z = A::to_c64(s);
    partials[slot + lane] = make_double2(z.re, z.im);
    if constexpr (A::dd) {
      const c64 zl = A::lo_c64(s);
      partials[slot + T.comp_off + lane] = make_double2(zl.re, zl.im);
    }
  }
  __syncthreads();
}

// ---- one CTA per task: the path of the task's first q signs, then the whole subtree below it,
// level by level in the CTA's own workspace (two node buffers and scratch, L2 resident)
template <class S>
static __global__ void __launch_bounds__(TREE_THREADS, 2) tree_cta_kernel(const TreeParams P) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ TreeInst T;
  __shared__ int s_task;
  S* sm = reinterpret_cast<S*>(smem);
  unsigned char* ws = P.ws + (long long)blockIdx.x * P.ws_stride;
  S* buf[2] = {reinterpret_cast<S*>(ws), reinterpret_cast<S*>(ws + P.off_b)};
  S* scr = reinterpret_cast<S*>(ws + P.off_s);
  const int tid = threadIdx.x, nthr = blockDim.x;
  for (;;) {
    if (tid == 0) s_task = (int)atomicAdd(P.counter, 1u);
    __syncthreads();
    const int task = s_task;
    if (task >= P.ntasks) break;
    int lo = 0, hi = P.ninst - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (P.inst[mid].task_base <= task) lo = mid; else hi = mid - 1;
    }
    {
      const int* src = reinterpret_cast<const int*>(P.inst + lo);
      int* dst = reinterpret_cast<int*>(&T);
      for (int w = tid; w < (int)(sizeof(TreeInst) / 4); w += nthr) dst[w] = src[w];
    }
    __syncthreads();
    int code = task - T.task_base;
    tree_root<S>(T, P.pool, buf[0], tid, nthr);
    __syncthreads();
    int cur = 0, np = 1;
    for (int q = 0; q < T.steps; ++q) {
      const int R = T.radix[q];
      int d0 = 0, nd = R;
      if (q < T.q) {
        d0 = code % R;
        code /= R;
        nd = 1;
      }
      const S* par = buf[cur];
      S* chi = buf[cur ^ 1];
      if (T.reps[q] == 1) {
        if (T.pL >= 0) {
          tree_m<S>(T, q, par, np, np, scr, tid, nthr);
          __syncthreads();
        }
        tree_unit<S>(T, q, par, np, np, scr, chi, d0, nd, tid, nthr);
      } else {
        const int Lc = T.deg[q] + 1 + T.reps[q];
        S* y = scr + 6ll * Lc * np * nd;
        tree_prep<S>(T, q, par, np, np, scr, chi, d0, nd, tid, nthr);
        __syncthreads();
        if (tree_width(T.X, T.E, q + 1) > 0) {
          tree_y<S>(T, q, par, np, np, scr, y, nd, tid, nthr);
          __syncthreads();
          tree_multi<S>(T, q, par, np, np, y, chi, nd, tid, nthr);
          if (T.pL >= 0) tree_gloop<S>(T, q, par, np, np, scr, y, chi, d0, nd, tid, nthr);
        }
      }
      np *= nd;
      cur ^= 1;
      __syncthreads();
    }
    if (T.steps < T.E && T.pO >= 0) {
      tree_m<S>(T, T.steps, buf[cur], np, np, scr, tid, nthr);
      __syncthreads();
    }
    const S sum = tree_leaf<S>(T, buf[cur], np, np, scr, sm, tid >> 5, tid, nthr);
    tree_store<S>(T, sum, T.part_base + (long long)(task - T.task_base) * T.pstride, P.partials, sm);
  }
}

// ---- one phase of one step over a whole block of nodes
template <class S>
static __global__ void __launch_bounds__(TREE_THREADS, 2) tree_grid_kernel(const TreeGrid G) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ TreeInst T;
  {
    const int* src = reinterpret_cast<const int*>(G.P.inst + G.inst);
    int* dst = reinterpret_cast<int*>(&T);
    for (int w = threadIdx.x; w < (int)(sizeof(TreeInst) / 4); w += blockDim.x) dst[w] = src[w];
  }
  __syncthreads();
  const int tid = blockIdx.x * blockDim.x + threadIdx.x, nthr = gridDim.x * blockDim.x;
  const S* par = reinterpret_cast<const S*>(G.par) + G.p0;
  S* chi = reinterpret_cast<S*>(G.chi);
  S* scr = reinterpret_cast<S*>(G.scr);
  switch (G.phase) {
    case TP_ROOT: tree_root<S>(T, G.P.pool, chi, tid, nthr); break;
    case TP_M: tree_m<S>(T, G.q, par, G.pstride, G.np, scr, tid, nthr); break;
    case TP_UNIT: tree_unit<S>(T, G.q, par, G.pstride, G.np, scr, chi, G.d0, G.nd, tid, nthr); break;
    case TP_PREP: tree_prep<S>(T, G.q, par, G.pstride, G.np, scr, chi, G.d0, G.nd, tid, nthr); break;
    case TP_LEAF: {
      const S sum = tree_leaf<S>(T, par, G.pstride, G.np, scr, reinterpret_cast<S*>(smem), threadIdx.x >> 5, tid, nthr);
      tree_store<S>(T, sum, G.part + (long long)blockIdx.x * T.pstride, G.P.partials, reinterpret_cast<S*>(smem));
      break;
    }
    default: {
      S* y = scr + 6ll * (T.deg[G.q] + 1 + T.reps[G.q]) * G.np * G.nd;
      if (G.phase == TP_Y) tree_y<S>(T, G.q, par, G.pstride, G.np, scr, y, G.nd, tid, nthr);
      else if (G.phase == TP_MULTI) tree_multi<S>(T, G.q, par, G.pstride, G.np, y, chi, G.nd, tid, nthr);
      else tree_gloop<S>(T, G.q, par, G.pstride, G.np, scr, y, chi, G.d0, G.nd, tid, nthr);
    }
  }
}

}  // namespace wg
