// Host runtime and C ABI of the hafnian sieve (see include/walrus_gb300.h).
//
// A plan turns a list of prepared instances into
//   * one device pool holding each instance's extended matrix [[A, D], [D^T, 0], [oddV], [oddV0]]
//     converted to the kernel's scalar type,
//   * a chunk queue: every instance's term range split into chunks whose cost is balanced
//     against the number of resident warps, largest instances first,
//   * the elimination tree of every instance that takes one (tree_kernel.cuh): one cooperative launch
//     per scalar type and workspace budget, whose rounds hold the levels of all its trees,
//   * for the others (term ranges, inclusion/exclusion, per-term precisions, matrices that are not
//     symmetric) one persistent sieve launch per (scalar type, resident warps per SM) group,
//   * one reduction launch that sums the partials in a fixed order (bitwise reproducible results);
//     a plan of a single tree launch and few outputs reduces in it.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/walrus_gb300.h"
#include "host_common.h"
#include "sieve_kernel.cuh"
#include "state_glue.cuh"
#include "tree_host.h"

namespace wg {

static thread_local std::string g_err;
// Per-device state: the selected device, and for every device the SM count and the La Budde
// schedule tables in its memory (the constant tables live in each device's copy of the module).
static int g_device = -1;
static int g_num_sms = 0;  // of g_device
constexpr int kMaxDev = 64;
struct DevTables {
  bool ready = false;
  int sms = 0;
  LbLane* lane = nullptr;
  LbOwner* own = nullptr;
  LbLane2* lane2 = nullptr;
  LbOwner2* own2 = nullptr;
};
static DevTables g_dev[kMaxDev];

static std::mutex g_init_mu;

// lets other translation units of the library report through wg_last_error()
void set_last_error(const char* msg) { g_err = msg; }

static int fail(int code, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  g_err = buf;
  return code;
}

#define CK(x)                                                                                   \
  do {                                                                                          \
    cudaError_t e_ = (x);                                                                       \
    if (e_ != cudaSuccess) return fail(WG_ECUDA, "%s: %s (%s:%d)", #x, cudaGetErrorString(e_), \
                                       __FILE__, __LINE__);                                     \
  } while (0)

// Pinned blocks for the one-shot calls: a call stages its upload in one and its kernels write the
// results there, so neither passes through pageable memory (a small call's result took 9 us to
// come back by a copy).  A call takes a block and returns it when it has waited for its stream; at
// most kMaxPinned are kept for the next calls of any thread, more are freed.
constexpr size_t kPinnedBytes = 256 << 10;
constexpr size_t kMaxPinned = 16;
static std::mutex g_pinned_mu;
static std::vector<unsigned char*> g_pinned;

static unsigned char* pinned_take() {
  {
    std::lock_guard<std::mutex> lk(g_pinned_mu);
    if (!g_pinned.empty()) {
      unsigned char* p = g_pinned.back();
      g_pinned.pop_back();
      return p;
    }
  }
  void* p = nullptr;
  if (cudaHostAlloc(&p, kPinnedBytes, cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  return (unsigned char*)p;
}
static void pinned_give(unsigned char* p) {
  if (!p) return;
  {
    std::lock_guard<std::mutex> lk(g_pinned_mu);
    if (g_pinned.size() < kMaxPinned) {
      g_pinned.push_back(p);
      return;
    }
  }
  cudaFreeHost(p);
}

static int ensure_init(int device) {
  std::lock_guard<std::mutex> lk(g_init_mu);
  if (g_device >= 0 && (device < 0 || device == g_device)) {
    CK(cudaSetDevice(g_device));
    return WG_OK;
  }
  int dev = device < 0 ? 0 : device;
  int count = 0;
  CK(cudaGetDeviceCount(&count));
  if (count <= 0) return fail(WG_ECUDA, "no CUDA device");
  if (dev >= count || dev >= kMaxDev) return fail(WG_EINVAL, "device %d not present (%d devices)", dev, count);
  CK(cudaSetDevice(dev));
  DevTables& T = g_dev[dev];
  if (T.ready) {
    g_device = dev;
    g_num_sms = T.sms;
    return WG_OK;
  }
  CK(cudaDeviceGetAttribute(&T.sms, cudaDevAttrMultiProcessorCount, dev));
  // stream-ordered plans (one-shot calls, serving batches) allocate from this process's default
  // pool of the device: keep up to 1.5 GiB of freed memory (a large tree's levels) there instead of releasing it to the
  // CUDA driver at every synchronisation, so a repeated call reuses it
  cudaMemPool_t pool;
  CK(cudaDeviceGetDefaultMemPool(&pool, dev));
  unsigned long long keep = 1536ull << 20;
  CK(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
  // constant tables: binomials and reciprocals
  static double binom[BINOM_N][BINOM_N];
  for (int i = 0; i < BINOM_N; ++i)
    for (int j = 0; j < BINOM_N; ++j) {
      if (j > i) { binom[i][j] = 0; continue; }
      long double b = 1;
      for (int q = 0; q < j; ++q) b = b * (long double)(i - q) / (long double)(q + 1);
      binom[i][j] = (double)b;
    }
  double inv[256];
  inv[0] = 0;
  for (int k = 1; k < 256; ++k) inv[k] = 1.0 / (double)k;
  CK(sieve_tables_all(&binom[0][0], inv));
  // La Budde lane schedules for every triangle size (built once, kept for the process lifetime)
  std::vector<LbLane> lanes((LB_KMAX + 1) * 32);
  std::vector<LbOwner> own((LB_KMAX + 1) * (LB_KMAX + 1));
  for (int k = 0; k <= LB_KMAX; ++k)
    if (!lb_schedule(k, &lanes[k * 32], &own[k * (LB_KMAX + 1)]))
      return fail(WG_EINVAL, "no La Budde schedule for %d coefficients", k);
  CK(cudaMalloc(&T.lane, sizeof(LbLane) * lanes.size()));
  CK(cudaMalloc(&T.own, sizeof(LbOwner) * own.size()));
  CK(cudaMemcpy(T.lane, lanes.data(), sizeof(LbLane) * lanes.size(), cudaMemcpyHostToDevice));
  CK(cudaMemcpy(T.own, own.data(), sizeof(LbOwner) * own.size(), cudaMemcpyHostToDevice));
  std::vector<LbLane2> lanes2(LB2_IDS * 32);
  std::vector<LbOwner2> own2(LB2_IDS * (LB2_KMAX + 1));
  if (!lb_schedule2_all(lanes2.data(), own2.data())) return fail(WG_EINVAL, "no two-row La Budde schedule");
  CK(cudaMalloc(&T.lane2, sizeof(LbLane2) * lanes2.size()));
  CK(cudaMalloc(&T.own2, sizeof(LbOwner2) * own2.size()));
  CK(cudaMemcpy(T.lane2, lanes2.data(), sizeof(LbLane2) * lanes2.size(), cudaMemcpyHostToDevice));
  CK(cudaMemcpy(T.own2, own2.data(), sizeof(LbOwner2) * own2.size(), cudaMemcpyHostToDevice));
  T.ready = true;
  g_device = dev;
  g_num_sms = T.sms;
  return WG_OK;
}


// What the choice of evaluation looks at in a matrix: symmetric to rounding (and finite), real
// entries of both signs, indices that fall into uncoupled blocks (zero entries between them).
struct MatrixForm {
  bool symmetric = false, signs = false, blocks = false;
  bool mixed = false;  // complex entries have parts of like size (mixed_rows)
  bool full = false;   // finite, with no entry zero
  double diff = 0;     // largest difference between the triangles
};

// sums over entries of the smaller and of the larger part (mixed_rows)
struct PartSums {
  double low = 0, high = 0;
  void add(double re, double im) {
    const double x = std::fabs(re), y = std::fabs(im);
    low += std::min(x, y);
    high += std::max(x, y);
  }
  void add(c64 a, c64 b) { add(a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re); }
  bool mixed() const { return low >= 0.125 * high; }
};

struct Prepared {
  InstDev d;
  int stype;
  int rows_max, mb_max, m_max, kc_max, nser_need, narr;
  bool tile_ok;  // every term can keep its La Budde rows in dead tile columns
  double term_cost;
  std::vector<double> scales;
  std::vector<unsigned char> ext;  // extended matrix in the kernel's scalar type (empty: formed on device)
  size_t ext_bytes = 0;
  long long t_lo = 0, t_hi = 0;  // sieve terms [t_lo, t_hi) of this instance
  bool tree = false;             // evaluated as an elimination tree
  TreeInst T;
  std::vector<double> ascale;    // the input prescale's share of each output
  int precision;
  bool mixed = false;            // (MatrixForm)
  bool forced = false;           // WG_PREC_TREE
  std::vector<double> tscales() const;  // output scales of the tree's sum
  int ttype() const {            // the tree's node type
    const bool cplx = stype == ST_CPLX64 || stype == ST_CPLXDF || stype == ST_CPLXDD;
    return cplx && !mixed ? stype | TREE_PARTS : stype;
  }
};

struct Group {
  int stype;
  WarpLayout L;
  int wpc, ctas;
  int chunk_begin, chunk_count;
};

// the evaluations that may be added to a precision
constexpr int kEvaluations = WG_PREC_TERMS | WG_PREC_TREE;

// One launch of the tree kernel: trees of one scalar type and the program that walks them.
struct TreeLaunch {
  int ttype, ctas, smem, sm_warp, sm_cache, sm_ws, cached, counter;
  int ninst, nrounds, nsegs;
  size_t prog_off;  // of the instances, rounds and segments in the plan's program bytes
  long long ws_off;
};

}  // namespace wg

struct wg_plan {
  std::vector<wg::InstDev> inst;
  std::vector<wg::ChunkDev> chunks;
  std::vector<wg::Group> groups;
  int total_out = 0;
  int nparts = 0;
  long long h2d_bytes = 0;
  int precision = 0;
  int primes = 1;           // > 1: every instance modulo so many primes, all instances of one first
  bool side_trees = false;  // the primes' trees run side by side in one launch
  bool fork_trees = false;  // the scalar types' on side streams, each on its share of the SMs
  void* dmem = nullptr;
  wg::InstDev* d_inst = nullptr;
  wg::ChunkDev* d_chunks = nullptr;
  unsigned char* d_pool = nullptr;
  double2* d_partials = nullptr;
  double* d_scales = nullptr;
  double2* d_out = nullptr;
  double* d_mag = nullptr;  // per output: sum |prefactor x term| x |final scale|
  unsigned int* d_counters = nullptr;
  int* d_err = nullptr;
  bool use_graph = false;
  cudaGraphExec_t graph_exec = nullptr;
  long long device_bytes = 0;
  bool async_alloc = false;
  cudaStream_t alloc_stream = nullptr;
  // groups after the first run on side streams forked from the caller's stream, so that one
  // group's persistent launch fills the SMs that another's tail leaves idle
  std::vector<cudaStream_t> side;
  std::vector<cudaEvent_t> side_done;
  cudaEvent_t fork = nullptr;
  unsigned char* pinned = nullptr;  // one-shot plans: a pinned block (pinned_take)
  double2* h_out = nullptr;         // the outputs in it, written by the kernels
  int device = 0;  // the device the plan's memory and tables live on
  bool serial_groups = false;
  std::vector<wg::TreeLaunch> trees;
  std::vector<unsigned char> tree_prog;
  int ntrees = 0;          // instances
  int tree_parts = 0;  // most partials of a tree's output
  unsigned char* d_prog = nullptr;
  unsigned char* d_ws = nullptr;
  unsigned int polls = wg::TREE_POLLS;
  long long executions = 0;
  // a plan with trees answers the per-term queries (magnitudes, chunks, partials) by a plan over
  // the same device matrices that evaluates term by term, made when first asked and run once for every
  // execution that is asked about; one query at a time (terms_mu)
  std::vector<wg::Prepared> prep;
  wg_plan_options opt{};
  std::unique_ptr<std::mutex> terms_mu{new std::mutex};
  mutable wg_plan* terms = nullptr;
  mutable long long terms_of = -1;  // the execution that `terms` has run for
};

struct wg_state {
  int M = 0;
  wg::c64* d_B = nullptr;
  wg::c64* d_gamma = nullptr;
  std::vector<wg::c64> gamma;  // host copies: self-loop weights of unpaired modes, requests' forms
  std::vector<wg::c64> B;
  std::vector<wg::PartSums> parts;
  double alpha = 1.0;          // double-float prescale (power of two, from ||B||_inf)
  wg::MatrixForm form;         // of B
};

namespace wg {



static inline void put_scalar(unsigned char* dst, int st, double re, double im) {
  if (stype_mod(st)) {  // integer below 2^31 in magnitude (checked in prepare), Montgomery form
    const long long p = (long long)MOD_PRIMES[st - ST_MOD0];
    long long r = (long long)re % p;
    const uint64_t x = (uint64_t)(r < 0 ? r + p : r);
    const uint32_t v = (uint32_t)((x << 32) % (uint64_t)p);
    memcpy(dst, &v, 4);
    return;
  }
  switch (st) {
    case ST_REAL64: memcpy(dst, &re, 8); break;
    case ST_CPLX64: memcpy(dst, &re, 8); memcpy(dst + 8, &im, 8); break;
    case ST_REALDF: {
      float h = (float)re, l = (float)(re - (double)h);
      memcpy(dst, &h, 4); memcpy(dst + 4, &l, 4);
      break;
    }
    case ST_REALDD: {  // the input double is the high part exactly
      const double z = 0.0;
      memcpy(dst, &re, 8); memcpy(dst + 8, &z, 8);
      break;
    }
    case ST_CPLXDD: {
      const double z = 0.0;
      memcpy(dst, &re, 8); memcpy(dst + 8, &z, 8); memcpy(dst + 16, &im, 8); memcpy(dst + 24, &z, 8);
      break;
    }
    default: {
      float h = (float)re, l = (float)(re - (double)h);
      float hi = (float)im, li = (float)(im - (double)hi);
      memcpy(dst, &h, 4); memcpy(dst + 4, &l, 4); memcpy(dst + 8, &hi, 4); memcpy(dst + 12, &li, 4);
      break;
    }
  }
}

static inline bool prec_mod(int precision) { return precision >= WG_PREC_MOD0 && precision <= WG_PREC_MOD4; }

// 2^-e as the output scale: the FP64 value, or (modular precisions) the residue of 2^-e mod p
static inline double pow2_scale(int e, int precision) {
  if (!prec_mod(precision)) return std::ldexp(1.0, -e);
  const uint64_t p = MOD_PRIMES[precision - WG_PREC_MOD0], half = (p + 1) / 2;
  uint64_t r = 1;
  for (int i = 0; i < e; ++i) r = r * half % p;
  return (double)r;
}

static inline void get_val(const void* p, int dtype, size_t idx, double& re, double& im) {
  const double* d = (const double*)p;
  if (dtype == WG_COMPLEX128) { re = d[2 * idx]; im = d[2 * idx + 1]; }
  else { re = d[idx]; im = 0.0; }
}

// Largest |A_ij - A_ji| against the largest |A_ij| for which a matrix counts as symmetric.  The tree
// works on the mean of the two triangles; the sieve's value differs from the given matrix's only
// in second order of the antisymmetric part (tr(N X (S X)^(j-1)) = 0 for antisymmetric N, symmetric
// S and X), so differences of rounding size (a product U D U^T formed by BLAS) are far below the
// term arithmetic's roundoff: (2^-48)^2 = 2^-96 in FP64 and double-float, (2^-52)^2 in double-double.
static inline double tree_asymmetry(int precision) {
  return prec_mod(precision) ? 0.0 : std::ldexp(1.0, precision == WG_PREC_DD ? -52 : -48);
}

// Whether the parts of a complex matrix's entries are of like size.  A product of three real ones
// rounds a part relative to the whole, so that an imaginary part 1e-8 of the real one keeps 8 digits
// fewer than by four.  Every matching takes an entry of every row, A_ij or with loops D_i and another
// row's: where sum min(|re|, |im|) >= sum max(|re|, |im|) / 8 over a row's A_ij and D_i D_j, the rounding of
// those entries alone moves either part of the sum relative to the whole, and three products lose nothing.
// At least half of the rows have to say so (random phases: ratios of 0.41, and all but a few rows of two or
// three entries do; rows of purely real and purely imaginary entries have 0).
// of an instance's rows: `diag` with the diagonal, which edges of one pair each do not read; `fixed` without
// a batch's own mode, on which output 0 does not depend
static bool mixed_rows(const wg_instance& in, bool loops, bool odd, bool diag, bool fixed) {
  if (in.dtype != WG_COMPLEX128) return false;
  auto batch = [&](int i) {  // the vertices of the batch's edge, and the one that its odd mode is matched to
    return fixed && (i == 0 || i == in.n / 2 || (in.kind == WG_KIND_BATCH_ODD && i == in.n / 2 + 1));
  };
  const c64 *A = (const c64*)in.A, *D = (const c64*)in.D, *V = (const c64*)in.oddV;
  const c64 o = {in.oddloop[0], in.oddloop[1]};
  const int n = in.n;
  int rows = 0, all = odd;
  PartSums last;  // the unpaired vertex's row
  for (int i = 0; i < n; ++i) {
    if (batch(i)) continue;
    ++all;
    PartSums s;
    for (int j = 0; j < n; ++j)
      if ((j != i || diag) && !batch(j)) {
        s.add(A[(size_t)i * n + j].re, A[(size_t)i * n + j].im);
        if (loops) s.add(D[i], D[j]);
      }
    if (odd) {
      s.add(V[i].re, V[i].im);
      s.add(D[i], o);
      last.add(V[i].re, V[i].im);
      last.add(D[i], o);
    }
    rows += s.mixed();
  }
  if (odd) rows += last.mixed();
  return 2 * rows >= all;
}

static MatrixForm matrix_form(const void* A, int dtype, size_t n, double tol) {
  MatrixForm f;
  const int nc = dtype == WG_COMPLEX128 ? 2 : 1;
  const double* M = (const double*)A;
  double big = 0, diff = 0;
  bool pos = false, neg = false, finite = true, zeros = false;
  std::vector<int> comp(n);
  for (size_t i = 0; i < n; ++i) comp[i] = (int)i;
  size_t parts = n;
  auto root = [&](int x) {
    while (comp[x] != x) x = comp[x] = comp[comp[x]];
    return x;
  };
  for (size_t i = 0; i < n; ++i)
    for (size_t j = 0; j <= i; ++j) {
      const double *x = M + (i * n + j) * nc, *y = M + (j * n + i) * nc;
      bool zero = true;
      for (int c = 0; c < nc; ++c) {
        finite = finite && std::isfinite(x[c]) && std::isfinite(y[c]);
        big = std::max(big, std::fabs(x[c]));
        diff = std::max(diff, std::fabs(x[c] - y[c]));
        zero = zero && x[c] == 0;
      }
      zeros = zeros || zero;
      if (i != j) {
        pos = pos || x[0] > 0;
        neg = neg || x[0] < 0;
        if (!zero && parts > 1 && comp[i] != comp[j]) {
          const int a = root((int)i), b = root((int)j);
          parts -= a != b;
          comp[a] = b;
        }
      }
    }
  if (!finite) return f;
  f.symmetric = diff <= tol * big;
  f.signs = pos && neg;
  f.blocks = parts > 1;
  f.full = !zeros;
  f.diff = diff;
  return f;
}

// Whether an instance keeps the per-term evaluation although it has a tree: where the sum cancels
// so far that per-term results in this precision are good to little more than 1e-9, the tree's
// (closer to the exact value by 10 to 1000 times) would move them by more than that, and results
// stay what they were.  Share of random inputs whose results differ by more than 1e-9 relative:
//   FP64: real matrices of both signs 0 to 0.7 % for n <= 32, 1.7 % at 36, 9 % at 40, 17 % at 44 (all
//   positive: none); complex ones none to n = 40 (largest 1.1e-10); loop hafnians 0.5 % (real,
//   n = 21 to 33), none (complex); Gaussian states and generic matrices with multiple edges none of
//   200 for K <= 14, 1 % at K = 18; uncoupled blocks (a state and its conjugate, whose pairing
//   couples what the matrix does not) 0.6 % at K = 12, 8 to 23 % at 16, 70 % at 20;
//   double-float (roundoff 2^5 larger): complex n = 34 none of 140 (largest 8.5e-10), n = 36 none of 40 (9.0e-10),
//   n = 38 one of 40, n = 40 15 %;
//   real of both signs none at n = 14, 3 % at 20, 18 % at 32.
static bool keeps_terms(int stype, int kind, int K, const MatrixForm& f) {
  const bool real = stype == ST_REAL64 || stype == ST_REALDF, loops = kind != KIND_PLAIN;
  if (stype == ST_REAL64 || stype == ST_CPLX64)
    return (f.blocks && K > 12) || (real && f.signs && K > (loops ? 18 : 17));
  if (stype == ST_REALDF || stype == ST_CPLXDF)
    return f.blocks || K > (real && !f.signs && !loops ? TREE_MAX_K : (loops ? 10 : (real ? 8 : 17)));
  return false;  // residues are exact, double-double results agree to the last bits
}

std::vector<double> Prepared::tscales() const {
  std::vector<double> s;
  for (double a : ascale) s.push_back(pow2_scale(tree_scale_exp(T), precision) * a);
  return s;
}

// takes the tree when the instance has one
static void take_tree(Prepared& P, int precision, const std::vector<double>& ascale, const MatrixForm& f) {
  P.mixed = f.mixed;
  P.tree = f.symmetric && tree_build(P.d, P.T) && tree_fits(P.T, tree_bytes(P.ttype())) &&
           (P.forced || !keeps_terms(P.stype, P.d.kind, P.T.K, f));
  if (!P.tree) return;
  P.T.comp_off = stype_dd(P.stype) ? P.d.nout : 0;
  P.T.pstride = (stype_dd(P.stype) ? 2 : 1) * P.d.nout;
  P.ascale = ascale;
  P.precision = precision;
}

static int prepare(const wg_instance& in, int precision, Prepared& P) {
  const bool terms_only = (precision & WG_PREC_TERMS) != 0;
  P.forced = (precision & WG_PREC_TREE) != 0;
  precision &= ~kEvaluations;
  memset(&P.d, 0, sizeof(P.d));
  InstDev& d = P.d;
  if (in.dtype != WG_FLOAT64 && in.dtype != WG_COMPLEX128) return fail(WG_EINVAL, "dtype must be WG_FLOAT64 or WG_COMPLEX128");
  if (in.n < 0 || in.E < 0) return fail(WG_EINVAL, "negative size");
  if (in.n > 0 && !in.A) return fail(WG_EINVAL, "A is NULL");
  std::vector<int> reps;
  int kind = in.kind;
  int nb = 0, ne = 0;
  if (kind == WG_KIND_PLAIN || kind == WG_KIND_LOOP) {
    if (in.n != 2 * in.E) return fail(WG_EINVAL, "prepared matrix must be 2E x 2E (n=%d, E=%d)", in.n, in.E);
    for (int i = 0; i < in.E; ++i) reps.push_back((int)in.edge_reps[i]);
    if (kind == WG_KIND_LOOP) {
      nb = 1;
      if (!in.D) return fail(WG_EINVAL, "D is NULL");
      if (in.has_odd) {
        ne = 1;
        if (!in.oddV) return fail(WG_EINVAL, "oddV is NULL");
        kind = KIND_LOOP_ODD;
      }
    }
  } else if (kind == WG_KIND_BATCH_EVEN || kind == WG_KIND_BATCH_ODD) {
    const bool odd = kind == WG_KIND_BATCH_ODD;
    const int nbe = odd ? 2 : 1;
    if (in.n != 2 * (in.E + nbe)) return fail(WG_EINVAL, "batch matrix must be 2(E+%d) square", nbe);
    if (!in.D) return fail(WG_EINVAL, "D is NULL");
    if (in.batch_max < 0 || in.cutoff < 0 || in.cutoff > 1) return fail(WG_EINVAL, "bad batch_max / cutoff");
    reps.push_back(in.batch_max);
    if (odd) reps.push_back(1);
    for (int i = 0; i < in.E; ++i) reps.push_back((int)in.edge_reps[i]);
    nb = 1;
    ne = odd ? 2 : 1;
  } else {
    return fail(WG_EINVAL, "unknown kind %d", in.kind);
  }
  const int E = (int)reps.size();
  if (E > MAX_EDGES) return fail(WG_EINVAL, "at most %d edges per sieve (got %d)", MAX_EDGES, E);
  long long sumr = 0;
  int maxr = 0;
  for (int r : reps) {
    if (r < 0) return fail(WG_EINVAL, "negative edge repetition");
    if (r > BINOM_N - 1) return fail(WG_EINVAL, "edge repetition %d above the supported %d", r, BINOM_N - 1);
    sumr += r;
    maxr = std::max(maxr, r);
  }
  d.kind = kind;
  d.n = in.n;
  d.E = E;
  d.glynn = in.glynn ? 1 : 0;
  d.nb = nb;
  d.ne = ne;
  d.lda = in.n + 1;
  d.unit_binoms = maxr <= 1;
  int nout = 1;
  double alpha = 1.0;  // input prescale (double-float only): A -> alpha A, D -> sqrt(alpha) D
  if (precision == WG_PREC_DF) {
    double rs = 0;
    for (int i = 0; i < in.n; ++i) {
      double s = 0, re, im;
      for (int j = 0; j < in.n; ++j) { get_val(in.A, in.dtype, (size_t)i * in.n + j, re, im); s += std::hypot(re, im); }
      rs = std::max(rs, s);
    }
    if (rs > 0 && std::isfinite(rs)) alpha = std::exp2(-std::round(std::log2(rs)));
  }
  const double salpha = std::sqrt(alpha);
  std::vector<double> ascale;
  int Nf = 0;
  if (kind == KIND_PLAIN || kind == KIND_LOOP) {
    d.N = (int)(2 * sumr);
    d.K = d.N / 2;
    d.Nodd = 0;
    d.half_first = d.glynn;
    const int e = d.glynn ? d.N / 2 - 1 : 0;
    ascale.push_back(std::pow(alpha, -0.5 * d.N));
    P.scales.push_back(pow2_scale(e, precision) * ascale.back());
  } else if (kind == KIND_LOOP_ODD) {
    d.N = (int)(2 * sumr + 1);
    d.K = d.N / 2;
    d.Nodd = d.N;
    d.half_first = 0;
    const int e = d.glynn ? d.N / 2 : 0;
    ascale.push_back(std::pow(alpha, -0.5 * d.N));
    P.scales.push_back(pow2_scale(e, precision) * ascale.back());
    d.oddloop = {in.oddloop[0] * salpha, in.oddloop[1] * salpha};
  } else {
    const bool odd = kind == KIND_BATCH_ODD;
    long long sf = 0;
    for (int i = 0; i < in.E; ++i) sf += in.edge_reps[i];
    Nf = (int)(2 * sf + (odd ? 1 : 0));
    const int Nmax = odd ? Nf + 2 * in.batch_max + in.cutoff + 1 : Nf + 2 * in.batch_max + in.cutoff;
    nout = odd ? 2 * in.batch_max + in.cutoff + 2 : 2 * in.batch_max + in.cutoff + 1;
    if (nout > 32) return fail(WG_EINVAL, "batch output length %d above 32", nout);
    d.N = Nf;
    d.K = Nmax / 2;
    d.Nodd = Nmax;
    d.batch_max = in.batch_max;
    d.half_first = 0;
    double re, im;
    get_val(in.D, in.dtype, 0, re, im);
    d.oddloop = {re * salpha, im * salpha};
    if (odd) {
      get_val(in.D, in.dtype, 1, re, im);
      d.oddloop0 = {re * salpha, im * salpha};
    }
    for (int o = 0; o < nout; ++o) {
      const int x = Nf + o;
      ascale.push_back(std::pow(alpha, -0.5 * x));
      P.scales.push_back(pow2_scale(d.glynn ? x / 2 : 0, precision) * ascale.back());
    }
  }
  d.nout = nout;
  long long steps = 1;
  for (int i = 0; i < E; ++i) {
    const int R = (i == 0 && d.half_first) ? (reps[0] + 2) / 2 : reps[i] + 1;
    d.radix[i] = R;
    d.reps[i] = reps[i];
    if (steps > (1LL << 62) / R) return fail(WG_EINVAL, "too many sieve terms");
    steps *= R;
  }
  d.steps = steps;
  if (in.term_begin == 0 && in.term_end == 0) {
    P.t_lo = 0;
    P.t_hi = steps;
  } else {
    if (in.term_begin < 0 || in.term_end < in.term_begin || in.term_end > steps)
      return fail(WG_EINVAL, "term range [%lld, %lld) outside the %lld sieve terms", (long long)in.term_begin,
                  (long long)in.term_end, steps);
    P.t_lo = in.term_begin;
    P.t_hi = in.term_end;
  }
  // term matrix size bounds
  const int m_max = 2 * (int)std::count_if(reps.begin(), reps.end(), [](int r) { return r > 0; });
  P.m_max = m_max;
  P.mb_max = m_max + nb;
  P.rows_max = m_max + nb + ne;
  P.kc_max = std::min(d.K, m_max);
  // plain kinds keep det coefficients and the series (K + 1 each); loop kinds also the odd
  // series (Nodd, Nf) and the border series and their weights (K + 1 each)
  P.nser_need = kind == KIND_PLAIN ? d.K + 2 : std::max(std::max(d.K, d.Nodd), Nf) + 2;
  P.narr = (kind == KIND_PLAIN) ? 2 : 8;
  {
    // a term with m < K+1 and no border/extra rows has columns shorter than Kc+1: only when
    // some delta can vanish (an even repetition, or inclusion/exclusion)
    bool all_odd = d.glynn != 0;
    for (int r : reps) all_odd = all_odd && (r % 2 == 1);
    P.tile_ok = (nb + ne >= 1) || (all_odd && d.K < m_max);
  }
  P.term_cost = (double)P.mb_max * P.mb_max * P.mb_max + 64.0;
  if (P.rows_max > 80) return fail(WG_EINVAL, "term matrix of %d rows above the supported 80", P.rows_max);
  if (P.kc_max > 64) return fail(WG_EINVAL, "more than 64 characteristic coefficients");
  if (d.Nodd > 250 || d.K > 250) return fail(WG_EINVAL, "photon number above the supported 250");
  const bool cplx = in.dtype == WG_COMPLEX128;
  if (prec_mod(precision)) {
    // exact sieve: integer-valued real inputs below 2^31, binomial products exact in FP64 slots
    if (cplx) return fail(WG_EINVAL, "exact precision needs float64 (real) inputs");
    auto integral = [](double v) { return std::isfinite(v) && v == std::floor(v) && std::fabs(v) < 2147483648.0; };
    for (size_t i = 0; i < (size_t)in.n * in.n; ++i)
      if (!integral(((const double*)in.A)[i])) return fail(WG_EINVAL, "exact precision needs integer matrix entries below 2^31");
    if (in.D)
      for (int i = 0; i < in.n; ++i)
        if (!integral(((const double*)in.D)[i])) return fail(WG_EINVAL, "exact precision needs integer loop weights below 2^31");
    if (in.oddV)
      for (int i = 0; i < in.n; ++i)
        if (!integral(((const double*)in.oddV)[i])) return fail(WG_EINVAL, "exact precision needs integer entries below 2^31");
    if (kind == KIND_LOOP_ODD && !integral(in.oddloop[0])) return fail(WG_EINVAL, "exact precision needs an integer self-loop weight");
    if (maxr > 50) return fail(WG_EINVAL, "exact precision supports edge repetitions up to 50");
    P.stype = ST_MOD0 + (precision - WG_PREC_MOD0);
    d.modp = MOD_PRIMES[precision - WG_PREC_MOD0];
  } else {
    P.stype = precision == WG_PREC_DF   ? (cplx ? ST_CPLXDF : ST_REALDF)
              : precision == WG_PREC_DD ? (cplx ? ST_CPLXDD : ST_REALDD)
                                        : (cplx ? ST_CPLX64 : ST_REAL64);
  }
  // extended matrix [[A, D], [D^T, 0], [oddV, 0], [oddV0, 0]]  ((n+3) x (n+1))
  const int n = in.n, lda = n + 1;
  const size_t sb = stype_bytes(P.stype);
  P.ext.assign((size_t)(n + 3) * lda * sb, 0);
  P.ext_bytes = P.ext.size();
  auto at = [&](int r, int c) { return P.ext.data() + ((size_t)r * lda + c) * sb; };
  double re, im;
  for (int r = 0; r < n; ++r)
    for (int c = 0; c < n; ++c) {
      get_val(in.A, in.dtype, (size_t)r * n + c, re, im);
      put_scalar(at(r, c), P.stype, re * alpha, im * alpha);
    }
  if (nb) {
    for (int i = 0; i < n; ++i) {
      get_val(in.D, in.dtype, i, re, im);
      put_scalar(at(i, n), P.stype, re * salpha, im * salpha);
      put_scalar(at(n, i), P.stype, re * salpha, im * salpha);
    }
  }
  if (kind == KIND_LOOP_ODD) {
    for (int i = 0; i < n; ++i) {
      get_val(in.oddV, in.dtype, i, re, im);
      put_scalar(at(n + 1, i), P.stype, re * alpha, im * alpha);
    }
  }
  if (kind == KIND_BATCH_EVEN || kind == KIND_BATCH_ODD) {
    for (int i = 0; i < n; ++i) {  // oddV = A[0, :]
      get_val(in.A, in.dtype, (size_t)i, re, im);
      put_scalar(at(n + 1, i), P.stype, re * alpha, im * alpha);
    }
    if (kind == KIND_BATCH_ODD)
      for (int i = 0; i < n; ++i) {  // oddV0 = A[1, :]
        get_val(in.A, in.dtype, (size_t)n + i, re, im);
        put_scalar(at(n + 2, i), P.stype, re * alpha, im * alpha);
      }
  }
  if (!terms_only && in.term_begin == 0 && in.term_end == 0) {
    MatrixForm f = matrix_form(in.A, in.dtype, (size_t)n, tree_asymmetry(precision));
    const bool batch = kind >= KIND_BATCH_EVEN;
    f.mixed = mixed_rows(in, nb > 0, kind == KIND_LOOP_ODD, maxr > 1 || batch, false) &&
              (!batch || mixed_rows(in, true, false, true, true));
    take_tree(P, precision, ascale, f);
  }
  return WG_OK;
}


// Device-side formation of instance pools from a resident Gaussian state (serving).
struct GatherDev {
  long long a_off;  // pool byte offset of the instance's extended matrix
  int x_off;        // first index of the instance's pairing in the index array
  int n;            // 2E
  int oddmode;      // -1: none
  int stype;
  double alpha, salpha;
};
struct GatherSpec {
  const c64* B = nullptr;
  const c64* gamma = nullptr;
  int M = 0;
  std::vector<GatherDev> desc;
  std::vector<int> idx;
};

static int finalize_plan(std::vector<Prepared>& P, int precision, const wg_plan_options& opt, wg_plan* pl,
                         GatherSpec* gs, unsigned char* ext_pool);

// One block per instance: writes [[B[x][:,x], gamma[x]], [gamma[x]^T, 0], [B[o, x], 0], [0]]
// (alpha / sqrt(alpha) prescaled) into the instance's pool slot in its scalar type.
static __global__ void gather_kernel(const GatherDev* __restrict__ gd, const int* __restrict__ idx,
                                     const c64* __restrict__ B, const c64* __restrict__ gamma, int M,
                                     unsigned char* __restrict__ pool) {
  const GatherDev G = gd[blockIdx.x];
  const int n = G.n, lda = n + 1;
  const int* x = idx + G.x_off;
  const int total = (n + 3) * lda;
  for (int e = threadIdx.x; e < total; e += blockDim.x) {
    const int i = e / lda, j = e % lda;
    c64 v = {0.0, 0.0};
    double sc = 0.0;
    if (i < n && j < n) { v = B[(size_t)x[i] * M + x[j]]; sc = G.alpha; }
    else if (i < n && j == n) { v = gamma[x[i]]; sc = G.salpha; }
    else if (i == n && j < n) { v = gamma[x[j]]; sc = G.salpha; }
    else if (i == n + 1 && j < n && G.oddmode >= 0) { v = B[(size_t)G.oddmode * M + x[j]]; sc = G.alpha; }
    const double re = v.re * sc, im = v.im * sc;
    unsigned char* dst = pool + G.a_off;
    if (G.stype == ST_CPLX64) {
      reinterpret_cast<c64*>(dst)[e] = {re, im};
    } else {
      const float hr = __double2float_rn(re), hi = __double2float_rn(im);
      reinterpret_cast<cdf*>(dst)[e] = {{hr, __double2float_rn(re - (double)hr)}, {hi, __double2float_rn(im - (double)hi)}};
    }
  }
}

// What mixed_rows adds up, of every entry of the state's matrix
static void state_parts(wg_state& st) {
  const int M = st.M;
  st.parts.assign((size_t)M * M, PartSums());
  for (int i = 0; i < M; ++i)
    for (int j = 0; j < M; ++j) {
      PartSums& s = st.parts[(size_t)i * M + j];
      s.add(st.B[(size_t)i * M + j].re, st.B[(size_t)i * M + j].im);
      s.add(st.gamma[i], st.gamma[j]);
    }
}
// mixed_rows of a request's matrix, the unpaired mode a row like the others: a ns an entry, and half of
// the rows are enough
static bool request_mixed(const wg_request& r, const wg_state& st, bool diag) {
  int modes[2 * MAX_EDGES + 1], n = 2 * r.E, rows = 0;
  std::copy(r.x, r.x + n, modes);
  if (r.oddmode >= 0) modes[n++] = r.oddmode;
  for (int i = 0; i < n && 2 * rows < n; ++i) {
    const PartSums* row = &st.parts[(size_t)modes[i] * st.M];
    PartSums s;
    for (int j = 0; j < n; ++j)
      if (j != i || diag) {
        s.low += row[modes[j]].low;
        s.high += row[modes[j]].high;
      }
    rows += s.mixed();
  }
  return 2 * rows >= n;
}

// matrix_form of a request's matrix, so that it takes the route that it takes alone.  In a state without
// zero entries there are no blocks, and one entry large against what the triangles differ by says that
// they agree: 0.1 us, and 2 to 3 us for 28 photons otherwise.
static MatrixForm request_form(const wg_request& r, const wg_state& st) {
  const double tol = tree_asymmetry(WG_PREC_FP64);
  const int n = 2 * r.E;
  MatrixForm f;
  const c64 any = st.B[(size_t)r.x[0] * st.M + r.x[n - 1]];
  if (st.form.full && st.form.diff <= tol * std::max(std::fabs(any.re), std::fabs(any.im))) {
    f.symmetric = true;
    return f;
  }
  std::vector<c64> A((size_t)n * n);
  for (int i = 0; i < n; ++i)
    for (int j = 0; j < n; ++j) A[(size_t)i * n + j] = st.B[(size_t)r.x[i] * st.M + r.x[j]];
  return matrix_form(A.data(), WG_COMPLEX128, n, tol);
}

// Loop-hafnian instance of one serving request (the host part of prepare() for WG_KIND_LOOP,
// without a host copy of the matrix).
static int prepare_request(const wg_request& r, const wg_state& st, int precision, Prepared& P, GatherDev& g,
                           std::vector<int>& idx) {
  const bool terms_only = (precision & WG_PREC_TERMS) != 0;
  P.forced = (precision & WG_PREC_TREE) != 0;
  precision &= ~kEvaluations;
  memset(&P.d, 0, sizeof(P.d));
  InstDev& d = P.d;
  if (r.E < 1 || r.E > MAX_EDGES || !r.x || !r.edge_reps) return fail(WG_EINVAL, "request needs 1..32 edges");
  const bool odd = r.oddmode >= 0;
  if (r.oddmode >= st.M) return fail(WG_EINVAL, "unpaired mode out of range");
  long long sumr = 0, steps = 1;
  int maxr = 0;
  for (int i = 0; i < r.E; ++i) {
    const long long rr = r.edge_reps[i];
    if (rr < 0 || rr > BINOM_N - 1) return fail(WG_EINVAL, "edge repetition out of range");
    sumr += rr;
    maxr = std::max(maxr, (int)rr);
  }
  for (int i = 0; i < 2 * r.E; ++i)
    if (r.x[i] < 0 || r.x[i] >= st.M) return fail(WG_EINVAL, "mode index out of range");
  const double alpha = precision == WG_PREC_DF ? st.alpha : 1.0, salpha = std::sqrt(alpha);
  d.kind = odd ? KIND_LOOP_ODD : KIND_LOOP;
  d.n = 2 * r.E;
  d.E = r.E;
  d.glynn = 1;
  d.nb = 1;
  d.ne = odd ? 1 : 0;
  d.lda = d.n + 1;
  d.unit_binoms = maxr <= 1;
  d.N = (int)(2 * sumr + (odd ? 1 : 0));
  d.K = d.N / 2;
  d.Nodd = odd ? d.N : 0;
  d.nout = 1;
  d.half_first = odd ? 0 : 1;
  if (odd) d.oddloop = {st.gamma[r.oddmode].re * salpha, st.gamma[r.oddmode].im * salpha};
  const int e = odd ? d.N / 2 : d.N / 2 - 1;
  const double ascale = std::pow(alpha, -0.5 * d.N);
  P.scales.assign(1, std::ldexp(1.0, -e) * ascale);
  for (int i = 0; i < r.E; ++i) {
    const int R = (i == 0 && d.half_first) ? (int)(r.edge_reps[0] + 2) / 2 : (int)r.edge_reps[i] + 1;
    d.radix[i] = R;
    d.reps[i] = (int)r.edge_reps[i];
    if (steps > (1LL << 62) / R) return fail(WG_EINVAL, "too many sieve terms");
    steps *= R;
  }
  d.steps = steps;
  P.t_lo = 0;
  P.t_hi = steps;
  int nnz = 0;
  bool all_odd = true;
  for (int i = 0; i < r.E; ++i) {
    nnz += r.edge_reps[i] > 0;
    all_odd = all_odd && (r.edge_reps[i] % 2 == 1);
  }
  P.m_max = 2 * nnz;
  P.mb_max = P.m_max + 1;
  P.rows_max = P.m_max + 1 + d.ne;
  P.kc_max = std::min(d.K, P.m_max);
  P.nser_need = std::max(d.K, d.Nodd) + 2;
  P.narr = 8;
  P.tile_ok = true;  // bordered tile
  P.term_cost = (double)P.mb_max * P.mb_max * P.mb_max + 64.0;
  if (P.rows_max > 80 || d.K > 250 || d.Nodd > 250) return fail(WG_EINVAL, "request too large");
  P.stype = precision == WG_PREC_DF ? ST_CPLXDF : ST_CPLX64;
  P.ext.clear();
  P.ext_bytes = (size_t)(d.n + 3) * (d.n + 1) * stype_bytes(P.stype);
  g.x_off = (int)idx.size();
  g.n = d.n;
  g.oddmode = r.oddmode;
  g.stype = P.stype;
  g.alpha = alpha;
  g.salpha = salpha;
  for (int i = 0; i < 2 * r.E; ++i) idx.push_back(r.x[i]);
  if (!terms_only) {
    MatrixForm f = request_form(r, st);
    f.mixed = request_mixed(r, st, maxr > 1);
    take_tree(P, precision, {ascale}, f);
  }
  return WG_OK;
}

static bool known_precision(int precision) {
  const int p = precision & ~kEvaluations;
  return p == WG_PREC_FP64 || p == WG_PREC_DF || p == WG_PREC_DD || prec_mod(p);
}
// the primes of WG_PREC_PRIMES(k) (0: another precision)
static int prec_primes(int precision) {
  const int k = (precision & ~kEvaluations) - WG_PREC_PRIMES(0);
  return k >= 1 && k <= MOD_N ? k : 0;
}

static int build_plan(const wg_instance* v, int count, int precision, const wg_plan_options& opt, wg_plan* pl) {
  if (count < 0 || (count > 0 && !v)) return fail(WG_EINVAL, "bad instance list");
  const int primes = prec_primes(precision);
  if (!known_precision(precision) && !primes) return fail(WG_EINVAL, "unknown precision %d", precision);
  pl->primes = std::max(primes, 1);
  std::vector<Prepared> P((size_t)count * pl->primes);
  for (int i = 0; i < count * pl->primes; ++i) {
    const int prec = primes ? (WG_PREC_MOD0 + i / count) | (precision & kEvaluations) : precision;
    int rc = prepare(v[i % count], prec, P[i]);
    if (rc) return fail(rc, "instance %d: %s", i % count, g_err.c_str());
  }
  if (primes) precision = WG_PREC_MOD0;
  return finalize_plan(P, precision, opt, pl, nullptr, nullptr);
}

// Per node type: SM clocks per multiply-add of a tree, measured over launches that fill the chip (four
// products instead of three: in proportion)
static double tree_mac_clocks(int ttype) {
  const int stype = tree_stype(ttype);
  if (ttype != stype) return 4.0 / 3.0 * tree_mac_clocks(stype);
  switch (stype) {
    case ST_REAL64: return 0.5;
    case ST_CPLX64: return 2.0;
    case ST_REALDF: return 0.2;
    case ST_CPLXDF: return 0.6;
    case ST_REALDD: return 9.0;
    case ST_CPLXDD: return 35.0;
    default: return 0.15;
  }
}

// and of one edge of a term's latency (tree_latency's unit)
static double tree_edge_clocks(int stype) {
  return stype == ST_CPLXDD ? 80000 : stype == ST_REALDD ? 32000 : 16000;
}

// The levels of a plan's trees, each within what `limit` bytes leave beside the trees' programs (about
// as many rounds and segments as phases); those that do not fit are summed by terms.  `limit` becomes
// what is left for the levels of a launch.
static std::vector<TreeLevels> place_trees(std::vector<Prepared>& P, double& limit) {
  std::vector<TreeLevels> lev(P.size());
  double programs = 0;
  for (size_t i = 0; i < P.size(); ++i) {
    if (!P[i].tree) continue;
    P[i].tree = tree_levels_within(P[i].T, tree_bytes(P[i].ttype()), limit, lev[i]);
    if (P[i].tree) programs += sizeof(TreeInst) + 512 + lev[i].phases * (sizeof(TreeRound) + sizeof(TreeSeg));
  }
  const double left = limit - programs;
  for (size_t i = 0; i < P.size(); ++i)
    if (P[i].tree && (double)lev[i].bytes > left)
      P[i].tree = tree_levels_within(P[i].T, tree_bytes(P[i].ttype()), left, lev[i]);
  limit = left;
  return lev;
}

// Groups the tree members of a plan into launches (one node type each, as many instances as share
// a workspace budget), makes their programs and lays out their partial slots.  Returns the
// workspace bytes; the launches run one after another and share it, or (an exact sum's primes) side
// by side.
static long long plan_trees(std::vector<Prepared>& P, const std::vector<TreeLevels>& lev, double limit, wg_plan* pl,
                            int& nparts) {
  // A launch's levels: beyond this the instances go to the next launch, which uses the same workspace.
  // (One instance alone may take more, up to place_trees' limit: complex FP64 1.3 GB at n = 40, 1.9 at 44,
  // 4.2 at 64.)
  const double kLaunchBytes = std::min(600e6, limit);
  const int count = (int)P.size();
  auto al = [](long long x) { return (x + 255) & ~255ll; };
  std::vector<int> order;
  for (int i = 0; i < count; ++i)
    if (P[i].tree) order.push_back(i);
  pl->ntrees = (int)order.size();
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) {
    return P[a].ttype() != P[b].ttype() ? P[a].ttype() < P[b].ttype() : lev[a].bytes > lev[b].bytes;
  });
  // Several primes side by side when their levels, of which two at a time are in use, keep to the L2:
  // graph counts modulo three, n = 36 (75 MB each) 886 us one after another and 723 side by side,
  // n = 38 (160 MB each) 1,508 and 1,642.
  constexpr double kSideBytes = 250e6;
  long long first = 0;
  for (size_t k = 0; k < order.size() && P[order[k]].ttype() == P[order[0]].ttype(); ++k) first += lev[order[k]].bytes;
  pl->side_trees = pl->primes > 1 && !order.empty() && (double)first * pl->primes <= std::min(kSideBytes, limit);
  // The launches of several scalar types side by side, each with SMs by its work and at least 30 % of an
  // even share: one's narrow rounds and barriers no longer wait for the other's.  us in turn and so, plans of
  // complex and real matrices: 8 of n = 8 to 12 72 and 55, 64 to n = 18 112 and 77, 160 to n = 28 833 and
  // 769 (even shares: 985), 40 to n = 32 853 and 746.  Not beyond a launch's workspace, where they evict one
  // another's levels from the L2 (250 to n = 30: 1,778 and 1,954).
  std::map<int, double> works;  // SM clocks of a node type
  double total = 0, work = 0;
  for (int i : order) {
    const double w = tree_work(P[i].T) * tree_mac_clocks(P[i].ttype());
    works[P[i].ttype()] += w;
    work += w;
    total += lev[i].bytes;
  }
  pl->fork_trees = !pl->side_trees && !pl->serial_groups && works.size() > 1 && total <= kLaunchBytes;
  const double least = 0.3 / works.size();
  long long ws = 0;
  for (size_t k = 0; k < order.size();) {
    TreeLaunch G;
    memset(&G, 0, sizeof(G));
    G.ttype = P[order[k]].ttype();
    const int sb = tree_bytes(G.ttype);
    const int tile = stype_mod(G.ttype) ? tree_tile<modp<MOD_PRIMES[0]>>()
                                        : (tree_stype(G.ttype) == ST_CPLXDD ? tree_tile<cdd>() : tree_tile<c64>());
    std::vector<TreeInst> insts;
    std::vector<TreeLevels> levels;
    const size_t k0 = k;
    long long bytes = 0;
    for (; k < order.size() && P[order[k]].ttype() == G.ttype; ++k) {
      if (k > k0 && (double)(bytes + lev[order[k]].bytes) > kLaunchBytes) break;
      bytes += lev[order[k]].bytes;
      insts.push_back(P[order[k]].T);
      insts.back().a_off = P[order[k]].d.a_off;
      levels.push_back(lev[order[k]]);
    }
    TreeProgram prog;
    std::vector<int> base, cnt;
    const double clk = tree_mac_clocks(G.ttype);
    const double share = pl->side_trees ? 1.0 / pl->primes
                         : pl->fork_trees ? least + (1 - least * works.size()) * works[G.ttype] / work : 1.0;
    const int sms = std::max((int)(g_num_sms * share), 1);
    G.ctas = tree_one_cta(insts, levels, clk, sms) ? 1 : sms;
    tree_program(insts, levels, sb, tile, G.ctas * TREE_THREADS, nparts, base, cnt, prog);
    for (size_t j = 0; j < insts.size(); ++j) {
      InstDev& d = P[order[k0 + j]].d;
      d.part_base = base[j];
      d.nchunks = cnt[j];
      d.pstride = insts[j].pstride;
      d.comp_off = insts[j].comp_off;
      d.mag_off = 0;
      pl->tree_parts = std::max(pl->tree_parts, cnt[j]);
    }
    G.ninst = (int)prog.insts.size();
    G.nrounds = (int)prog.rounds.size();
    G.nsegs = (int)prog.segs.size();
    const size_t b_inst = sizeof(TreeInst) * prog.insts.size(), b_rounds = sizeof(TreeRound) * prog.rounds.size(),
                 b_segs = sizeof(TreeSeg) * prog.segs.size();
    G.prog_off = pl->tree_prog.size();
    pl->tree_prog.resize(G.prog_off + al((long long)(b_inst + b_rounds + b_segs)));
    memcpy(pl->tree_prog.data() + G.prog_off, prog.insts.data(), b_inst);
    memcpy(pl->tree_prog.data() + G.prog_off + b_inst, prog.rounds.data(), b_rounds);
    memcpy(pl->tree_prog.data() + G.prog_off + b_inst + b_rounds, prog.segs.data(), b_segs);
    G.sm_warp = prog.smem;
    G.sm_cache = (int)al((long long)prog.smem * (TREE_THREADS / 32) * sb);
    G.smem = G.sm_cache;
    G.cached = G.smem + al((long long)(b_inst + b_rounds + b_segs)) <= TREE_SMEM_BYTES;
    if (G.cached) G.smem += (int)al((long long)(b_inst + b_rounds + b_segs));
    if (G.ctas == 1 && G.smem + prog.ws_bytes <= TREE_SMEM_BYTES) {
      G.sm_ws = G.smem;
      G.smem += (int)prog.ws_bytes;
    } else {
      G.ws_off = pl->side_trees || pl->fork_trees ? ws : 0;
      ws = std::max(ws, G.ws_off + al(prog.ws_bytes));
    }
    pl->trees.push_back(G);
  }
  return ws;
}

// whether the plan is one tree launch, which then also reduces (tree_finish): an output a warp of the
// last CTA (64 photon patterns, whose partials one CTA sums in 150 us: 631 -> 518 us by a launch of
// its own; one hafnian's launch 4 us)
static bool plan_single(const wg_plan* pl) {
  return pl->groups.empty() && (pl->trees.size() == 1 || pl->side_trees) && pl->total_out <= TREE_THREADS / 32 * pl->primes;
}
static int plan_counters(const wg_plan* pl) {
  return (int)(pl->groups.size() + 2 * pl->trees.size());  // a tree launch's barrier and its tree_finish
}
// warps that sum an output's partials, of the `nw` of a block: one, as the per-term launches
// always had, unless a tree left several hundred
static int plan_wpo(const wg_plan* pl, int nw) {
  int w = 1;
  while (w < nw && w * 64 < pl->tree_parts && w * (pl->total_out / pl->primes) < nw) w *= 2;
  return w;
}

// Few photon pairs: a multiple edge as simple ones costs more nodes but fewer and shorter rounds, where
// those are the time.  us before and after (FP64): loops [1, 1, 1, 2, 2, 2] 93 and 80, [1 x 8, 2, 2] 132
// and 115, batches [1, 2, 2, 3] 167 and 133; over 1064 calls of 1 to 12 edges 14 % less.  Not in a batch of
// at most five pairs in simple and double edges, whose leaves, a warp a node, are the time (batch [1, 2, 2]
// 92 us, split 104).
static void split_edges(std::vector<Prepared>& P) {
  constexpr int kSplitPairs = 16;
  auto splits = [](const Prepared& p) {
    const TreeInst& T = p.T;
    if (!p.tree || T.K == T.E || T.K > kSplitPairs) return false;
    return T.pB < 0 || T.K > 5 || *std::max_element(T.reps, T.reps + T.E) > 2;
  };
  if (std::none_of(P.begin(), P.end(), splits)) return;
  std::vector<TreeInst> alt(P.size());
  double lat = 0, lat1 = 0, work = 0, work1 = 0;
  for (size_t i = 0; i < P.size(); ++i) {
    if (!P[i].tree) continue;
    const TreeInst& T = P[i].T;
    const double clk = tree_mac_clocks(P[i].ttype()) / g_num_sms;
    const bool split = splits(P[i]) && tree_build(P[i].d, alt[i], true);
    const double unit = tree_edge_clocks(P[i].stype), w = tree_work(T) * clk;
    lat = std::max(lat, unit * tree_latency(T));
    lat1 = std::max(lat1, unit * tree_latency(split ? alt[i] : T));
    work += w;
    work1 += split ? tree_work(alt[i]) * clk : w;
    if (!split) alt[i].E = 0;
  }
  if (lat1 + work1 >= lat + work) return;
  for (size_t i = 0; i < P.size(); ++i)
    if (P[i].tree && alt[i].E) {
      alt[i].comp_off = P[i].T.comp_off;
      alt[i].pstride = P[i].T.pstride;
      P[i].T = alt[i];
    }
}

// Whether the terms of a plan's trees are summed sooner one by one.  The terms run side by side, so
// that their latency grows with the edges alone, and a tree's with its rounds: 0.7 of a term's edge for
// a simple one, 2 for a double edge, 4 for one of three photons or more (its root and exponential
// recurrences are chains of FP64 latencies).  What more terms than fit side by side cost grows with
// their number, a tree's time hardly.  One unit is 6.5 to 12.5 us (FP64 plain to batches; double-double
// 17 to 108); the weights are fitted to 2261 measured calls of 1 to 12 edges, multiplicities 1 to 12,
// 1 to 10^4 terms, all scalar types.  us by tree and by terms (complex FP64, plain): [1 x 8] 57 and 97,
// [3, 3, 3, 3] 136 and 76, [8, 8] 89 and 54, [1 x 6, 2, 2, 3] 118 and 203; of 1064 calls it takes the
// tree in 7 where that is slower by more than 10 % (double-double [1, 2, 2, 3, 3, 3] 645 and 390 us the worst).
static bool terms_sooner(const std::vector<Prepared>& P) {
  double tree = 0, terms = 0, work = 0;
  for (const Prepared& p : P) {
    if (!p.tree) continue;
    if (!tile_rows_ok(p.stype, p.rows_max)) return false;
    int E = 0, big = 0;
    double t = 0.5;
    for (int e = p.d.kind == KIND_BATCH_EVEN ? 1 : (p.d.kind == KIND_BATCH_ODD ? 2 : 0); e < p.d.E; ++e) {
      E += p.d.reps[e] > 0;
      big += p.d.reps[e] > 2;
      t *= p.d.reps[e] + 1;
    }
    const bool dd = stype_dd(p.stype);
    // per-term work against a tree's: no less of it where all edges are multiple, a batch has its outputs'
    const double share = p.d.nout > 1 ? 1.2 * p.d.nout : (E - big) / (double)std::max(E, 1);
    tree = std::max(tree, tree_latency(p.T));
    terms = std::max(terms, (dd ? 0.9 : 2.0) + E);
    work += (dd ? 3.75e-5 : 1.5e-5) * share * t * ((double)E * E * E + (double)p.T.K * p.T.K);
  }
  return tree > terms + work;
}

// What a plan whose allocation failed asks for next
constexpr double kLeastWorkspace = 64e6;

// ext_pool: the instances' matrices are on the device already, at their a_off
static int finalize_plan(std::vector<Prepared>& P, int precision, const wg_plan_options& opt, wg_plan* pl,
                         GatherSpec* gs, unsigned char* ext_pool) {
  precision &= ~kEvaluations;
  const int count = (int)P.size();
  const double chunk_scale = opt.chunk_scale > 0 ? opt.chunk_scale : 1.0;
  const int wpc_cap = opt.max_warps_per_cta > 0 ? std::min(opt.max_warps_per_cta, 8) : kDefaultWarpsPerCta;
  pl->use_graph = opt.use_graph != 0;
  pl->serial_groups = opt.serial_groups != 0;
  pl->precision = precision;
  pl->device = g_device;
  if (P.empty() || !P[0].forced) {
    split_edges(P);
    if (terms_sooner(P))
      for (Prepared& p : P) p.tree = false;
  }
  const bool roomy = opt.max_workspace <= 0 || opt.max_workspace > kLeastWorkspace;
  double limit = opt.max_workspace > 0 ? (double)opt.max_workspace : 1e18;
  const std::vector<TreeLevels> lev = place_trees(P, limit);
  // outputs and scales in instance order
  int out = 0;
  std::vector<double> scales;
  for (int i = 0; i < count; ++i) {
    P[i].d.out_base = out;
    P[i].d.scale_base = (int)scales.size();
    out += P[i].d.nout;
    const std::vector<double> sc = P[i].tree ? P[i].tscales() : P[i].scales;
    scales.insert(scales.end(), sc.begin(), sc.end());
  }
  pl->total_out = out;
  // launch shape per (scalar class, per-warp workspace), see best_shape
  std::map<std::pair<int, int>, std::pair<int, int>> shape_memo;
  auto shape = [&](int st, int bytes) -> std::pair<int, int> {
    const auto key = std::make_pair(st, bytes);
    const auto it = shape_memo.find(key);
    if (it != shape_memo.end()) return it->second;
    return shape_memo[key] = best_shape(st, bytes, wpc_cap);
  };
  // groups by (stype, resident warps per SM of the instance's own workspace), so that a small
  // instance does not run at the occupancy of a larger one's workspace; with merge_classes one
  // group per scalar type
  struct GKey { int st, res; };
  std::vector<GKey> keys;
  std::vector<int> gid(count, -1);
  for (int i = 0; i < count; ++i) {
    if (P[i].tree) continue;
    if (!tile_rows_ok(P[i].stype, P[i].rows_max)) return fail(WG_EINVAL, "instance %d: term matrix too large", i);
    int res = 0;
    if (!opt.merge_classes) {
      const WarpLayout Li = make_layout(P[i].stype, std::max(P[i].rows_max, 1), std::max(P[i].mb_max, 1),
                                        P[i].kc_max, std::max(P[i].nser_need, 2), std::max(P[i].narr, 2),
                                        P[i].tile_ok);
      const auto sh = shape(P[i].stype, Li.bytes);
      res = sh.first * sh.second;
    }
    int g = -1;
    for (size_t k = 0; k < keys.size(); ++k)
      if (keys[k].st == P[i].stype && (opt.merge_classes || keys[k].res == res)) g = (int)k;
    if (g < 0) { keys.push_back({P[i].stype, res}); g = (int)keys.size() - 1; }
    gid[i] = g;
  }
  // pool
  size_t pool_bytes = 0;
  for (int i = 0; i < count && !ext_pool; ++i) {
    P[i].d.a_off = (long long)pool_bytes;
    pool_bytes += (P[i].ext_bytes + 255) & ~(size_t)255;
  }
  if (gs)
    for (int i = 0; i < count; ++i) gs->desc[i].a_off = P[i].d.a_off;
  int nparts = 0;
  const long long ws_bytes = plan_trees(P, lev, limit, pl, nparts);
  for (size_t g = 0; g < keys.size(); ++g) {
    Group G;
    G.stype = keys[g].st;
    int rows = 1, mb = 1, kc = 0, nser = 2, narr = 2;
    bool tile = true;
    double total_cost = 0;
    std::vector<int> members;
    for (int i = 0; i < count; ++i)
      if (gid[i] == (int)g) {
        members.push_back(i);
        rows = std::max(rows, P[i].rows_max);
        mb = std::max(mb, P[i].mb_max);
        kc = std::max(kc, P[i].kc_max);
        nser = std::max(nser, P[i].nser_need);
        narr = std::max(narr, P[i].narr);
        tile = tile && P[i].tile_ok;
        total_cost += P[i].term_cost * (double)(P[i].t_hi - P[i].t_lo);
      }
    G.L = make_layout(G.stype, rows, mb, kc, nser, narr, tile);
    const auto sh = shape(G.stype, G.L.bytes);
    const int wpc = sh.first, per_sm = sh.second;
    if (wpc < 1) return fail(WG_EINVAL, "per-warp workspace of %d bytes does not fit", G.L.bytes);
    if (per_sm < 1) {
      cudaGetLastError();
      return fail(WG_ECUDA, "sieve kernel cannot be resident (workspace %d B x %d warps)", G.L.bytes, wpc);
    }
    G.wpc = wpc;
    const long long resident = (long long)g_num_sms * per_sm * wpc;
    // chunking by guided self-scheduling, largest instances first: a chunk is 1/(2 chunk_scale) of
    // a resident warp's share of the group's remaining work, capped at ~1000 term-equivalents of a
    // 40-row tile and floored at ~4 (less for small groups).  Chunk sizes fall geometrically, so
    // the last chunks -- the ones that decide when the launch ends -- are short: n = 40 takes
    // 276 ms instead of 302 ms with fixed chunks of a quarter of a warp's share.
    constexpr double kMaxChunkCost = 6.4e7, kMinChunkCost = 2.6e5;
    const double div = 2.0 * chunk_scale * (double)resident;
    const double min_cost = std::min(kMinChunkCost, total_cost / (4.0 * div));  // small groups: finer
    double remaining = total_cost;
    std::stable_sort(members.begin(), members.end(), [&](int a, int b) {
      return P[a].term_cost * (double)(P[a].t_hi - P[a].t_lo) > P[b].term_cost * (double)(P[b].t_hi - P[b].t_lo);
    });
    G.chunk_begin = (int)pl->chunks.size();
    for (int i : members) {
      InstDev& d = P[i].d;
      const double tc = P[i].term_cost;
      const long long hi = P[i].t_hi, pmin = std::max(1LL, (long long)std::ceil(min_cost / tc));
      d.part_base = nparts;
      // slots per chunk: sums; double-double kinds their compensations; floating-point kinds
      // the term magnitudes (the exact sieve's residues have none)
      const bool dd = stype_dd(P[i].stype), fl = !stype_mod(P[i].stype);
      d.comp_off = dd ? d.nout : 0;
      d.mag_off = fl ? (dd ? 2 : 1) * d.nout : 0;
      d.pstride = (1 + (dd ? 1 : 0) + (fl ? 1 : 0)) * d.nout;
      int nch = 0;
      for (long long t = P[i].t_lo; t < hi; ++nch) {
        const double want = std::min(remaining / div, kMaxChunkCost * chunk_scale);
        long long per = std::max(pmin, (long long)std::floor(want / tc));
        per = std::min(per, hi - t);
        ChunkDev ch;
        ch.inst = i;
        ch.part = nparts + nch * d.pstride;
        ch.t0 = t;
        ch.t1 = t + per;
        pl->chunks.push_back(ch);
        remaining -= (double)per * tc;
        t += per;
      }
      d.nchunks = nch;
      nparts += nch * d.pstride;
    }
    G.chunk_count = (int)pl->chunks.size() - G.chunk_begin;
    G.ctas = (int)std::min<long long>((long long)g_num_sms * per_sm, (G.chunk_count + wpc - 1) / wpc);
    G.ctas = std::max(G.ctas, 1);
    pl->groups.push_back(G);
  }
  pl->nparts = nparts;
  for (int i = 0; i < count; ++i) pl->inst.push_back(P[i].d);
  // one device allocation
  auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
  const size_t b_inst = al(sizeof(InstDev) * std::max(count, 1));
  const size_t b_chunks = al(sizeof(ChunkDev) * std::max<size_t>(pl->chunks.size(), 1));
  const size_t b_pool = al(std::max<size_t>(pool_bytes, 16));
  const size_t b_parts = al(sizeof(double2) * std::max(nparts, 1));
  const size_t b_scales = al(sizeof(double) * std::max<size_t>(scales.size(), 1));
  const size_t b_out = al(sizeof(double2) * std::max(out, 1));
  const size_t b_mag = al(sizeof(double) * std::max(out, 1));
  const size_t ncnt = (size_t)plan_counters(pl);
  int counter = (int)pl->groups.size();
  for (TreeLaunch& g : pl->trees) {
    g.counter = counter;
    counter += 2;
  }
  const size_t b_cnt = al(sizeof(unsigned int) * std::max<size_t>(ncnt, 1));
  const size_t b_tree = al(std::max<size_t>(pl->tree_prog.size(), 1));
  const size_t b_ws = al((size_t)ws_bytes);
  const size_t b_err = al(sizeof(int));
  const size_t b_gdesc = gs ? al(sizeof(GatherDev) * std::max<size_t>(gs->desc.size(), 1)) : 0;
  const size_t b_gidx = gs ? al(sizeof(int) * std::max<size_t>(gs->idx.size(), 1)) : 0;
  // what is uploaded (zeroed counters included) first, in one copy; the matrices last of it, since
  // serving forms them on the device
  const size_t o_tree = b_inst + b_chunks, o_scales = o_tree + b_tree, o_cnt = o_scales + b_scales;
  const size_t o_gdesc = o_cnt + b_cnt + b_err, o_pool = o_gdesc + b_gdesc + b_gidx;
  const size_t total = o_pool + b_pool + b_parts + b_out + b_mag + b_ws;
  cudaStream_t cs = (cudaStream_t)opt.stream;
  pl->alloc_stream = cs;
  pl->async_alloc = cs != nullptr;
  const cudaError_t ae = pl->async_alloc ? cudaMallocAsync(&pl->dmem, total, cs) : cudaMalloc(&pl->dmem, total);
  if (ae != cudaSuccess) {
    cudaGetLastError();
    if (!pl->trees.empty()) {  // with less workspace, then by terms
      wg_plan fresh;
      fresh.pinned = pl->pinned;
      fresh.primes = pl->primes;
      *pl = std::move(fresh);
      wg_plan_options less = opt;
      less.max_workspace = roomy ? (long long)kLeastWorkspace : 1;
      return finalize_plan(P, precision, less, pl, gs, ext_pool);
    }
    pl->dmem = nullptr;
    return fail(WG_ENOMEM, "device allocation of %zu bytes failed", total);
  }
  unsigned char* base = (unsigned char*)pl->dmem;
  pl->d_inst = (InstDev*)base; base += b_inst;
  pl->d_chunks = (ChunkDev*)base; base += b_chunks;
  pl->d_prog = base; base += b_tree;
  pl->d_scales = (double*)base; base += b_scales;
  pl->d_counters = (unsigned int*)base; base += b_cnt;
  pl->d_err = (int*)base; base += b_err;
  GatherDev* d_desc = (GatherDev*)base; base += b_gdesc;
  int* d_idx = (int*)base; base += b_gidx;
  pl->d_pool = ext_pool ? ext_pool : base; base += b_pool;
  pl->d_partials = (double2*)base; base += b_parts;
  pl->d_out = (double2*)base; base += b_out;
  pl->d_mag = (double*)base; base += b_mag;
  pl->d_ws = base;
  pl->device_bytes = (long long)total;
  // staging: one host buffer with the same layout for the upload, in the pinned block when it fits
  // there beside the outputs
  const size_t staged = o_pool + (gs || ext_pool ? 0 : b_pool);
  std::vector<unsigned char> pageable;
  unsigned char* host;
  if (pl->pinned && b_out + staged <= kPinnedBytes) {
    pl->h_out = (double2*)pl->pinned;
    pl->d_out = pl->h_out;
    host = pl->pinned + b_out;
    memset(host, 0, staged);
  } else {
    pageable.assign(staged, 0);
    host = pageable.data();
  }
  memcpy(host, pl->inst.data(), sizeof(InstDev) * count);
  if (!pl->chunks.empty()) memcpy(host + b_inst, pl->chunks.data(), sizeof(ChunkDev) * pl->chunks.size());
  if (!pl->tree_prog.empty()) memcpy(host + o_tree, pl->tree_prog.data(), pl->tree_prog.size());
  if (!scales.empty()) memcpy(host + o_scales, scales.data(), sizeof(double) * scales.size());
  if (gs) {
    memcpy(host + o_gdesc, gs->desc.data(), sizeof(GatherDev) * gs->desc.size());
    if (!gs->idx.empty()) memcpy(host + o_gdesc + b_gdesc, gs->idx.data(), sizeof(int) * gs->idx.size());
  }
  for (int i = 0; i < count; ++i)
    if (!P[i].ext.empty() && !ext_pool) memcpy(host + o_pool + P[i].d.a_off, P[i].ext.data(), P[i].ext.size());
  // uploads: stream-ordered on the creation stream when one is given (pageable sources are
  // staged before cudaMemcpyAsync returns), else synchronous
  auto up = [&](void* dst, const void* src, size_t bytes) -> cudaError_t {
    return cs ? cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, cs)
              : cudaMemcpy(dst, src, bytes, cudaMemcpyHostToDevice);
  };
  CK(up(pl->dmem, host, staged));
  pl->h2d_bytes = (long long)staged;
  if (gs && count > 0) {  // pools are formed on the device
    gather_kernel<<<count, 256, 0, cs>>>(d_desc, d_idx, gs->B, gs->gamma, gs->M, pl->d_pool);
    CK(cudaGetLastError());
  }
  if (!cs) CK(cudaStreamSynchronize(0));
  if (!pl->trees.empty()) {  // what a per-term plan of the same instances needs (terms_plan)
    pl->prep = std::move(P);
    for (Prepared& p : pl->prep) std::vector<unsigned char>().swap(p.ext);
    pl->opt = opt;
  }
  return WG_OK;
}

// The per-term plan of a plan with trees, made on first use over the same device matrices: its
// magnitudes, chunks and partials are those of the sieve's terms.  What the caller's streams have in
// flight may still write those matrices, and the query may come on any stream: the device is waited
// for, and the plan's own memory is allocated and filled synchronously.
static void destroy_plan(wg_plan* pl);
static int terms_plan(const wg_plan* pl, const wg_plan** out) {
  *out = pl;
  if (pl->prep.empty()) return WG_OK;
  if (!pl->terms) {
    int rc = ensure_init(pl->device);
    if (rc) return rc;
    CK(cudaDeviceSynchronize());
    std::vector<Prepared> P = pl->prep;
    for (Prepared& p : P) p.tree = false;
    wg_plan_options opt = pl->opt;
    opt.stream = nullptr;
    wg_plan* t = new wg_plan();
    rc = finalize_plan(P, pl->precision, opt, t, nullptr, pl->d_pool);
    if (rc) { destroy_plan(t); return rc; }
    pl->terms = t;
  }
  *out = pl->terms;
  return WG_OK;
}
static int launch_plan(wg_plan* pl, cudaStream_t st);
// The same, run for the plan's last execution
static int terms_run(const wg_plan* pl, cudaStream_t st, const wg_plan** out) {
  const int rc = terms_plan(pl, out);
  if (rc || *out == pl || pl->terms_of == pl->executions) return rc;
  const int rc2 = launch_plan(pl->terms, st);
  if (!rc2) pl->terms_of = pl->executions;
  return rc2;
}

// `n` side streams that start where `st` stands
static int fork_side(wg_plan* pl, cudaStream_t st, size_t n) {
  if (!pl->fork) CK(cudaEventCreateWithFlags(&pl->fork, cudaEventDisableTiming));
  while (pl->side.size() < n) {
    cudaStream_t s2;
    cudaEvent_t e2;
    CK(cudaStreamCreateWithFlags(&s2, cudaStreamNonBlocking));
    CK(cudaEventCreateWithFlags(&e2, cudaEventDisableTiming));
    pl->side.push_back(s2);
    pl->side_done.push_back(e2);
  }
  CK(cudaEventRecord(pl->fork, st));
  for (size_t g = 0; g < n; ++g) CK(cudaStreamWaitEvent(pl->side[g], pl->fork, 0));
  return WG_OK;
}
static int join_side(wg_plan* pl, cudaStream_t st, size_t g) {
  CK(cudaEventRecord(pl->side_done[g], pl->side[g]));
  CK(cudaStreamWaitEvent(st, pl->side_done[g], 0));
  return WG_OK;
}

static int launch_trees(wg_plan* pl, cudaStream_t st) {
  TreeMods side;
  side.n = 0;
  if (pl->fork_trees) {
    const int rc = fork_side(pl, st, pl->trees.size() - 1);
    if (rc) return rc;
  }
  for (size_t i = 0; i < pl->trees.size(); ++i) {
    const TreeLaunch& G = pl->trees[i];
    const bool forked = pl->fork_trees && i > 0;
    TreeParams p;
    memset(&p, 0, sizeof(p));
    p.pool = pl->d_pool;
    p.partials = pl->d_partials;
    p.ws = pl->d_ws + G.ws_off;
    p.polls = pl->polls;
    p.err = pl->d_err;
    p.ninst = G.ninst;
    p.nrounds = G.nrounds;
    p.nsegs = G.nsegs;
    p.inst = (const TreeInst*)(pl->d_prog + G.prog_off);
    p.rounds = (const TreeRound*)(p.inst + G.ninst);
    p.segs = (const TreeSeg*)(p.rounds + G.nrounds);
    p.cached = G.cached;
    p.sm_warp = G.sm_warp;
    p.sm_cache = G.sm_cache;
    p.sm_ws = G.sm_ws;
    p.bar = pl->d_counters + G.counter;
    if (plan_single(pl)) {
      p.fin.inst = pl->d_inst;
      p.fin.ninst = (int)pl->inst.size();
      p.fin.partials = pl->d_partials;
      p.fin.scales = pl->d_scales;
      p.fin.out = pl->d_out;
      p.fin.mags = pl->d_mag;
      p.fin.err = pl->d_err;
      p.fin.counters = pl->d_counters + G.counter;
      p.fin.ncounters = 2;
      p.fin.done = p.fin.counters + 1;
      const int each = pl->total_out / pl->primes, g = side.n;
      p.fin.first_out = g * each;
      p.fin.end_out = (g + 1) * each;
      p.fin.wpo = plan_wpo(pl, TREE_THREADS / 32);
    }
    if (pl->side_trees) {
      side.prime[side.n] = G.ttype - ST_MOD0;
      side.p[side.n++] = p;  // the primes' programs are alike: G.ctas and G.smem too
      if (side.n < (int)pl->trees.size()) continue;
    }
    const cudaError_t e = pl->side_trees ? tree_launch_mods(side, G.ctas * side.n, G.smem, st)
                                         : tree_launch(G.ttype, p, G.ctas, G.smem, forked ? pl->side[i - 1] : st);
    if (e != cudaSuccess) return fail(WG_ECUDA, "tree launch: %s", cudaGetErrorString(e));
    if (forked) {
      const int rc = join_side(pl, st, i - 1);
      if (rc) return rc;
    }
  }
  return WG_OK;
}

static int launch_plan(wg_plan* pl, cudaStream_t st) {
  const int trc = launch_trees(pl, st);
  if (trc) return trc;
  const size_t ng = pl->groups.size();
  const bool side = ng > 1 && !pl->serial_groups;
  if (side) {
    const int rc = fork_side(pl, st, ng - 1);
    if (rc) return rc;
  }
  for (size_t g = 0; g < ng; ++g) {
    const Group& G = pl->groups[g];
    SieveParams p;
    const DevTables& T = g_dev[pl->device];
    p.lb_lane = T.lane;
    p.lb_own = T.own;
    p.lb_lane2 = T.lane2;
    p.lb_own2 = T.own2;
    p.inst = pl->d_inst;
    p.chunks = pl->d_chunks + G.chunk_begin;
    p.nchunks = G.chunk_count;
    p.pool = pl->d_pool;
    p.partials = pl->d_partials;
    p.counter = pl->d_counters + g;
    p.err = pl->d_err;
    p.L = G.L;
    const cudaStream_t gs = (g == 0 || !side) ? st : pl->side[g - 1];
    const cudaError_t e = sieve_launch(G.stype, p, G.ctas, G.wpc, gs);
    if (e != cudaSuccess) return fail(WG_ECUDA, "sieve launch: %s", cudaGetErrorString(e));
    if (g > 0 && side) {
      const int rc = join_side(pl, st, g - 1);
      if (rc) return rc;
    }
  }
  const int ninst = (int)pl->inst.size();
  if (ninst > 0 && !plan_single(pl)) {
    const int threads = 256, wpo = plan_wpo(pl, threads / 32);
    const int per = threads / 32 / wpo, blocks = (pl->total_out + per - 1) / per;
    reduce_kernel<<<std::max(blocks, 1), threads, 0, st>>>(pl->d_inst, ninst, pl->d_partials, pl->d_scales, pl->d_out,
                                                           pl->d_counters, plan_counters(pl), pl->total_out, wpo,
                                                           pl->d_mag, pl->d_err);
    CK(cudaGetLastError());
  }
  return WG_OK;
}

// Direct launches, or -- with use_graph -- one CUDA graph captured on first use (the launch
// attributes are set by a direct execution first) and replayed on the caller's stream.
static int execute_plan(wg_plan* pl, cudaStream_t st) {
  ++pl->executions;
  if (!pl->use_graph) return launch_plan(pl, st);
  if (!pl->graph_exec) {
    int rc = launch_plan(pl, st);  // sets the kernels' shared-memory attributes, warms up
    if (rc) return rc;
    CK(cudaStreamSynchronize(st));
    cudaStream_t cap;
    CK(cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking));
    cudaGraph_t graph = nullptr;
    cudaError_t e = cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess) {
      rc = launch_plan(pl, cap);
      e = cudaStreamEndCapture(cap, &graph);
    }
    if (e == cudaSuccess && rc == 0) e = cudaGraphInstantiate(&pl->graph_exec, graph, 0);
    if (graph) cudaGraphDestroy(graph);
    cudaStreamDestroy(cap);
    if (rc) return rc;
    if (e != cudaSuccess) return fail(WG_ECUDA, "graph capture: %s", cudaGetErrorString(e));
    return WG_OK;  // this call already executed the plan once
  }
  CK(cudaGraphLaunch(pl->graph_exec, st));
  return WG_OK;
}

// The outputs, when `st` has come to them (written into pinned memory by the kernels, or copied).  An
// execution whose launch gave up is an error, reported once: the flag is cleared for the next one.
static int read_outputs(wg_plan* pl, double* out, cudaStream_t st) {
  const size_t bytes = sizeof(double2) * pl->total_out;
  if (bytes && !pl->h_out) CK(cudaMemcpyAsync(out, pl->d_out, bytes, cudaMemcpyDeviceToHost, st));
  CK(cudaStreamSynchronize(st));
  if (bytes && pl->h_out) memcpy(out, pl->h_out, bytes);
  for (int i = 0; i < pl->total_out; ++i) {
    if (memcmp(out + 2 * i, &GAVE_UP, sizeof(GAVE_UP))) continue;
    CK(cudaMemsetAsync(pl->d_err, 0, sizeof(int), st));
    return fail(WG_ECUDA, "a tree launch gave up waiting for its own blocks");
  }
  return WG_OK;
}

static void destroy_plan(wg_plan* pl) {
  if (!pl) return;
  destroy_plan(pl->terms);
  if (pl->graph_exec) cudaGraphExecDestroy(pl->graph_exec);
  for (cudaStream_t s2 : pl->side) cudaStreamDestroy(s2);
  for (cudaEvent_t e2 : pl->side_done) cudaEventDestroy(e2);
  if (pl->fork) cudaEventDestroy(pl->fork);
  if (pl->dmem) {
    if (pl->async_alloc) cudaFreeAsync(pl->dmem, pl->alloc_stream);
    else cudaFree(pl->dmem);
  }
  delete pl;
}

// ---------------------------------------------------------------- FP pipe microbenchmark
template <typename T>
__global__ void fma_peak_kernel(T* out, int iters, T a, T b) {
  T x[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) x[c] = (T)(threadIdx.x + c);
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int c = 0; c < 8; ++c) x[c] = x[c] * a + b;
  }
  T s = 0;
#pragma unroll
  for (int c = 0; c < 8; ++c) s += x[c];
  out[blockIdx.x * blockDim.x + threadIdx.x] = s;
}

template <typename T>
static int time_peak(int blocks, int threads, int iters, double* tflops) {
  T* buf = nullptr;
  CK(cudaMalloc(&buf, sizeof(T) * blocks * threads));
  cudaEvent_t e0, e1;
  CK(cudaEventCreate(&e0));
  CK(cudaEventCreate(&e1));
  float best = 1e30f;
  for (int rep = 0; rep < 4; ++rep) {
    CK(cudaEventRecord(e0));
    fma_peak_kernel<T><<<blocks, threads>>>(buf, iters, (T)0.999999, (T)1e-7);
    CK(cudaEventRecord(e1));
    CK(cudaEventSynchronize(e1));
    float ms = 0;
    CK(cudaEventElapsedTime(&ms, e0, e1));
    if (rep > 0) best = std::min(best, ms);
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(buf);
  *tflops = 2.0 * 8.0 * (double)blocks * threads * (double)iters / (best * 1e-3) / 1e12;
  return WG_OK;
}

}  // namespace wg

using namespace wg;

extern "C" {

int wg_init(int device) { return ensure_init(device); }

const char* wg_last_error(void) { return g_err.c_str(); }

int wg_instance_outputs(const wg_instance* in) {
  if (!in) return fail(WG_EINVAL, "NULL instance");
  if (in->kind == WG_KIND_BATCH_EVEN) return 2 * in->batch_max + in->cutoff + 1;
  if (in->kind == WG_KIND_BATCH_ODD) return 2 * in->batch_max + in->cutoff + 2;
  return 1;
}

long long wg_instance_terms(const wg_instance* in) {
  if (!in) return fail(WG_EINVAL, "NULL instance");
  Prepared P;
  wg_instance whole = *in;
  whole.term_begin = whole.term_end = 0;
  const int rc = prepare(whole, WG_PREC_FP64, P);
  return rc ? (long long)rc : P.d.steps;
}

int wg_plan_create_ex(const wg_instance* inst, int count, int precision, const wg_plan_options* options,
                      wg_plan** plan) {
  if (!plan) return fail(WG_EINVAL, "plan is NULL");
  *plan = nullptr;
  if (!known_precision(precision)) return fail(WG_EINVAL, "unknown precision %d", precision);
  int rc = ensure_init(-1);
  if (rc) return rc;
  wg_plan_options opt;
  memset(&opt, 0, sizeof(opt));
  opt.chunk_scale = 1.0;
  if (options) opt = *options;
  wg_plan* pl = new wg_plan();
  rc = build_plan(inst, count, precision, opt, pl);
  if (rc) { destroy_plan(pl); return rc; }
  *plan = pl;
  return WG_OK;
}

int wg_plan_create(const wg_instance* inst, int count, int precision, double chunk_scale, wg_plan** plan) {
  wg_plan_options opt;
  memset(&opt, 0, sizeof(opt));
  opt.chunk_scale = chunk_scale;
  return wg_plan_create_ex(inst, count, precision, &opt, plan);
}

int wg_plan_execute(wg_plan* plan, void* stream) {
  if (!plan) return fail(WG_EINVAL, "plan is NULL");
  int rc = ensure_init(-1);
  if (rc) return rc;
  return execute_plan(plan, (cudaStream_t)stream);
}

int wg_plan_read(wg_plan* plan, double* out, void* stream) {
  if (!plan || (!out && plan->total_out > 0)) return fail(WG_EINVAL, "NULL argument");
  return read_outputs(plan, out, (cudaStream_t)stream);
}

int wg_plan_barrier_polls(wg_plan* plan, unsigned int polls) {
  if (!plan) return fail(WG_EINVAL, "plan is NULL");
  plan->polls = polls ? polls : TREE_POLLS;
  return WG_OK;
}

int wg_plan_read_magnitudes(wg_plan* plan, double* out, void* stream) {
  if (!plan || (!out && plan->total_out > 0)) return fail(WG_EINVAL, "NULL argument");
  cudaStream_t st = (cudaStream_t)stream;
  std::lock_guard<std::mutex> lk(*plan->terms_mu);
  const wg_plan* terms = nullptr;
  const int rc = terms_run(plan, st, &terms);
  if (rc) return rc;
  if (plan->total_out > 0)
    CK(cudaMemcpyAsync(out, terms->d_mag, sizeof(double) * plan->total_out, cudaMemcpyDeviceToHost, st));
  CK(cudaStreamSynchronize(st));
  return WG_OK;
}

int wg_plan_outputs(const wg_plan* plan) { return plan ? plan->total_out : fail(WG_EINVAL, "plan is NULL"); }

int wg_plan_trees(const wg_plan* plan) { return plan ? plan->ntrees : fail(WG_EINVAL, "plan is NULL"); }

int wg_plan_kernel_launches(const wg_plan* plan) {
  if (!plan) return fail(WG_EINVAL, "plan is NULL");
  const size_t trees = plan->side_trees ? 1 : plan->trees.size();
  return (int)(plan->groups.size() + trees) + (plan->inst.empty() || plan_single(plan) ? 0 : 1);
}

int wg_plan_partials(wg_plan* plan, double* out, int capacity, void* stream) {
  if (!plan) return fail(WG_EINVAL, "plan is NULL");
  cudaStream_t st = (cudaStream_t)stream;
  std::lock_guard<std::mutex> lk(*plan->terms_mu);
  const wg_plan* terms = nullptr;
  int rc = terms_plan(plan, &terms);
  if (rc) return rc;
  if (!out || capacity < terms->nparts) return terms->nparts;
  rc = terms_run(plan, st, &terms);
  if (rc) return rc;
  if (terms->nparts > 0)
    CK(cudaMemcpyAsync(out, terms->d_partials, sizeof(double2) * terms->nparts, cudaMemcpyDeviceToHost, st));
  CK(cudaStreamSynchronize(st));
  return terms->nparts;
}

int wg_plan_chunk(const wg_plan* plan, int chunk, int* inst, int* part, long long* t0, long long* t1) {
  if (!plan) return fail(WG_EINVAL, "bad chunk index");
  std::lock_guard<std::mutex> lk(*plan->terms_mu);
  const wg_plan* terms = nullptr;
  const int rc = terms_plan(plan, &terms);
  if (rc) return rc;
  if (chunk < 0 || chunk >= (int)terms->chunks.size()) return fail(WG_EINVAL, "bad chunk index");
  const ChunkDev& c = terms->chunks[chunk];
  if (inst) *inst = c.inst;
  if (part) *part = c.part;
  if (t0) *t0 = c.t0;
  if (t1) *t1 = c.t1;
  return (int)terms->chunks.size();
}

int wg_state_create(const double* B, const double* gamma, int M, wg_state** state) {
  if (!state || !B || !gamma || M < 1) return fail(WG_EINVAL, "bad state arguments");
  *state = nullptr;
  int rc = ensure_init(-1);
  if (rc) return rc;
  wg_state* st = new wg_state();
  st->M = M;
  st->gamma.resize(M);
  double rs = 0;
  for (int i = 0; i < M; ++i) {
    st->gamma[i] = {gamma[2 * i], gamma[2 * i + 1]};
    double s = 0;
    for (int j = 0; j < M; ++j) s += std::hypot(B[2 * ((size_t)i * M + j)], B[2 * ((size_t)i * M + j) + 1]);
    rs = std::max(rs, s);
  }
  if (rs > 0 && std::isfinite(rs)) st->alpha = std::exp2(-std::round(std::log2(rs)));
  if (cudaMalloc(&st->d_B, sizeof(c64) * (size_t)M * M) != cudaSuccess ||
      cudaMalloc(&st->d_gamma, sizeof(c64) * M) != cudaSuccess) {
    cudaGetLastError();
    if (st->d_B) cudaFree(st->d_B);
    delete st;
    return fail(WG_ENOMEM, "state allocation failed");
  }
  CK(cudaMemcpy(st->d_B, B, sizeof(c64) * (size_t)M * M, cudaMemcpyHostToDevice));
  CK(cudaMemcpy(st->d_gamma, gamma, sizeof(c64) * M, cudaMemcpyHostToDevice));
  st->form = matrix_form(B, WG_COMPLEX128, (size_t)M, tree_asymmetry(WG_PREC_FP64));
  st->B.resize((size_t)M * M);
  memcpy(st->B.data(), B, sizeof(c64) * st->B.size());
  state_parts(*st);
  *state = st;
  return WG_OK;
}

int wg_state_create_from_cov(const double* cov, const double* mu, int M, double hbar, wg_state** state,
                             double vacuum[2], double* B_out, double* gamma_out) {
  if (!state || !cov || !mu || !vacuum || M < 1 || M > 512 || !(hbar > 0))
    return fail(WG_EINVAL, "bad state arguments (1 <= M <= 512 modes, hbar > 0)");
  *state = nullptr;
  int rc = ensure_init(-1);
  if (rc) return rc;
  const int n = 2 * M;
  double *d_cov = nullptr, *d_mu = nullptr, *d_out = nullptr;
  c64 *d_Q = nullptr, *d_X = nullptr;
  wg_state* st = new wg_state();
  st->M = M;
  auto release = [&]() {
    if (d_cov) cudaFree(d_cov);
    if (d_mu) cudaFree(d_mu);
    if (d_out) cudaFree(d_out);
    if (d_Q) cudaFree(d_Q);
    if (d_X) cudaFree(d_X);
  };
  auto abandon = [&](int code, const char* what) {
    cudaGetLastError();
    release();
    if (st->d_B) cudaFree(st->d_B);
    if (st->d_gamma) cudaFree(st->d_gamma);
    delete st;
    return fail(code, "%s", what);
  };
  if (cudaMalloc(&st->d_B, sizeof(c64) * (size_t)M * M) != cudaSuccess ||
      cudaMalloc(&st->d_gamma, sizeof(c64) * M) != cudaSuccess ||
      cudaMalloc(&d_cov, sizeof(double) * (size_t)n * n) != cudaSuccess ||
      cudaMalloc(&d_mu, sizeof(double) * n) != cudaSuccess || cudaMalloc(&d_out, sizeof(double) * 8) != cudaSuccess ||
      cudaMalloc(&d_Q, sizeof(c64) * (size_t)n * n) != cudaSuccess ||
      cudaMalloc(&d_X, sizeof(c64) * (size_t)n * M) != cudaSuccess)
    return abandon(WG_ENOMEM, "state allocation failed");
  if (cudaMemcpy(d_cov, cov, sizeof(double) * (size_t)n * n, cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemcpy(d_mu, mu, sizeof(double) * n, cudaMemcpyHostToDevice) != cudaSuccess)
    return abandon(WG_ECUDA, "state upload failed");
  gaussian_state_kernel<<<1, 1024>>>(d_cov, d_mu, M, hbar, d_Q, d_X, st->d_B, st->d_gamma, d_out);
  double out[8] = {0};
  if (cudaGetLastError() != cudaSuccess || cudaMemcpy(out, d_out, sizeof(double) * 5, cudaMemcpyDeviceToHost) != cudaSuccess)
    return abandon(WG_ECUDA, "state kernel failed");
  if (out[4] != 0.0) return abandon(WG_EINVAL, "covariance is not a physical state: its Husimi matrix Q is not positive definite");
  st->gamma.resize(M);
  if (cudaMemcpy(st->gamma.data(), st->d_gamma, sizeof(c64) * M, cudaMemcpyDeviceToHost) != cudaSuccess)
    return abandon(WG_ECUDA, "state readback failed");
  if (B_out && cudaMemcpy(B_out, st->d_B, sizeof(c64) * (size_t)M * M, cudaMemcpyDeviceToHost) != cudaSuccess)
    return abandon(WG_ECUDA, "state readback failed");
  if (gamma_out) memcpy(gamma_out, st->gamma.data(), sizeof(c64) * M);
  st->B.resize((size_t)M * M);
  if (cudaMemcpy(st->B.data(), st->d_B, sizeof(c64) * st->B.size(), cudaMemcpyDeviceToHost) != cudaSuccess)
    return abandon(WG_ECUDA, "state readback failed");
  st->form = matrix_form(st->B.data(), WG_COMPLEX128, (size_t)M, tree_asymmetry(WG_PREC_FP64));
  state_parts(*st);
  release();
  const double rs = out[3];
  if (rs > 0 && std::isfinite(rs)) st->alpha = std::exp2(-std::round(std::log2(rs)));
  // <0|psi> = exp(-quad / 2) / det(Q)^(1/4)
  const double mag = std::exp(-0.5 * out[1] - 0.25 * out[0]);
  vacuum[0] = mag * std::cos(-0.5 * out[2]);
  vacuum[1] = mag * std::sin(-0.5 * out[2]);
  *state = st;
  return WG_OK;
}

int wg_state_destroy(wg_state* state) {
  if (!state) return WG_OK;
  if (state->d_B) cudaFree(state->d_B);
  if (state->d_gamma) cudaFree(state->d_gamma);
  delete state;
  return WG_OK;
}

int wg_plan_create_requests(const wg_state* state, const wg_request* req, int count, int precision,
                            const wg_plan_options* options, wg_plan** plan) {
  if (!plan || !state || count < 0 || (count > 0 && !req)) return fail(WG_EINVAL, "bad request list");
  *plan = nullptr;
  if ((precision & ~kEvaluations) != WG_PREC_FP64 && (precision & ~kEvaluations) != WG_PREC_DF)
    return fail(WG_EINVAL, "unknown precision %d", precision);
  int rc = ensure_init(-1);
  if (rc) return rc;
  wg_plan_options opt;
  memset(&opt, 0, sizeof(opt));
  opt.chunk_scale = 1.0;
  if (options) opt = *options;
  std::vector<Prepared> P(count);
  GatherSpec gs;
  gs.B = state->d_B;
  gs.gamma = state->d_gamma;
  gs.M = state->M;
  gs.desc.resize(count);
  for (int i = 0; i < count; ++i) {
    rc = prepare_request(req[i], *state, precision, P[i], gs.desc[i], gs.idx);
    if (rc) return fail(rc, "request %d: %s", i, g_err.c_str());
  }
  wg_plan* pl = new wg_plan();
  rc = finalize_plan(P, precision, opt, pl, &gs, nullptr);
  if (rc) { destroy_plan(pl); return rc; }
  *plan = pl;
  return WG_OK;
}

long long wg_plan_device_bytes(const wg_plan* plan) { return plan ? plan->device_bytes : 0; }

int wg_plan_transfer_bytes(const wg_plan* plan, long long* h2d, long long* d2h) {
  if (!plan) return fail(WG_EINVAL, "plan is NULL");
  if (h2d) *h2d = plan->h2d_bytes;
  if (d2h) *d2h = (long long)sizeof(double2) * plan->total_out;
  return WG_OK;
}

int wg_plan_destroy(wg_plan* plan) {
  destroy_plan(plan);
  return WG_OK;
}

// One-shot plans run stream-ordered on the caller's stream, or on the calling thread's default
// stream: their memory comes from the stream-ordered pool and goes back to it without a
// device-wide synchronisation, and the uploads need none either; upload and results go through a
// pinned block.
int wg_run(const wg_instance* inst, int count, int precision, double* out, void* stream) {
  const cudaStream_t st = stream ? (cudaStream_t)stream : cudaStreamPerThread;
  wg_plan_options opt;
  memset(&opt, 0, sizeof(opt));
  opt.chunk_scale = 1.0;
  opt.stream = st;
  int rc = ensure_init(-1);
  if (rc) return rc;
  wg_plan* pl = new wg_plan();
  pl->pinned = pinned_take();
  rc = build_plan(inst, count, precision, opt, pl);
  if (!rc) rc = execute_plan(pl, st);
  if (!rc && !out && pl->total_out > 0) rc = fail(WG_EINVAL, "NULL argument");
  if (!rc) rc = read_outputs(pl, out, st);
  // nothing in flight may still read or write the block that the next call takes
  if (rc) cudaStreamSynchronize(st);
  pinned_give(pl->pinned);
  destroy_plan(pl);
  return rc;
}

// An ordinary (loop) hafnian straight from the caller's matrix: the checks of the public function
// (finite, symmetric and not diagonal in numpy.allclose's sense, not integer-valued, paired rows of
// comparable sums), the pairing of single indices (n-1 with n-2, n-3 with n-4, ...; 0 is left over
// when n is odd), and the run.  *done = 0, with nothing computed, whenever a check says that
// the general route has to answer.
int wg_hafnian_direct(const void* A, int n, int dtype, int loop, double rtol, double atol, double out[2], int* done) {
  if (!done || !out || !A) return fail(WG_EINVAL, "NULL argument");
  *done = 0;
  if (n < 5 || (n % 2 && !loop) || n / 2 > MAX_EDGES || !(rtol >= 0) || !(atol >= 0)) return WG_OK;
  if (dtype != WG_FLOAT64 && dtype != WG_COMPLEX128) return WG_OK;
  const double* a = (const double*)A;
  const size_t nn = (size_t)n * n;
  const bool cx = dtype == WG_COMPLEX128;
  bool imag = false, integral = true;
  for (size_t k = 0; k < nn; ++k) {
    const double re = cx ? a[2 * k] : a[k], im = cx ? a[2 * k + 1] : 0.0;
    if (!(std::isfinite(re) && std::isfinite(im))) return WG_OK;
    imag = imag || im != 0;
    integral = integral && re == std::nearbyint(re);
  }
  if (!imag && integral) return WG_OK;
  // real values of a complex matrix run the real tree
  std::vector<double> real;
  if (cx && !imag) {
    real.resize(nn);
    for (size_t k = 0; k < nn; ++k) real[k] = a[2 * k];
    a = real.data();
  }
  auto mod = [&](int i, int j) {
    const size_t k = (size_t)i * n + j;
    return imag ? std::hypot(a[2 * k], a[2 * k + 1]) : std::fabs(a[k]);
  };
  bool diagonal = true;
  std::vector<double> rows(n, 0.0);
  for (int i = 0; i < n; ++i)
    for (int j = 0; j < n; ++j) {
      const double m = mod(i, j);
      if (n % 2 == 0 || j) rows[i] += m;  // of the paired vertices, as _pair_balance's
      if (i == j) {
        if (loop) rows[i] += m;
        continue;
      }
      diagonal = diagonal && m <= atol + rtol * m;
      const size_t x = (size_t)i * n + j, y = (size_t)j * n + i;  // |A_ji - A_ij| against |A_ij|
      const double d = imag ? (a[2 * x] == a[2 * y] && a[2 * x + 1] == a[2 * y + 1]
                                   ? 0.0
                                   : std::hypot(a[2 * y] - a[2 * x], a[2 * y + 1] - a[2 * x + 1]))
                            : std::fabs(a[y] - a[x]);
      if (!(d <= atol + rtol * m)) return WG_OK;
    }
  if (diagonal) return WG_OK;
  const int E = n / 2;
  std::vector<int> x(2 * E);
  for (int e = 0; e < E; ++e) {
    x[e] = n - 1 - 2 * e;
    x[E + e] = n - 2 - 2 * e;
    const double ra = rows[x[e]], rb = rows[x[E + e]];
    if (ra > 0 && rb > 0 && !(ra <= 16.0 * rb && rb <= 16.0 * ra)) return WG_OK;  // _pair_balance's spread
  }
  const int w = imag ? 2 : 1, m = 2 * E;
  std::vector<double> Ax((size_t)m * m * w), D, V;
  for (int i = 0; i < m; ++i)
    for (int j = 0; j < m; ++j) memcpy(&Ax[((size_t)i * m + j) * w], a + ((size_t)x[i] * n + x[j]) * w, sizeof(double) * w);
  std::vector<int64_t> reps(E, 1);
  wg_instance in;
  memset(&in, 0, sizeof(in));
  in.kind = loop ? WG_KIND_LOOP : WG_KIND_PLAIN;
  in.n = m;
  in.E = E;
  in.dtype = imag ? WG_COMPLEX128 : WG_FLOAT64;
  in.glynn = 1;
  in.edge_reps = reps.data();
  in.A = Ax.data();
  if (loop) {
    D.resize((size_t)m * w);
    for (int i = 0; i < m; ++i) memcpy(&D[(size_t)i * w], a + ((size_t)x[i] * n + x[i]) * w, sizeof(double) * w);
    in.D = D.data();
    if (n % 2) {
      V.resize((size_t)m * w);
      for (int i = 0; i < m; ++i) memcpy(&V[(size_t)i * w], a + (size_t)x[i] * w, sizeof(double) * w);
      in.has_odd = 1;
      in.oddV = V.data();
      memcpy(in.oddloop, a, sizeof(double) * w);
    }
  }
  const int rc = wg_run(&in, 1, WG_PREC_FP64, out, nullptr);
  if (!rc) *done = 1;
  return rc;
}

// Pairing of repeated indices into edges with multiplicities (thewalrus/_hafnian.py:80-159): the two
// largest remaining counts (ties: the larger index first) pair as often as the second allows; one
// that exceeds twice the second, or is alone, pairs with itself.  x: the edges' first ends, then
// their second ends (2 * *E entries, room for 4 n: an index pairs with itself at most once, which
// leaves it 1 or 0, and every other edge uses an index up, so there are at most 2 n edges); mult: *E
// entries (room for 2 n); *odd: the index left over, or -1.
int wg_matched_reps(const int64_t* reps, int n, int64_t* x, int64_t* mult, int* E, int* odd) {
  if ((n > 0 && (!reps || !x || !mult)) || n < 0 || !E || !odd) return fail(WG_EINVAL, "bad pairing arguments");
  *E = 0;
  *odd = -1;
  __int128 sum = 0;
  std::vector<std::pair<int64_t, int>> pool;  // a heap by count, then index
  for (int i = 0; i < n; ++i) {
    sum += reps[i];
    if (reps[i] > 0) pool.emplace_back(reps[i], i);
  }
  if (sum == 0) return WG_OK;
  std::make_heap(pool.begin(), pool.end());
  auto pop = [&] {
    std::pop_heap(pool.begin(), pool.end());
    const auto t = pool.back();
    pool.pop_back();
    return t;
  };
  auto push = [&](int64_t r, int i) {
    pool.emplace_back(r, i);
    std::push_heap(pool.begin(), pool.end());
  };
  std::vector<int64_t> right;
  int e = 0;
  while (pool.size() > 1 || (pool.size() == 1 && pool.front().first > 1)) {
    const auto top = pop();
    if (pool.empty() || top.first - pool.front().first > pool.front().first) {
      x[e] = top.second;
      right.push_back(top.second);
      mult[e++] = top.first / 2;
      if (top.first % 2) push(1, top.second);
    } else {
      const auto sec = pop();
      x[e] = top.second;
      right.push_back(sec.second);
      mult[e++] = sec.first;
      if (top.first > sec.first) push(top.first - sec.first, top.second);
    }
  }
  std::copy(right.begin(), right.end(), x + e);
  *E = e;
  if (pool.size() == 1) *odd = pool.front().second;
  return WG_OK;
}

int wg_hafnian(const void* A, int n, int dtype, const int64_t* edge_reps, int E, int glynn, int precision,
               double out[2], void* stream) {
  wg_instance in;
  memset(&in, 0, sizeof(in));
  in.kind = WG_KIND_PLAIN;
  in.n = n;
  in.E = E;
  in.dtype = dtype;
  in.glynn = glynn;
  in.edge_reps = edge_reps;
  in.A = A;
  return wg_run(&in, 1, precision, out, stream);
}

int wg_loop_hafnian(const void* A, const void* D, int n, int dtype, const int64_t* edge_reps, int E, int has_odd,
                    const double oddloop[2], const void* oddV, int glynn, int precision, double out[2],
                    void* stream) {
  wg_instance in;
  memset(&in, 0, sizeof(in));
  in.kind = WG_KIND_LOOP;
  in.n = n;
  in.E = E;
  in.dtype = dtype;
  in.glynn = glynn;
  in.has_odd = has_odd;
  in.edge_reps = edge_reps;
  in.A = A;
  in.D = D;
  in.oddV = oddV;
  if (has_odd && oddloop) { in.oddloop[0] = oddloop[0]; in.oddloop[1] = oddloop[1]; }
  return wg_run(&in, 1, precision, out, stream);
}

int wg_loop_hafnian_batch(const void* A, const void* D, int n, int dtype, const int64_t* fixed_edge_reps, int E,
                          int batch_max, int cutoff, int odd, int glynn, int precision, double* out, void* stream) {
  wg_instance in;
  memset(&in, 0, sizeof(in));
  in.kind = odd ? WG_KIND_BATCH_ODD : WG_KIND_BATCH_EVEN;
  in.n = n;
  in.E = E;
  in.dtype = dtype;
  in.glynn = glynn;
  in.batch_max = batch_max;
  in.cutoff = cutoff;
  in.edge_reps = fixed_edge_reps;
  in.A = A;
  in.D = D;
  return wg_run(&in, 1, precision, out, stream);
}

// Device arithmetic primitives of the kernels, evaluated elementwise for checks against IEEE and
// exact references: 0 recip_newton(x); 1 dd_recip((x, lo)) -> (hi, lo); 2 dd_div_int((x, lo), k)
// with k = (int)y -> (hi, lo); 3 dd_mul((x, lo), (y, lo2)) -> (hi, lo).  Inputs per element:
// in[4i .. 4i+3] = x, x_lo, y, y_lo; outputs out[2i], out[2i+1].
static __global__ void arith_check_kernel(int op, const double* __restrict__ in, int n, double* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double x = in[4 * i], xl = in[4 * i + 1], y = in[4 * i + 2], yl = in[4 * i + 3];
  ddr r = {0.0, 0.0};
  switch (op) {
    case 0: r.hi = recip_newton(x); break;
    case 1: r = dd_recip({x, xl}); break;
    case 2: r = dd_div_int({x, xl}, (int)y); break;
    case 3: r = dd_mul({x, xl}, {y, yl}); break;
    case 4: {  // double-float reciprocal (inputs: the float parts)
      const dfr q = Ar<dfr>::recip({(float)x, (float)xl});
      r = {(double)q.hi, (double)q.lo};
      break;
    }
    case 5: {  // complex double-float reciprocal: out = (re, im), each part's hi + lo in FP64
      const cdf q = Ar<cdf>::recip({{(float)x, (float)xl}, {(float)y, (float)yl}});
      r = {df_to_d(q.re), df_to_d(q.im)};
      break;
    }
    default: {  // double-float division by a small integer
      const dfr q = df_div_int({(float)x, (float)xl}, (int)y);
      r = {(double)q.hi, (double)q.lo};
      break;
    }
  }
  out[2 * i] = r.hi;
  out[2 * i + 1] = r.lo;
}

int wg_check_arith(int op, const double* in, int n, double* out) {
  if (op < 0 || op > 6 || n < 0 || (n > 0 && (!in || !out))) return fail(WG_EINVAL, "bad arithmetic check arguments");
  if (n == 0) return WG_OK;
  int rc = ensure_init(-1);
  if (rc) return rc;
  double *d_in = nullptr, *d_out = nullptr;
  if (cudaMalloc(&d_in, sizeof(double) * 4 * (size_t)n) != cudaSuccess ||
      cudaMalloc(&d_out, sizeof(double) * 2 * (size_t)n) != cudaSuccess) {
    cudaGetLastError();
    if (d_in) cudaFree(d_in);
    return fail(WG_ENOMEM, "arithmetic check allocation failed");
  }
  cudaError_t e = cudaMemcpy(d_in, in, sizeof(double) * 4 * (size_t)n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    arith_check_kernel<<<(n + 255) / 256, 256>>>(op, d_in, n, d_out);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(out, d_out, sizeof(double) * 2 * (size_t)n, cudaMemcpyDeviceToHost);
  cudaFree(d_in);
  cudaFree(d_out);
  if (e != cudaSuccess) return fail(WG_ECUDA, "arithmetic check: %s", cudaGetErrorString(e));
  return WG_OK;
}

int wg_measure_fp_peaks(double* fp64_tflops, double* fp32_tflops) {
  int rc = ensure_init(-1);
  if (rc) return rc;
  if (fp64_tflops) {
    rc = time_peak<double>(g_num_sms * 4, 256, 2000, fp64_tflops);
    if (rc) return rc;
  }
  if (fp32_tflops) {
    rc = time_peak<float>(g_num_sms * 8, 256, 20000, fp32_tflops);
    if (rc) return rc;
  }
  return WG_OK;
}

}  // extern "C"
