// The tree kernel for residues, for every prime: the prime is a CTA's, read from shared memory into
// registers (a kernel per prime takes five times the code and could not run several side by side).
#include "kernels.h"

namespace wg {

struct ModPrime {
  uint32_t p, neg_inv, r1, r2;  // as in Montgomery<P>
  int index;
};
template <int I>
constexpr ModPrime mod_prime() {
  using M = Montgomery<MOD_PRIMES[I]>;
  return {MOD_PRIMES[I], M::NEG_INV, M::R1, M::R2, I};
}
static __constant__ ModPrime c_primes[MOD_N] = {mod_prime<0>(), mod_prime<1>(), mod_prime<2>(), mod_prime<3>(), mod_prime<4>()};
static __constant__ uint32_t c_inverses[MOD_N][256];
__device__ __forceinline__ ModPrime& cta_prime() {
  __shared__ ModPrime s_prime;
  return s_prime;
}

struct modr {
  uint32_t v;  // Montgomery form, as modp<P>
};
template <>
struct Ar<modr> {
  using S = modr;
  using Comp = modr;
  static constexpr int NC = 1;
  static constexpr bool cplx = false, fp64 = true, modular = true, dd = false;
  __device__ static __forceinline__ uint32_t fold(uint32_t s, uint32_t p) {  // s - p if that is not negative
    const uint32_t r = s - p;
    return s < r ? s : r;
  }
  __device__ static __forceinline__ uint32_t redc(uint64_t t) {
    const uint32_t p = cta_prime().p, m = (uint32_t)t * cta_prime().neg_inv;
    return fold((uint32_t)((t + (uint64_t)m * p) >> 32), p);
  }
  __device__ static __forceinline__ S zero() { return S{0u}; }
  __device__ static __forceinline__ S one() { return S{cta_prime().r1}; }
  __device__ static __forceinline__ S add(S a, S b) { return S{fold(a.v + b.v, cta_prime().p)}; }
  __device__ static __forceinline__ S sub(S a, S b) { return S{a.v >= b.v ? a.v - b.v : a.v + cta_prime().p - b.v}; }
  __device__ static __forceinline__ S neg(S a) { return sub(zero(), a); }
  __device__ static __forceinline__ S mul(S a, S b) { return S{redc((uint64_t)a.v * b.v)}; }
  __device__ static __forceinline__ S fma(S a, S b, S c) { return add(mul(a, b), c); }
  __device__ static __forceinline__ S of_int(long long k) {
    const long long p = cta_prime().p;
    if (k < 0 || k >= p) {
      k %= p;
      if (k < 0) k += p;
    }
    return S{redc((uint64_t)k * cta_prime().r2)};
  }
  __device__ static __forceinline__ S half() { return S{c_inverses[cta_prime().index][2]}; }
  // exact for the integers and half-integers the kernel scales by
  __device__ static __forceinline__ S scale(S a, double s) { return mul(mul(a, of_int(__double2ll_rn(2.0 * s))), half()); }
  // plain residues (< 2^31) travel through FP64 slots exactly
  __device__ static __forceinline__ S from_c64(c64 z) { return of_int(__double2ll_rn(z.re)); }
  __device__ static __forceinline__ c64 to_c64(S a) { return {(double)redc(a.v), 0.0}; }
  __device__ static __forceinline__ Comp comp(const S& a, int) { return a; }
  __device__ static __forceinline__ void set_comp(S& a, int, Comp v) { a = v; }
  __device__ static __forceinline__ Comp cadd(Comp a, Comp b) { return add(a, b); }
  __device__ static __forceinline__ Comp shfl_xor(Comp a, int m) { return S{__shfl_xor_sync(0xffffffffu, a.v, m)}; }
  __device__ static __forceinline__ S shfl(S a, int src) { return S{__shfl_sync(0xffffffffu, a.v, src)}; }
};
template <>
__device__ __forceinline__ modr inv_of<modr>(int k) {  // k < 256: at most 2 x 63 photon pairs
  return modr{c_inverses[cta_prime().index][k]};
}

// The products' 64-bit sum, below p 2^32 after every step (one multiply-add with a 64-bit addend and a
// conditional subtraction in the high word), is reduced when it is read: graph counts of n = 32 582 ->
// 459 us, n = 24 210 -> 191.
template <>
struct RealAcc<modr> {
  uint64_t v;
  __device__ static __forceinline__ RealAcc of(modr x) { return {(uint64_t)x.v << 32}; }
  __device__ __forceinline__ void fma(modr a, modr b) {
    v += (uint64_t)a.v * b.v;  // < 2^63 + 2^62
    v = (uint64_t)Ar<modr>::fold((uint32_t)(v >> 32), cta_prime().p) << 32 | (uint32_t)v;
  }
  __device__ __forceinline__ modr sum() const { return {Ar<modr>::redc(v)}; }
};

// An exact sum takes two to five primes, and one after another their narrow rounds leave the chip idle
// and wait for as many barriers each; side by side they take the time of one until the rounds fill
// the chip (graph counts, n = 24: 191 -> 123 us, n = 32: 459 -> 265, n = 36: 886 -> 723).
static __global__ void __launch_bounds__(TREE_THREADS, 1) tree_mods_kernel(const TreeMods M) {
  __shared__ TreeParams P;
  const int g = blockIdx.x % M.n;
  const int* src = reinterpret_cast<const int*>(&M.p[g]);
  for (int i = threadIdx.x; i < (int)(sizeof(TreeParams) / sizeof(int)); i += blockDim.x)
    reinterpret_cast<int*>(&P)[i] = src[i];
  if (threadIdx.x == 0) cta_prime() = c_primes[M.prime[g]];
  __syncthreads();
  tree_body<modr>(P, blockIdx.x / M.n, gridDim.x / M.n);
}

cudaError_t tree_launch_mods(const TreeMods& m, int ctas, int smem, cudaStream_t st) {
  return tree_launch_kernel<tree_mods_kernel>(m, ctas, ctas / m.n, smem, st);
}

cudaError_t sieve_tables_mods(const double* binom, const double* inv) {
  cudaError_t e = cudaMemcpyToSymbol(c_binom, binom, sizeof(c_binom));
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_inv, inv, sizeof(c_inv));
  if (e != cudaSuccess) return e;
  uint32_t inverses[MOD_N][256];
  for (int i = 0; i < MOD_N; ++i) mod_inverses(MOD_PRIMES[i], inverses[i]);
  return cudaMemcpyToSymbol(c_inverses, inverses, sizeof(inverses));
}

}  // namespace wg
