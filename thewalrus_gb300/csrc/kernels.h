// Sieve-kernel instantiations live in one translation unit per scalar class (kernels_c64.cu,
// kernels_cdf.cu, kernels_f64.cu, kernels_fdf.cu, kernels_cdd.cu, kernels_fdd.cu,
// kernels_mod{0..4}.cu: residues modulo one prime each) so that they compile in parallel.  Each unit
// instantiates sieve_kernel<S> and the tree kernel (the residues' is kernels_mods.cu, for all primes) and
// holds its own copy of the constant tables (binomials, reciprocals), which the host fills through
// sieve_tables_*.
#pragma once
#include <cuda_runtime.h>

#include <atomic>

#include "sieve_kernel.cuh"
#include "tree_kernel.cuh"

namespace wg {

#define WG_KERNEL_UNIT_DECL(T)                                                                      \
  cudaError_t sieve_launch_##T(const SieveParams& p, int ctas, int wpc, cudaStream_t st); \
  int sieve_occupancy_##T(int wpc, int smem);                                             \
  cudaError_t sieve_tables_##T(const double* binom, const double* inv);

WG_KERNEL_UNIT_DECL(c64)
WG_KERNEL_UNIT_DECL(cdf)
WG_KERNEL_UNIT_DECL(f64)
WG_KERNEL_UNIT_DECL(fdf)
WG_KERNEL_UNIT_DECL(cdd)
WG_KERNEL_UNIT_DECL(fdd)
WG_KERNEL_UNIT_DECL(mod0)
WG_KERNEL_UNIT_DECL(mod1)
WG_KERNEL_UNIT_DECL(mod2)
WG_KERNEL_UNIT_DECL(mod3)
WG_KERNEL_UNIT_DECL(mod4)
#undef WG_KERNEL_UNIT_DECL
#define WG_TREE_UNIT_DECL(T) \
  cudaError_t tree_launch_##T(const TreeParams& p, bool parts, int ctas, int smem, cudaStream_t st);
WG_TREE_UNIT_DECL(c64)
WG_TREE_UNIT_DECL(cdf)
WG_TREE_UNIT_DECL(f64)
WG_TREE_UNIT_DECL(fdf)
WG_TREE_UNIT_DECL(cdd)
WG_TREE_UNIT_DECL(fdd)
#undef WG_TREE_UNIT_DECL
cudaError_t tree_launch_mods(const TreeMods& m, int ctas, int smem, cudaStream_t st);
cudaError_t sieve_tables_mods(const double* binom, const double* inv);

// Lets a kernel's launches on the current device ask for all the dynamic shared memory there is beside
// its static part.  Once and always the same: launches of several threads, each with its own size, would
// otherwise lower it for one another between setting it and launching.
template <auto K>
static inline cudaError_t allow_shared() {
  static std::atomic<unsigned long long> done{0};  // a bit per device
  int dev = 0, most = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || (dev < 64 && (done.load() >> dev & 1))) return e;
  cudaFuncAttributes a;
  e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, K);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, most - (int)a.sharedSizeBytes);
  if (e == cudaSuccess && dev < 64) done |= 1ull << dev;
  return e;
}

// A launch of `ctas` CTAs whose trees are shared by `group` of them: these wait for one another, so
// that more than one are launched cooperatively.
template <auto K, class Params>
static inline cudaError_t tree_launch_kernel(const Params& p, int ctas, int group, int smem, cudaStream_t st) {
  const cudaError_t e = allow_shared<K>();
  if (e != cudaSuccess) return e;
  if (group == 1) {
    K<<<ctas, TREE_THREADS, smem, st>>>(p);
    return cudaGetLastError();
  }
  Params arg = p;
  void* args[] = {&arg};
  return cudaLaunchCooperativeKernel((const void*)K, dim3(ctas), dim3(TREE_THREADS), args, (size_t)smem, st);
}

// 1/k modulo a prime in Montgomery form, k < 256, by k * inv(k) = 1: inv(k) = -(p / k) inv(p mod k)
static inline void mod_inverses(uint64_t p, uint32_t* inv) {
  uint32_t plain[256] = {0, 1};
  for (uint64_t k = 2; k < 256; ++k) plain[k] = (uint32_t)((p - (p / k) * plain[p % k] % p) % p);
  for (int k = 0; k < 256; ++k) inv[k] = (uint32_t)(((uint64_t)plain[k] << 32) % p);
}

}  // namespace wg
