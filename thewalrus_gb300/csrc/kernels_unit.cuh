// Body of one kernel translation unit: define WG_UNIT_SCALAR (the scalar type), WG_UNIT_NAME (the
// suffix of the entry points) and, for the residue types, WG_UNIT_PRIME, then include this file.
#include "kernels.h"

namespace wg {

#define WG_CAT2(a, b) a##b
#define WG_CAT(a, b) WG_CAT2(a, b)

cudaError_t WG_CAT(sieve_launch_, WG_UNIT_NAME)(const SieveParams& p, int ctas, int wpc, cudaStream_t st) {
  const cudaError_t e = allow_shared<sieve_kernel<WG_UNIT_SCALAR>>();
  if (e != cudaSuccess) return e;
  sieve_kernel<WG_UNIT_SCALAR><<<ctas, 32 * wpc, wpc * p.L.bytes, st>>>(p);
  return cudaGetLastError();
}

int WG_CAT(sieve_occupancy_, WG_UNIT_NAME)(int wpc, int smem) {
  int nb = 0;
  if (allow_shared<sieve_kernel<WG_UNIT_SCALAR>>() != cudaSuccess) return 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, sieve_kernel<WG_UNIT_SCALAR>, 32 * wpc, smem) != cudaSuccess)
    return 0;
  return nb;
}

#ifndef WG_UNIT_PRIME  // (residues: kernels_mods.cu)
cudaError_t WG_CAT(tree_launch_, WG_UNIT_NAME)(const TreeParams& p, bool parts, int ctas, int smem, cudaStream_t st) {
  if (parts) return tree_launch_kernel<tree_kernel<WG_UNIT_SCALAR>>(p, ctas, ctas, smem, st);
  return tree_launch_kernel<tree_kernel<typename TreeScalar<WG_UNIT_SCALAR>::T>>(p, ctas, ctas, smem, st);
}
#endif

cudaError_t WG_CAT(sieve_tables_, WG_UNIT_NAME)(const double* binom, const double* inv) {
  cudaError_t e = cudaMemcpyToSymbol(c_binom, binom, sizeof(c_binom));
  if (e != cudaSuccess) return e;
  e = cudaMemcpyToSymbol(c_inv, inv, sizeof(c_inv));
#ifdef WG_UNIT_PRIME
  if (e != cudaSuccess) return e;
  uint32_t invmod[256];
  mod_inverses(WG_UNIT_PRIME, invmod);
  e = cudaMemcpyToSymbol(c_invmod, invmod, sizeof(invmod));
#endif
  return e;
}

#undef WG_CAT
#undef WG_CAT2

}  // namespace wg
