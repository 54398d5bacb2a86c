// Near field with a complex wavenumber (near.cuh).
#include "near.cuh"

namespace bem2d_gpu {

int launch_near_ck(const DevGeom& g, const DevRules& r, const NearPair* pairs, int npairs, int nb,
                   int kernel, double k, double ki, double eta, double alpha, double beta,
                   double2* out, long long ld, cudaStream_t s) {
  if (npairs == 0) return BEM2D_OK;
  if (nb > 1)
    launch_near_m<false, true, kNearBasis>(g, r, pairs, npairs, kernel, k, ki, eta, alpha, beta,
                                           nullptr, out, ld, nullptr, 0, s);
  else
    launch_near_m<false, true, 1>(g, r, pairs, npairs, kernel, k, ki, eta, alpha, beta, nullptr,
                                  out, ld, nullptr, 0, s);
  return BEM2D_OK;
}

}  // namespace bem2d_gpu
