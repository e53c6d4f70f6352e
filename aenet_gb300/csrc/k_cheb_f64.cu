// FP64 instantiations of the Chebyshev descriptor and adjoint kernels (the
// plain path).
#include "k_cheb_rows.cuh"

int ae_cheb_f64(const PotDevice& pd, const DescBuffers& b, bool adjoint, cudaStream_t s) {
  return chebr::dispatch_rows<double>(pd, b, adjoint, s);
}

bool ae_cheb_moments_f64(const PotDevice& pd) {
  return chebr::moment_sizes<double>(chebr::sizes(pd));
}
