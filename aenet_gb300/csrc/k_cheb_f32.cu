// FP32 instantiations of the Chebyshev descriptor and adjoint kernels (the
// mixed-precision path; the adjoint in moment form is k_cheb_mom.cu's) and the
// launch entry points of both precisions.
#include "k_cheb_impl.cuh"
#include "k_cheb_rows.cuh"

int ae_cheb_f64(const PotDevice& pd, const DescBuffers& b, bool adjoint, cudaStream_t s);
bool ae_cheb_moments_f64(const PotDevice& pd);

namespace {
int cheb_f32(const PotDevice& pd, const DescBuffers& b, bool adjoint, cudaStream_t s) {
  // the adjoint in moment form where the forward left moments
  if (adjoint && chebr::moment_form<float>(pd, b)) return cheb::dispatch_adjoint_mom(pd, b, s);
  return chebr::dispatch_rows<float>(pd, b, adjoint, s);
}
}  // namespace

bool ae_cheb_moments(const PotDevice& pd, int fp64) {
  return fp64 ? ae_cheb_moments_f64(pd) : chebr::moment_sizes<float>(chebr::sizes(pd));
}

int ae_launch_chebyshev_forward(const PotDevice& pd, const DescBuffers& b, int fp64,
                                cudaStream_t s) {
  if (b.natoms <= 0) return 0;
  return fp64 ? ae_cheb_f64(pd, b, false, s) : cheb_f32(pd, b, false, s);
}

int ae_launch_chebyshev_adjoint(const PotDevice& pd, const DescBuffers& b, int fp64,
                                cudaStream_t s) {
  if (b.natoms <= 0) return 0;
  return fp64 ? ae_cheb_f64(pd, b, true, s) : cheb_f32(pd, b, true, s);
}
