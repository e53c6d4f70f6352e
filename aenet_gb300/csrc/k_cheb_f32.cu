// FP32 instantiations of the Chebyshev descriptor and adjoint kernels with
// the angular terms as pair sums (mixed-precision path) and the launch entry
// points of both precisions.
#include "k_cheb_impl.cuh"
#include "k_cheb_rows.cuh"

int ae_cheb_f64(const PotDevice& pd, const DescBuffers& b, bool adjoint, cudaStream_t s);

namespace {
int cheb_f32(const PotDevice& pd, const DescBuffers& b, bool adjoint, cudaStream_t s) {
  // the moment form where it is instantiated and asked for, pair sums
  // otherwise
  if (b.M && pd.qleg && !b.nb_rank) {
    const int e = cheb::dispatch_moments(pd, b, adjoint, s);
    if (e != cheb::AE_MOM_NA) return e;
  }
  return chebr::dispatch_rows<float>(pd, b, adjoint, true, s);
}
}  // namespace

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
