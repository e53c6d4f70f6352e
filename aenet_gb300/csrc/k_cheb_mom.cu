// Instantiations of the FP32 Chebyshev adjoint with the angular terms in
// moment form (mixed-precision path).
#include "k_cheb_impl.cuh"

namespace cheb {

int dispatch_adjoint_mom(const PotDevice& pd, const DescBuffers& b, cudaStream_t s) {
  int rN, aN;
  if (!uniform_sizes(pd, rN, aN)) return AE_MOM_NA;
  if ((size_t)b.mom_pad < (size_t)(2 * aN * aN)) return AE_MOM_NA;
  if (rN == 11 && aN == 5) return adjoint_mom<11, 5>(pd, b, s);
  if (rN == 13 && aN == 7) return adjoint_mom<13, 7>(pd, b, s);
  if (rN == 17 && aN == 5) return adjoint_mom<17, 5>(pd, b, s);
  return AE_MOM_NA;
}

}  // namespace cheb
