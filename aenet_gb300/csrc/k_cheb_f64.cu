// FP64 Chebyshev descriptor and adjoint kernels: launch entry points.  Exact
// instantiations for the common (radial, angular) sizes and spins within
// -1 .. 1 (up to three species), guarded ones for everything else.
#include "k_cheb64.cuh"

int ae_cheb_f64(const PotDevice& pd, const DescBuffers& b, bool adjoint, cudaStream_t s) {
  using namespace cheb64;
  int rN = 0, aN = 0, spin = SPIN_NONE;
  bool same = true;
  for (int t = 0; t < pd.ntypes; ++t) {
    const ChebTable& ct = pd.sp[t].cheb;
    if (t > 0 && (ct.r_N != rN || ct.a_N != aN)) same = false;
    rN = max(rN, ct.r_N);
    aN = max(aN, ct.a_N);
    if (!ct.multi) continue;
    spin = max(spin, (int)SPIN_UNIT);
    for (int q = 0; q < pd.ntypes; ++q)
      if (ct.spin[q] < -1.f || ct.spin[q] > 1.f) spin = SPIN_ANY;
  }
  if (same && spin != SPIN_ANY && !b.nb_rank) {
    const bool mom = b.M64 && pd.qleg64 && b.mom_pad >= 2 * aN * aN;
    if (rN == 11 && aN == 5)
      return mom ? launch_spin<11, 5, true>(pd, b, spin, adjoint, s)
                 : launch_spin<11, 5, false>(pd, b, spin, adjoint, s);
    if (rN == 17 && aN == 5)
      return mom ? launch_spin<17, 5, true>(pd, b, spin, adjoint, s)
                 : launch_spin<17, 5, false>(pd, b, spin, adjoint, s);
    if (rN == 13 && aN == 7) return launch_spin<13, 7, false>(pd, b, spin, adjoint, s);
    if (rN == 17 && aN == 9) return launch_spin<17, 9, false>(pd, b, spin, adjoint, s);
  }
  if (rN <= 24 && aN <= 16) return launch<24, 16, true, SPIN_ANY, false>(pd, b, adjoint, s);
  if (rN <= 32 && aN <= 32) return launch<32, 32, true, SPIN_ANY, false>(pd, b, adjoint, s);
  return (int)cudaErrorInvalidValue;
}
