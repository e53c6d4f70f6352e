// The cosine cut-off fc = (1 + cos sqrt(y)) / 2, y = (pi r / Rc)^2, as an FP64
// series in y.  cos sqrt(y) is an entire function of y; its Taylor series
// about pi^2/2 to degree 13 leaves less than 1e-18 on [0, pi^2] (the terms
// stay below one, so that the rounding is that of the value itself) and
// needs no square root, no sine and no division.  The FP64 pipe (two lanes
// per clock and SM) bounds the kernels that use it: 14 multiply-adds for fc
// and 13 for its derivative stand for about 60 instructions of r, sin and
// cos.
#pragma once

constexpr double FC_Y0 = 4.9348022005446793094;   // pi^2 / 2

// fc at z = y - pi^2/2
__device__ __forceinline__ double fc_series(double z) {
  double p = -1.1311932861159658242e-27;
  p = fma(p, z, 7.2986588589149819688e-25);
  p = fma(p, z, -3.9940266677874554912e-22);
  p = fma(p, z, 1.8262231133604611914e-19);
  p = fma(p, z, -6.8529250117771331873e-17);
  p = fma(p, z, 2.0645516741852144221e-14);
  p = fma(p, z, -4.8575286692910524617e-12);
  p = fma(p, z, 8.612487525263789767e-10);
  p = fma(p, z, -1.0965771688152239754e-7);
  p = fma(p, z, 9.3591834506349915894e-6);
  p = fma(p, z, -0.00048082314182966815651);
  p = fma(p, z, 0.012207779738690289425);
  p = fma(p, z, -0.089546946503311004436);
  return fma(p, z, 0.1971500664605932856);
}
// d fc / dy
__device__ __forceinline__ double fc_series_d(double z) {
  double p = -13.0 * 1.1311932861159658242e-27;
  p = fma(p, z, 12.0 * 7.2986588589149819688e-25);
  p = fma(p, z, -11.0 * 3.9940266677874554912e-22);
  p = fma(p, z, 10.0 * 1.8262231133604611914e-19);
  p = fma(p, z, -9.0 * 6.8529250117771331873e-17);
  p = fma(p, z, 8.0 * 2.0645516741852144221e-14);
  p = fma(p, z, -7.0 * 4.8575286692910524617e-12);
  p = fma(p, z, 6.0 * 8.612487525263789767e-10);
  p = fma(p, z, -5.0 * 1.0965771688152239754e-7);
  p = fma(p, z, 4.0 * 9.3591834506349915894e-6);
  p = fma(p, z, -3.0 * 0.00048082314182966815651);
  p = fma(p, z, 2.0 * 0.012207779738690289425);
  return fma(p, z, -0.089546946503311004436);
}
