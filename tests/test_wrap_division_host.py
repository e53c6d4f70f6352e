"""The wrap kernel's division by 2 pi (two corrections with fused
multiply-adds, Markstein 1990) against IEEE division: the same bits, over
magnitudes from 1e-12 to 1e12 and around the multiples of 2 pi where
coordinates wrap."""
import ctypes
import ctypes.util

import numpy as np

TWO_PI = 6.283185307179586


def test_division_by_two_pi_is_correctly_rounded():
    libm = ctypes.CDLL(ctypes.util.find_library("m"))
    libm.fma.restype = ctypes.c_double
    libm.fma.argtypes = [ctypes.c_double] * 3
    fma, inv = libm.fma, 1.0 / TWO_PI
    rng = np.random.default_rng(5)
    x = rng.normal(size=30000) * 10.0 ** rng.uniform(-12, 12, 30000)
    k = rng.integers(-50, 51, 10000) * TWO_PI
    x = np.concatenate([x, k, np.nextafter(k, 1e300), np.nextafter(k, -1e300)])
    for v in x.tolist():
        q = v * inv
        q = fma(fma(-q, TWO_PI, v), inv, q)
        q = fma(fma(-q, TWO_PI, v), inv, q)
        assert q == v / TWO_PI, v
