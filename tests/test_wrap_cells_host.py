"""The wrap kernel's integer forms: a small integer as a double by its bits,
and floor(x) as the low word of x + 2^52 rounded down, against the plain
expressions."""
import ctypes
import ctypes.util
import struct

import numpy as np

FE_DOWNWARD = {"x86_64": 0x400, "aarch64": 0x800000}
FE_TONEAREST = 0


def test_small_integers_by_bits():
    for n in list(range(1, 1025)) + [4095, 65537, (1 << 20) - 1]:
        e = n.bit_length() - 1
        hi = ((1023 + e) << 20) | ((n << (20 - e)) & 0xFFFFF)
        assert struct.unpack("<d", struct.pack("<II", 0, hi))[0] == float(n)


def test_floor_by_rounding_down():
    import platform
    import pytest
    down = FE_DOWNWARD.get(platform.machine())
    if down is None:
        pytest.skip("unknown machine")
    libm = ctypes.CDLL(ctypes.util.find_library("m"))
    rng = np.random.default_rng(4)
    nc = rng.integers(1, 1024, 20000)
    s = rng.random(20000)
    k = rng.integers(0, 1024, 20000)
    edge = np.minimum(k / nc, 1.0)
    x = np.concatenate([s * nc, edge * nc, np.nextafter(edge, 0) * nc, [0.0, 5e-324, 1.0, 1023.0]])
    want = np.floor(x)
    assert libm.fesetround(down) == 0
    try:
        got = [v + 4503599627370496.0 for v in x.tolist()]
    finally:
        libm.fesetround(FE_TONEAREST)
    low = [struct.unpack("<II", struct.pack("<d", v))[0] for v in got]
    assert np.array_equal(low, want)
