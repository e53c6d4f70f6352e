"""The FP64 exponential of the Behler kernels (a table of 2^(k/32), a series
and the exponent's bits), reached by G4 product grids: an atom between two
others one angstrom away, cos = -1, lambda = -1, zeta = 1, so that the atom's
energy is 2 fc(1)^2 fc(2) e^-eta e^-eta e^(-4 eta), the last factor by the
table.  Arguments of the factors are exact, and no constant is added to the
product, so that each value is compared relative to itself."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_table_exponential_by_g4_grids(tmp_path):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from aenet_gb300 import nnfile
    from aenet_gb300.core import ANNPotentials, FP64
    rng = np.random.default_rng(8)
    # a grid holds eight etas at most: 0 and seven more each
    etas = np.concatenate([10.0 ** rng.uniform(-9, 0, 28), rng.uniform(0.0, 116.0, 70),
                           (np.arange(35) + 32 * rng.integers(0, 600, 35)) * np.log(2.0) / 128,
                           [174.9, 175.0, 175.1, 1e3, 1e6, 1e100, 1e300]])
    k = np.rint(-4.0 * etas * 32 / np.log(2.0))
    k = k[(etas < 117) & (etas > 0.05)].astype(int)
    assert set(k & 31) == set(range(32)) and len(set(k >> 5)) > 50
    pos = np.array([[-1.0, 0, 0], [0, 0, 0], [1.0, 0, 0]])
    one = np.ones(8)
    for q in range(0, len(etas), 7):
        es = np.concatenate([[0.0], etas[q:q + 7]])
        setup = nnfile.behler_setup("Ti", ["Ti"], [
            {"G": 4, "type2": "Ti", "type3": "Ti", "Rc": 8.0, "lambda": -1.0, "zeta": 1.0,
             "eta": float(e)} for e in es], 0.5)
        setup.update(sfval_min=0 * one, sfval_max=one, sfval_avg=0 * one, sfval_cov=one)
        path = str(tmp_path / ("Ti%d.nn" % q))
        nnfile.write_nn(path, nnfile.make_network([8, 1], np.zeros(9)), setup,
                        {"scale": 0.5, "shift": 0.0, "typeName": ["Ti"], "E_atom": [0.0]})
        ann = ANNPotentials({"Ti": path}, angular_domain="current")
        got = []
        try:
            for j in range(8):
                W = np.zeros((1, 9))
                W[0, j] = 1.0
                ann.set_weights(W.ravel(order="F"))
                r = ann.structure_energy_forces(pos, np.ones(3, np.int32), None, pbc=False,
                                                precision=FP64)
                got.append(r["atomic_energies"][1])
        finally:
            ann.release()
        got = np.array(got, dtype=np.longdouble)
        assert got[0] > 0
        ref = np.exp(-6 * es.astype(np.longdouble))
        for e, ratio, want in zip(es, got / got[0], ref):
            if 6 * e < 700:
                # two exponentials of the library (an ulp each), the table's
                # (under one) and ten products of half an ulp
                assert abs(ratio / want - 1) <= 8 * 2.3e-16, (e, float(ratio / want - 1))
            else:
                # underflow of the product, whichever way the table's factor takes
                assert 0 <= ratio <= 1e-290, e
