"""Two neighbours nearly in line with their centre, so that (1 + cos) / 2
rounds to zero in FP32 while the gradient of the cosine does not: the mixed
path's forces across the line against FP64.  With zeta = 1 they come from the
derivative by the cosine, which is one everywhere; higher zetas leave none of
the size compared, and below one the derivative grows without bound (finite
is all that is asked there)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("zetas", [(1.0, 2.0), (4.0, 1.0), (2.5, 1.0), (0.5, 1.0)])
def test_forces_of_neighbours_in_line(zetas, tmp_path):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from aenet_gb300 import nnfile
    from aenet_gb300.core import ANNPotentials, FP64, MIXED
    funcs = [{"G": 5, "type2": "Ti", "type3": "Ti", "Rc": 3.0, "lambda": lam, "zeta": z,
              "eta": eta} for z in zetas for lam in (1.0, -1.0) for eta in (0.01, 0.1)]
    n = len(funcs)
    one = np.ones(n)
    setup = nnfile.behler_setup("Ti", ["Ti"], funcs, 0.5)
    setup.update(sfval_min=0 * one, sfval_max=one, sfval_avg=0 * one, sfval_cov=one)
    path = str(tmp_path / "Ti.nn")
    nnfile.write_nn(path, nnfile.make_network([n, 1], np.zeros(n + 1)), setup,
                    {"scale": 0.5, "shift": 0.0, "typeName": ["Ti"], "E_atom": [0.0]})
    ann = ANNPotentials({"Ti": path}, angular_domain="current")
    try:
        for k, f in enumerate(funcs):
            W = np.zeros(n + 1)
            W[k] = 1.0
            ann.set_weights(W)
            for tilt in (2e-4, 1e-4, 3e-5):
                pos = np.array([[-1.9, 0, 0], [0, 0, 0], [1.9, 1.9 * tilt, 0]])
                F = {p: ann.structure_energy_forces(pos, np.ones(3, np.int32), None, pbc=False,
                                                    precision=p)["forces"][:, 1]
                     for p in (FP64, MIXED)}
                assert np.all(np.isfinite(F[MIXED]))
                if f["lambda"] > 0 and f["zeta"] < 1:
                    continue
                big = np.abs(F[FP64]).max()
                if f["lambda"] > 0 and f["zeta"] == 1:
                    assert big > 0.005 * tilt
                # FP32 rounding of the directions: some 1e-6 of the tilt
                assert np.abs(F[MIXED] - F[FP64]).max() <= 0.01 * max(big, 0.005 * tilt), f
    finally:
        ann.release()
