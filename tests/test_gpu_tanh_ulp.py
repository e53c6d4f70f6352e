"""The FP64 tanh of the networks against the extended-precision value, in units
in the last place, over the arguments where its parts round worst (a network
whose energy is tanh of a bias)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_tanh_within_one_and_a_half_ulp(tmp_path):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from aenet_gb300 import nnfile
    from aenet_gb300.core import ANNPotentials, FP64
    if np.finfo(np.longdouble).eps > 2e-19:
        pytest.skip("no extended precision")
    rng = np.random.default_rng(14)
    setup = nnfile.chebyshev_setup("Cu", ["Cu"], 4.0, 2, 3.0, 1, 1.0)
    nsf = setup["nsf"]
    one = np.ones(nsf)
    setup.update(sfval_min=0 * one, sfval_max=one, sfval_avg=0 * one, sfval_cov=one)
    path = str(tmp_path / "Cu.nn")
    nnfile.write_nn(path, nnfile.make_network([nsf, 1, 1], np.zeros((nsf + 1) + 2)), setup,
                    {"scale": 0.5, "shift": 0.0, "typeName": ["Cu"], "E_atom": [0.0]})
    x = np.concatenate([rng.uniform(0.1, 0.36, 3000), rng.uniform(0.36, 2.0, 1500),
                        rng.uniform(2.0, 23.0, 500), 10.0 ** rng.uniform(-300, -1, 300),
                        [0.0, 5e-324, 22.0, 1e300]])
    ann = ANNPotentials({"Cu": path}, angular_domain="current")
    got = []
    try:
        for v in x:
            W = np.zeros(nsf + 3)
            W[nsf], W[nsf + 1] = v, 1.0
            ann.set_weights(W)
            got.append(ann.structure_energy_forces(np.zeros((1, 3)), np.array([1]), None, pbc=False,
                                                   precision=FP64)["energy"] / 2.0)
    finally:
        ann.release()
    ref = np.tanh(x.astype(np.longdouble))
    # half a unit each from the last rounding and the rounding of the reduced
    # argument, 0.36 from the series' truncation, and second-order terms
    err = np.abs(np.array(got).astype(np.longdouble) - ref) / np.spacing(ref.astype(np.float64))
    assert float(err.max()) <= 1.5, (x[int(err.argmax())], float(err.max()))
