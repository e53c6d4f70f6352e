"""The FP64 networks: tanh without branches against libm's over its whole
range (a network whose energy is tanh of a bias), and layers narrower, wider
and deeper than a warp, different per species, for few and many atoms, against
the oracle (1e-10 eV/atom, 1e-9 eV/A)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _torch():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    return torch


def _cell(rng, n_types):
    from aenet_gb300 import workloads
    pos, cell = workloads.fcc_positions(2, 4.0)
    pos = pos + rng.normal(0, 0.15, pos.shape)
    typ = (np.arange(len(pos)) % n_types + 1).astype(np.int32)
    return workloads.Structure(pos, typ, cell)


def test_fp64_tanh_is_accurate(tmp_path):
    _torch()
    from aenet_gb300 import nnfile, workloads
    from aenet_gb300.core import ANNPotentials, FP64
    rng = np.random.default_rng(2)
    setup = nnfile.chebyshev_setup("Cu", ["Cu"], 4.0, 2, 3.0, 1, 1.0)
    nsf = setup["nsf"]
    one = np.ones(nsf)
    setup.update(sfval_min=0 * one, sfval_max=one, sfval_avg=0 * one, sfval_cov=one)
    # E = 2 tanh(bias): one hidden node with zero weights, no shift, no E_atom
    net = nnfile.make_network([nsf, 1, 1], np.zeros((nsf + 1) + 2))
    path = str(tmp_path / "Cu.nn")
    nnfile.write_nn(path, net, setup, {"scale": 0.5, "shift": 0.0, "typeName": ["Cu"],
                                       "E_atom": [0.0]})
    x = np.concatenate([10.0 ** rng.uniform(-18, 1.5, 300), rng.uniform(0, 3, 200),
                        [0.0, 0.17328, 0.3466, 0.34658, 0.55, 18.9, 19.1, 22.0, 22.5, 1e3, 1e300]])
    x = np.concatenate([x, -x])
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
    got, ref = np.array(got), np.tanh(x)
    # one rounding in each of: the reduced argument, the series, m, m + 2, the
    # quotient -- 4 ulp with libm's own
    assert np.all(np.abs(got - ref) <= 4 * np.spacing(np.abs(ref)))
    assert np.all(np.sign(got) == np.sign(x))


@pytest.mark.parametrize("reps", [1, 160])
@pytest.mark.parametrize("archs", [((20, 20),), ((25, 7), (40, 33)), ((64,), (3, 5, 4)),
                                   ((), (12, 12))])
def test_fp64_network_shapes_match_oracle(oracle, tmp_path, archs, reps):
    _torch()
    from aenet_gb300 import nnfile, workloads
    from aenet_gb300.core import ANNPotentials, FP64
    rng = np.random.default_rng(len(archs[0]) + 3)
    types = ["Li", "Si"][:len(archs)]
    s = _cell(rng, len(types))
    setups, nets = {}, {}
    for t, hidden in zip(types, archs):
        st = nnfile.chebyshev_setup(t, types, 4.5, 6, 3.5, 3, 1.0)
        n = st["nsf"]
        st.update(sfval_min=np.zeros(n), sfval_max=np.zeros(n), sfval_avg=np.zeros(n),
                  sfval_cov=np.full(n, 30.0))
        setups[t] = st
        arch = [n, *hidden, 1]
        size = sum((a + 1) * b for a, b in zip(arch, arch[1:]))
        nets[t] = nnfile.make_network(arch, rng.uniform(-0.4, 0.4, size))
    paths = {}
    for t in types:
        paths[t] = str(tmp_path / (t + ".nn"))
        nnfile.write_nn(paths[t], nets[t], setups[t],
                        {"scale": 0.5, "shift": -1.0, "typeName": types,
                         "E_atom": [-1.0] * len(types)})
    ann = ANNPotentials(paths, angular_domain="current")
    try:
        r = ann.batch_energy_forces([(s.positions, s.types, s.cell, True)] * reps, precision=FP64)
    finally:
        ann.release()
    oracle.load(types, paths)
    _, et, F, _ = oracle.structure(s.cell, s.positions, s.types)
    assert np.abs(r["energy"] - et).max() / s.natoms < 1e-10
    assert np.abs(r["forces"].reshape(reps, -1, 3) - F).max() < 1e-9
