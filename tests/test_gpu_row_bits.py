"""A single row gives the same bits every time: per-atom calls, fused and
through the batch kernels (Chebyshev and Behler), whose launches share an atom
out over several blocks for few atoms, and neighbour-list calls of one local
atom."""
import numpy as np
import pytest

from tests.test_gpu_behler_pairs import LISTS, _workload

pytestmark = pytest.mark.gpu


def _calls(ann, types, rng, n, precisions):
    from aenet_gb300.core import set_option
    d = rng.normal(size=(n, 3))
    d *= (1.5 + 3.4 * rng.random(n) / np.linalg.norm(d, axis=1))[:, None]
    sym = [types[k] for k in rng.integers(0, len(types), n)]
    idx = np.arange(2, n + 2, dtype=np.int32)
    for path in ("graph", "block", "cluster"):
        set_option("per_atom_kernel", path)
        first = None
        for _ in range(40):
            F = np.zeros((n + 1, 3))
            e = ann.atomic_energy_and_forces(np.zeros(3), types[0], 1, d, sym, idx, F)
            if first is None:
                first = (e, F)
            assert e == first[0] and np.array_equal(F, first[1]), path
    x = np.vstack([np.zeros((1, 3)), d])
    typ = np.array([1] + [types.index(s) + 1 for s in sym], np.int32)
    for prec in precisions:
        first = None
        for _ in range(12):
            r = ann.neighbor_list_energy_forces(x, typ, np.array([0, n]), np.arange(1, n + 1), 1,
                                                precision=prec)
            if first is None:
                first = r
            assert r["energy"] == first["energy"]
            assert np.array_equal(r["forces"], first["forces"])


@pytest.mark.parametrize("n", [30, 150])
@pytest.mark.parametrize("which", ["chebyshev", "chain", "no_grid"])
def test_single_rows_repeat(which, n, tmp_path):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from aenet_gb300 import nnfile, workloads
    from aenet_gb300.core import ANNPotentials, FP64, MIXED, set_option
    rng = np.random.default_rng(n)
    if which == "chebyshev":
        types = ["Au", "Cu"]
        setups = {t: nnfile.chebyshev_setup(t, types, 6.0, 16, 4.0, 8, 1.0) for t in types}
        nsf = setups["Au"]["nsf"]
        w = workloads.Workload("row", types, setups, [nsf, 10, 10, 1], [], 5)
        w.networks = workloads.glorot_networks(rng, types, w.arch)
    else:
        w = _workload(LISTS[which], (30, 34), 3)
        types, nsf = w.types, w.arch[0]
    one = np.ones(nsf)
    stats = {t: (0 * one, 0 * one, 0 * one, 100.0 * one) for t in types}
    ann = ANNPotentials(workloads.write_potentials(w, str(tmp_path), stats=stats),
                        angular_domain="current")
    try:
        _calls(ann, types, rng, n, (FP64, MIXED))
    finally:
        set_option("per_atom_kernel", "fused")
        ann.release()
