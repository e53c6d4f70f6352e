"""The one-launch per-atom kernels (one block, and a cluster) against the graph
of the batch kernels (1e-10 eV, 1e-9 eV/A): one species and two, the smallest
and largest orders of both instantiations, layers from one node to sixty-four
with every activation, rows around the staging passes and pair rounds,
neighbours on and beyond the cut-offs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

E_TOL, F_TOL = 1e-10, 1e-9


@pytest.mark.parametrize("types,r_order,a_order,arch,act", [
    (["Cu"], 16, 8, [1, 1], [1, 1, 0]),
    (["Cu"], 1, 1, [64], [3, 0]),
    (["Cu"], 23, 15, [20, 20], [1, 1, 0]),
    (["Cu"], 16, 8, [33, 7, 2], [4, 2, 1, 3]),
    (["Cu", "Au"], 16, 8, [20, 20], [1, 1, 0]),
    (["Cu", "Au"], 17, 2, [9], [0, 0]),
    (["Cu", "Au"], 2, 9, [64, 64], [1, 1, 0]),
])
@pytest.mark.parametrize("angular", ["current", "legacy"])
def test_per_atom_kernels_against_graph(types, r_order, a_order, arch, act, angular, tmp_path):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from aenet_gb300 import nnfile, workloads
    from aenet_gb300.core import ANNPotentials, set_option
    rng = np.random.default_rng(r_order + a_order + len(arch))
    r_Rc, a_Rc = 6.0, 4.0
    setups = {t: nnfile.chebyshev_setup(t, types, r_Rc, r_order, a_Rc, a_order, 1.0) for t in types}
    nsf = setups[types[0]]["nsf"]
    arch = [nsf] + arch + [1]
    w = workloads.Workload("edges", types, setups, arch, [], 5)
    w.networks = workloads.glorot_networks(rng, types, arch)
    for t in types:
        w.networks[t]["f_a"] = np.array(act)
    one = np.ones(nsf)
    stats = {t: (0 * one, 0 * one, 0 * one, 100.0 * one) for t in types}
    ann = ANNPotentials(workloads.write_potentials(w, str(tmp_path), stats=stats),
                        angular_domain=angular)
    centre = np.array([0.3, -1.0, 2.0])
    try:
        for n in (0, 1, 2, 3, 18, 19, 40, 95, 96, 97, 129, 200):
            d = rng.normal(size=(n, 3))
            d /= np.maximum(np.linalg.norm(d, axis=1), 1e-9)[:, None]
            length = 1.2 + 5.2 * rng.random(n) ** 0.6
            length[3:6] = [r_Rc, a_Rc, 40.0][:max(0, min(3, n - 3))]
            coo = centre + d * length[:, None]
            sym = [types[k] for k in rng.integers(0, len(types), n)]
            idx = np.arange(2, n + 2, dtype=np.int32)
            got = {}
            for path in ("graph", "block", "cluster"):
                set_option("per_atom_kernel", path)
                F = np.zeros((n + 1, 3))
                e = ann.atomic_energy_and_forces(centre, types[-1], 1, coo, sym, idx, F)
                assert abs(ann.atomic_energy(centre, types[-1], coo, sym) - e) <= E_TOL
                got[path] = (e, F)
            for path in ("block", "cluster"):
                assert abs(got[path][0] - got["graph"][0]) <= E_TOL * max(1.0, abs(e)), (path, n)
                big = max(1.0, np.abs(got["graph"][1]).max())
                assert np.abs(got[path][1] - got["graph"][1]).max() <= F_TOL * big, (path, n)
    finally:
        set_option("per_atom_kernel", "fused")
        ann.release()
