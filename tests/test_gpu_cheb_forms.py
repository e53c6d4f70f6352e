"""The Chebyshev kernels of both precisions over the forms that they accept: exact and
guarded orders, one species, spins within -1 .. 1 (three species) and beyond
(five), both angular domains, the pair and the moment form of the angular
terms, rows with none, one, two and more angular neighbours than lanes, and
both widths (a warp per atom for few atoms, four atoms per warp for many).
Against the oracle at the suite's tolerances (1e-10 eV/atom, 1e-9 eV/A)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TYPES = ["Li", "Si", "O", "Ti", "Cu"]


def _workload(ntypes, orders, seed):
    from aenet_gb300 import nnfile, workloads
    rng = np.random.default_rng(seed)
    types = TYPES[:ntypes]
    # a dense half (beside up to ~60 angular neighbours) and a dilute one
    # (atoms with no, one or two angular neighbours)
    m = 4
    g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)
    dense = g * 1.75 + rng.uniform(-0.2, 0.2, g.shape)
    thin = np.array([[11.0, 1.0, 1.0], [14.0, 5.0, 3.0], [14.6, 6.9, 3.4], [18.0, 2.0, 6.0],
                     [18.2, 4.1, 6.3], [19.9, 3.0, 5.2]]) + rng.uniform(-0.1, 0.1, (6, 3))
    pos = np.concatenate([dense, thin])
    typ = rng.integers(1, ntypes + 1, len(pos)).astype(np.int32)
    typ[:ntypes] = np.arange(1, ntypes + 1)
    cell = np.diag([24.0, 9.0, 9.0])
    ro, ao = orders
    setups = {t: nnfile.chebyshev_setup(t, types, 5.0, ro, 3.4, ao, 0.8) for t in types}
    nsf = setups[types[0]]["nsf"]
    w = workloads.Workload("cheb64", types, setups, [nsf, 8, 8, 1],
                           [workloads.Structure(pos, typ, cell)], seed)
    w.networks = workloads.glorot_networks(rng, types, w.arch)
    return w


@pytest.mark.parametrize("domain", ["current", "legacy"])
@pytest.mark.parametrize("ntypes", [1, 3, 5])
@pytest.mark.parametrize("orders", [(10, 4), (16, 4), (12, 6), (16, 8), (7, 3), (25, 17)])
def test_chebyshev_forms_match_oracle(oracle, tmp_path, orders, ntypes, domain):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from aenet_gb300 import workloads
    from aenet_gb300.core import ANNPotentials, FP64, MIXED, set_option
    w = _workload(ntypes, orders, 3 + ntypes)
    s = w.structures[0]
    nsf = w.arch[0]
    stats = {t: (np.zeros(nsf), np.zeros(nsf), np.zeros(nsf), np.full(nsf, 400.0))
             for t in w.types}
    paths = workloads.write_potentials(w, str(tmp_path), stats=stats)
    ann = ANNPotentials({t: paths[t] for t in w.types}, angular_domain=domain)
    got = {}
    try:
        one = (s.positions, s.types, s.cell, True)
        # enough atoms for two and for four per warp
        many = [1300 // s.natoms + 1, 3100 // s.natoms + 1]
        for terms in ("moments", "pairs"):
            set_option("angular_terms", terms)
            got[terms] = ann.structure_energy_forces(*one[:3], precision=FP64, virial=True)
            got[terms + "8"] = [ann.batch_energy_forces([one] * r, precision=FP64, virial=True)
                                for r in many]
            got[terms + "32"] = [ann.batch_energy_forces([one] * r, precision=MIXED, virial=True)
                                 for r in [1] + many]
    finally:
        set_option("angular_terms", "moments")
        set_option("angular_domain", "current")
        ann.release()
    oracle.load(w.types, paths, angular=domain)
    _, et, F, Ea = oracle.structure(s.cell, s.positions, s.types)
    scale = max(1.0, np.abs(F).max())
    for terms in ("moments", "pairs"):
        r = got[terms]
        assert np.abs(r["atomic_energies"] - Ea).max() < 1e-10 * scale
        assert np.abs(r["forces"] - F).max() < 1e-9 * scale
        for r8 in got[terms + "8"]:
            assert np.abs(r8["energy"] - et).max() / s.natoms < 1e-10 * scale
            assert np.abs(r8["forces"].reshape(-1, s.natoms, 3) - F).max() < 1e-9 * scale
            assert np.abs(r8["virial"] - r["virial"]).max() < 1e-8 * scale
        # FP32: the mixed path's contract (1 meV/atom, 20 meV/A RMS)
        for r32 in got[terms + "32"]:
            assert np.abs(r32["energy"] - et).max() / s.natoms < 1e-3
            dF = r32["forces"].reshape(-1, s.natoms, 3) - F
            assert np.sqrt(np.mean(dF ** 2)) < 2e-2
            assert np.abs(r32["virial"] - r["virial"]).max() < 1e-3 * scale * s.natoms
    assert np.abs(got["moments"]["virial"] - got["pairs"]["virial"]).max() < 1e-8 * scale
