"""The pair schedule and power forms of the Behler kernels where they can go
wrong: buckets of one, two, an odd or an even number of neighbours and below
or above 32 of them, signs of lambda without an entry, odd numbers of etas,
zetas that are chains of squarings, too many for one pass or not integers,
G5 without the r_jk cut, and angular lists that form no product grid.  FP64
against the oracle at the suite's tolerances (1e-10 eV/atom, 1e-9 eV/A), the
mixed path against FP64 at 1 meV/atom and 20 meV/A RMS."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RC = 5.0
LISTS = {
    "chain": [(4, z, lam, e) for z in (1, 4, 16) for lam in (1, -1) for e in (0.01, 0.1)],
    "one_sign_three_etas": [(4, z, 1, e) for z in (2, 4) for e in (0.01, 0.05, 0.2)],
    "five_zetas": [(4, z, lam, 0.02) for z in (1, 2, 4, 8, 16) for lam in (1, -1)],
    "real_zetas": [(4, z, lam, 0.02) for z in (1, 2.5, 3) for lam in (1, -1)],
    "g5": [(5, z, lam, e) for z in (1, 2) for lam in (1, -1) for e in (0.01, 0.1)],
    "no_grid": [(4, 1, 1, 0.01), (4, 2, -1, 0.05), (5, 4, 1, 0.02)],
}


def _workload(entries, counts, seed):
    from aenet_gb300 import nnfile, workloads
    rng = np.random.default_rng(seed)
    types = ["Ti", "O"]
    n = sum(counts)
    # jittered sites of a cubic grid, 2.1 A apart: up to ~55 neighbours
    m = int(np.ceil(n ** (1 / 3)))
    site = rng.permutation(m ** 3)[:n]
    pos = np.stack([site // (m * m), site // m % m, site % m], -1) * 2.1
    pos = pos + rng.uniform(-0.25, 0.25, pos.shape)
    typ = np.repeat(np.array([1, 2], dtype=np.int32), counts)[rng.permutation(n)]
    cell = np.eye(3) * (m * 2.1)
    funcs = []
    for t in types:
        for eta in (0.02, 0.3):
            funcs.append({"G": 2, "type2": t, "Rc": RC, "Rs": 0.5, "eta": eta})
    for i, a in enumerate(types):
        for b in types[i:]:
            for kind, zeta, lam, eta in entries:
                funcs.append({"G": kind, "type2": a, "type3": b, "Rc": RC, "lambda": float(lam),
                              "zeta": float(zeta), "eta": eta})
    setups = {t: nnfile.behler_setup(t, types, funcs, 1.0) for t in types}
    w = workloads.Workload("behler_pairs", types, setups, [len(funcs), 10, 10, 1],
                           [workloads.Structure(pos, typ, cell)], seed)
    w.networks = workloads.glorot_networks(rng, types, w.arch)
    return w


# species counts: whole lists of one and two neighbours, a rare species,
# odd and even buckets on both sides of 32
@pytest.mark.parametrize("counts", [(1, 2), (3, 24), (30, 34), (62, 2)])
@pytest.mark.parametrize("which", sorted(LISTS))
def test_behler_pair_lists_match_oracle(oracle, tmp_path, which, counts):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from aenet_gb300 import workloads
    from aenet_gb300.core import ANNPotentials, FP64, MIXED
    w = _workload(LISTS[which], counts, 7 + len(which))
    s = w.structures[0]
    # fixed statistics (mean 0, deviation 10): three atoms give none
    nsf = w.arch[0]
    stats = {t: (np.zeros(nsf), np.zeros(nsf), np.zeros(nsf), np.full(nsf, 100.0))
             for t in w.types}
    paths = workloads.write_potentials(w, str(tmp_path), stats=stats)
    ann = ANNPotentials({t: paths[t] for t in w.types}, angular_domain="current")
    try:
        r64 = ann.structure_energy_forces(s.positions, s.types, s.cell, precision=FP64)
        r32 = ann.structure_energy_forces(s.positions, s.types, s.cell, precision=MIXED)
    finally:
        ann.release()
    oracle.load(w.types, paths)
    _, et, F, Ea = oracle.structure(s.cell, s.positions, s.types)
    scale = max(1.0, np.abs(F).max())
    assert np.abs(r64["atomic_energies"] - Ea).max() < 1e-10 * scale
    assert np.abs(r64["forces"] - F).max() < 1e-9 * scale
    assert abs(r32["energy"] - r64["energy"]) / s.natoms < 1e-3
    assert np.sqrt(np.mean((r32["forces"] - r64["forces"]) ** 2)) < 2e-2 * scale
