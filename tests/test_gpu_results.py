"""The launch that writes a pass's results: energies summed beside the force
output (a warp per structure, or blocks per chunk) against the sums of a
forward pass (the same order: the same bits), the atoms' energies and forces
with and without the other outputs, and atoms grouped by species beside the
search over all pairs up to and beyond its limit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[1], [255], [256], [257], [2048], [2049], [5000], [3] * 9,
                                   [2049, 1, 40], [500] * 8, [600] * 7])
def test_results_against_forward(sizes, tmp_path):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from aenet_gb300 import nnfile, workloads
    from aenet_gb300.core import ANNPotentials, FP64, MIXED
    from aenet_gb300.plan import Plan
    rng = np.random.default_rng(len(sizes) + sizes[0])
    types = ["Li", "Si", "O"]
    setups = {t: nnfile.chebyshev_setup(t, types, 4.0, 4, 3.4, 2, 1.0) for t in types}
    w = workloads.Workload("results", types, setups, [16, 8, 8, 1], [], 5)
    w.networks = workloads.glorot_networks(rng, types, w.arch)
    stats = {t: (np.zeros(16), np.zeros(16), np.zeros(16), np.full(16, 25.0)) for t in types}
    ann = ANNPotentials(workloads.write_potentials(w, str(tmp_path), stats=stats),
                        angular_domain="current")
    pos, cells = [], []
    for n in sizes:
        m = max(3, int(np.ceil(n ** (1 / 3) - 1e-9)))
        g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
        pos.append((g + rng.uniform(-0.15, 0.15, g.shape)) * 2.8)
        cells.append(np.eye(3) * (2.8 * m))
    n = sum(sizes)
    p = torch.tensor(np.concatenate(pos), device="cuda")
    t = torch.tensor(rng.integers(1, 4, n).astype(np.int32), device="cuda")
    try:
        for prec in (FP64, MIXED):
            plan = Plan(sizes, np.array(cells), np.ones(len(sizes), np.int32), precision=prec)
            Ea = torch.empty(n, dtype=torch.float64, device="cuda")
            E = plan.forward(p, t, E_atoms=Ea).clone()
            full = plan.run(p, t, virial=True, atomic=True)
            assert torch.equal(full["E"], E) and torch.equal(full["E_atoms"], Ea)
            some = plan.run(p, t, forces=False, virial=True)
            assert torch.equal(some["E"], E)
            plain = plan.run(p, t)
            assert torch.equal(plain["E"], E)
            plan.check()
            # forces: atomic sums in any order
            tol = (1e-12 if prec == FP64 else 1e-5) * max(1.0, float(plain["F"].abs().max()))
            assert float((plain["F"] - full["F"]).abs().max()) <= tol
            assert float((plain["F"] + plan.backward()).abs().max()) <= tol
            sums = torch.stack([x.sum() for x in torch.split(Ea, sizes)])
            size = torch.stack([x.abs().sum() for x in torch.split(Ea, sizes)])
            assert bool(((E - sums).abs() <= 64 * 2.2e-16 * size).all())
            plan.close()
    finally:
        ann.release()
