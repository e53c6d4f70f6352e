"""Energy-only weight gradients of plans whose atoms the one-block cell lists
group by species: the neighbour rows, the grouping and every sum have a fixed
order, so that each call returns the same bits (a tile of atoms, a ragged last
tile, the largest such plan; a species without atoms)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,kinds", [(1024, 3), (4001, 3), (12288, 3), (6000, 2)])
def test_energy_gradients_repeat_bit_for_bit(n, kinds, tmp_path):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from aenet_gb300 import nnfile, workloads
    from aenet_gb300.core import ANNPotentials, FP64, MIXED
    from aenet_gb300.plan import Plan
    rng = np.random.default_rng(n)
    pos, cell = workloads.fcc_positions(int(np.ceil((n / 4) ** (1 / 3))), 3.9)
    pos = pos[rng.permutation(len(pos))[:n]] + rng.normal(0, 0.1, (n, 3))
    types = ["Li", "Si", "O"]
    setups = {t: nnfile.chebyshev_setup(t, types, 4.5, 4, 3.4, 2, 1.0) for t in types}
    w = workloads.Workload("bits", types, setups, [16, 8, 8, 1], [], n)
    w.networks = workloads.glorot_networks(rng, types, w.arch)
    stats = {t: (np.zeros(16), np.zeros(16), np.zeros(16), np.full(16, 25.0)) for t in types}
    ann = ANNPotentials(workloads.write_potentials(w, str(tmp_path), stats=stats),
                        angular_domain="current")
    p = torch.tensor(pos, device="cuda")
    t = torch.tensor(rng.integers(1, kinds + 1, n).astype(np.int32), device="cuda")
    target = torch.tensor([-3.0 * n], dtype=torch.float64, device="cuda")
    try:
        for prec in (FP64, MIXED):
            plan = Plan([n], cell[None], np.array([1]), precision=prec)
            loss, grad = (x.clone() for x in plan.loss_gradient(p, t, target))
            plan.check()
            assert bool(grad.abs().max() > 0)
            for _ in range(20):
                again = plan.loss_gradient(p, t, target)
                assert torch.equal(again[0], loss) and torch.equal(again[1], grad)
            plan.close()
    finally:
        ann.release()
