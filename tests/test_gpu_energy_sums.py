"""Energy sums of ragged plans: structures without atoms before, between and
after others, of one chunk and of several, against the sums of the atoms'
energies (rounding of a sum of n terms in tree order), and the time of the sums
of thousands of small structures beside one that is longer than a chunk."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ann(tmp_path):
    from aenet_gb300 import nnfile, workloads
    from aenet_gb300.core import ANNPotentials
    rng = np.random.default_rng(9)
    types = ["Li", "Si"]
    setups = {t: nnfile.chebyshev_setup(t, types, 3.0, 4, 2.9, 2, 1.0) for t in types}
    w = workloads.Workload("sums", types, setups, [16, 8, 1], [], 9)
    w.networks = workloads.glorot_networks(rng, types, w.arch)
    stats = {t: (np.zeros(16), np.zeros(16), np.zeros(16), np.full(16, 25.0)) for t in types}
    return ANNPotentials(workloads.write_potentials(w, str(tmp_path), stats=stats),
                         angular_domain="current")


def _plan(torch, sizes, precision):
    from aenet_gb300.plan import Plan
    rng = np.random.default_rng(len(sizes))
    pos, cells = [], []
    for n in sizes:
        m = max(1, int(np.ceil(n ** (1 / 3) - 1e-9)))
        g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
        pos.append((g + rng.uniform(-0.15, 0.15, g.shape)) * 2.8)
        cells.append(np.eye(3) * (2.8 * m))
    n = sum(sizes)
    plan = Plan(sizes, np.array(cells), np.ones(len(sizes), np.int32), precision=precision)
    p = torch.tensor(np.concatenate(pos), device="cuda")
    t = torch.tensor(rng.integers(1, 3, n).astype(np.int32), device="cuda")
    return plan, p, t


@pytest.mark.parametrize("sizes", [[0, 0, 3, 0, 2049, 0, 0, 5000, 1, 0], [0, 7], [4097, 0],
                                   [2048, 2049, 4096, 4097, 1]])
def test_ragged_sums(sizes, tmp_path):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from aenet_gb300.core import FP64, MIXED
    ann = _ann(tmp_path)
    try:
        for prec in (FP64, MIXED):
            plan, p, t = _plan(torch, sizes, prec)
            Ea = torch.empty(sum(sizes), dtype=torch.float64, device="cuda")
            nan = torch.full((len(sizes),), float("nan"), dtype=torch.float64, device="cuda")
            for _ in range(3):            # (the counters are back at zero every time)
                E = plan.forward(p, t, E=nan.clone(), E_atoms=Ea).clone()
                r = plan.run(p, t, out={"E": nan.clone()})
                assert torch.equal(r["E"], E)
                sums = torch.stack([x.sum() for x in torch.split(Ea, sizes)])
                size = torch.stack([x.abs().sum() for x in torch.split(Ea, sizes)])
                assert bool(((E - sums).abs() <= 64 * 2.2e-16 * size).all())
            plan.check()
            plan.close()
    finally:
        ann.release()


def test_one_long_structure_does_not_slow_the_sums(tmp_path):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from aenet_gb300.core import MIXED
    ann = _ann(tmp_path)
    best = []
    try:
        for sizes in ([8] * 8192, [8] * 8191 + [2049]):
            plan, p, t = _plan(torch, sizes, MIXED)
            ms = [plan.profile(p, t)["energy_reduce"] for _ in range(6)]
            best.append(min(ms[1:]))
            plan.check()
            plan.close()
    finally:
        ann.release()
    # the chunks are summed beside the others; a chain over the structures
    # takes about 80 times as long
    assert best[1] <= 10 * best[0] + 0.02, best
