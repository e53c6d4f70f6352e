"""FP64 networks of many species: their stage of a pass of a thousand atoms takes
no more than some loads of the larger weights longer than that of one species
(a block's warps all wait for its copy of the weights)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NAMES = ["H", "Li", "O", "Si", "Ti", "Cu", "Au", "Fe"]


def _networks_us(torch, tmp_path, nt):
    from aenet_gb300 import nnfile, workloads
    from aenet_gb300.core import ANNPotentials, FP64
    from aenet_gb300.plan import Plan
    rng = np.random.default_rng(nt)
    types = NAMES[:nt]
    # 32 features with one species and with several
    order = (24, 6) if nt == 1 else (10, 4)
    setups = {t: nnfile.chebyshev_setup(t, types, 3.5, order[0], 3.0, order[1], 1.0) for t in types}
    nsf = setups["H"]["nsf"]
    w = workloads.Workload("times", types, setups, [nsf, 32, 32, 1], [], nt)
    w.networks = workloads.glorot_networks(rng, types, w.arch)
    stats = {t: (np.zeros(nsf), np.zeros(nsf), np.zeros(nsf), np.full(nsf, 100.0)) for t in types}
    ann = ANNPotentials(workloads.write_potentials(w, str(tmp_path), stats=stats),
                        angular_domain="current")
    try:
        g = np.stack(np.meshgrid(*[np.arange(10)] * 3, indexing="ij"), -1).reshape(-1, 3) * 2.6
        plan = Plan([1000], 26.0 * np.eye(3)[None], np.array([1]), precision=FP64)
        p = torch.tensor(g + rng.uniform(-0.2, 0.2, g.shape), device="cuda")
        t = torch.tensor(rng.integers(1, nt + 1, 1000).astype(np.int32), device="cuda")
        plan.run(p, t)
        us = min(1e3 * plan.profile(p, t)["networks"] for _ in range(10))
        plan.check()
        plan.close()
    finally:
        ann.release()
    return us


def test_many_species_do_not_slow_small_plans(tmp_path):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    one, eight = (_networks_us(torch, tmp_path, nt) for nt in (1, 8))
    # the weights of eight species are 150 KB more a block, some 10 us
    assert eight <= 2.2 * one, (one, eight)
