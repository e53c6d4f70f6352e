"""The options for lanes per atom: each value reaches the descriptor and adjoint
kernels of both precisions and both angular forms (sums in another order, so
that some last bits differ), with the same results to rounding; rows too long
for the lanes asked take more, and so do few atoms where 8 are asked."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("orders,edge", [((10, 4), 10), ((16, 8), 10), ((7, 3), 10),
                                         ((10, 4), 4), ((16, 8), 4)])
def test_lanes_reach_the_kernels(orders, edge, tmp_path):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from aenet_gb300 import nnfile, workloads
    from aenet_gb300.core import ANNPotentials, FP64, MIXED, set_option
    from aenet_gb300.plan import Plan
    rng = np.random.default_rng(31)
    types = ["Li", "Si"]
    setups = {t: nnfile.chebyshev_setup(t, types, 5.0, orders[0], 4.5, orders[1], 1.0)
              for t in types}
    nsf = setups["Li"]["nsf"]
    w = workloads.Workload("lanes", types, setups, [nsf, 8, 1], [], 31)
    w.networks = workloads.glorot_networks(rng, types, w.arch)
    stats = {t: (np.zeros(nsf), np.zeros(nsf), np.zeros(nsf), np.full(nsf, 50.0)) for t in types}
    ann = ANNPotentials(workloads.write_potentials(w, str(tmp_path), stats=stats),
                        angular_domain="current")
    pos, cell = workloads.fcc_positions(edge, 3.9)
    pos = pos + rng.normal(0, 0.1, pos.shape)
    n = len(pos)
    p = torch.tensor(pos, device="cuda")
    t = torch.tensor(rng.integers(1, 3, n).astype(np.int32), device="cuda")
    try:
        for prec, tol in ((FP64, 1e-12), (MIXED, 2e-5)):
            G, F = {}, {}
            for lanes in (8, 16, 32):
                set_option("lanes_per_atom", lanes)
                plan = Plan([n], cell[None], np.array([1]), precision=prec)
                F[lanes] = plan.run(p, t)["F"].clone()
                G[lanes] = plan.descriptors()[:, :nsf].clone()
                for adj in (8, 16, 32):
                    set_option("adjoint_lanes_per_atom", adj)
                    f = plan.run(p, t)["F"]
                    assert float((f - F[lanes]).abs().max()) <= tol * float(F[8].abs().max())
                set_option("adjoint_lanes_per_atom", 0)
                plan.check()
                plan.close()
            size = float(G[8].abs().max())
            for a in (16, 32):
                assert float((G[a] - G[8]).abs().max()) <= tol * size
            if edge == 4:       # 256 atoms take 32 lanes by themselves
                assert torch.equal(G[16], G[32]) and torch.equal(G[8], G[32])
            else:
                assert not torch.equal(G[8], G[32])
    finally:
        set_option("lanes_per_atom", 16)
        set_option("adjoint_lanes_per_atom", 0)
        ann.release()


def test_lanes_give_way_to_long_rows(tmp_path):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from aenet_gb300 import nnfile, workloads
    from aenet_gb300.core import ANNPotentials, FP64, set_option
    from aenet_gb300.plan import Plan
    rng = np.random.default_rng(32)
    setup = nnfile.chebyshev_setup("Cu", ["Cu"], 10.0, 16, 10.0, 8, 1.0)
    nsf = setup["nsf"]
    w = workloads.Workload("long", ["Cu"], {"Cu": setup}, [nsf, 4, 1], [], 32)
    w.networks = workloads.glorot_networks(rng, ["Cu"], w.arch)
    stats = {"Cu": (np.zeros(nsf), np.zeros(nsf), np.zeros(nsf), np.full(nsf, 1e4))}
    ann = ANNPotentials(workloads.write_potentials(w, str(tmp_path), stats=stats),
                        angular_domain="current")
    g = np.stack(np.meshgrid(*[np.arange(4)] * 3, indexing="ij"), -1).reshape(-1, 3)
    pos = (g + rng.uniform(-0.1, 0.1, g.shape)) * 2.1     # 450 neighbours, 700 staged at most
    p = torch.tensor(pos, device="cuda")
    t = torch.ones(len(pos), dtype=torch.int32, device="cuda")
    got = []
    try:
        for lanes in (16, 8):
            set_option("adjoint_lanes_per_atom", lanes)
            plan = Plan([len(pos)], 8.4 * np.eye(3)[None], np.array([1]), precision=FP64)
            r = plan.run(p, t)
            plan.check()
            got.append([r["E"].clone(), r["F"].clone()])
            plan.close()
    finally:
        set_option("adjoint_lanes_per_atom", 0)
        ann.release()
    assert abs(float(got[0][0] - got[1][0])) <= 1e-10
    assert float((got[0][1] - got[1][1]).abs().max()) <= 1e-10
