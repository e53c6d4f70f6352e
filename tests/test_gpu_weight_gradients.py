"""Loss and weight gradients where their kernels' blocks, tiles and quadruples
end: narrow and odd layers, one atom and no atom of a species, fewer atoms
than blocks, one structure and more structures than blocks.  The loss against
its definition, the gradient against differences of the loss along random
directions (Richardson, relative 1e-6) and mixed against FP64 (2e-3 of the
norm)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("arch,sizes", [
    ([16, 3, 2, 1], [1]),
    ([16, 7, 1], [33]),
    ([16, 1, 1], [64, 1, 31]),
    ([16, 4, 5, 1], [700]),
    ([16, 33, 3, 6, 1], [2, 129]),
    ([16, 32, 32, 1], [3] * 400),
])
@pytest.mark.parametrize("absent", [False, True])
def test_edges(arch, sizes, absent, tmp_path):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from aenet_gb300 import nnfile, workloads
    from aenet_gb300.core import ANNPotentials, FP64, MIXED
    from aenet_gb300.plan import Plan
    rng = np.random.default_rng(len(sizes) + arch[1])
    types = ["Li", "Si", "O"]
    setups = {t: nnfile.chebyshev_setup(t, types, 4.0, 4, 3.4, 2, 1.0) for t in types}
    w = workloads.Workload("edges", types, setups, arch, [], 5)
    w.networks = workloads.glorot_networks(rng, types, arch)
    stats = {t: (np.zeros(16), np.zeros(16), np.zeros(16), np.full(16, 25.0)) for t in types}
    ann = ANNPotentials(workloads.write_potentials(w, str(tmp_path), stats=stats),
                        angular_domain="current")
    n = sum(sizes)
    edge = [max(3.0, (12.0 * k) ** (1 / 3)) for k in sizes]
    cells = np.array([np.diag([e] * 3) for e in edge])
    pos = []
    for k, e in zip(sizes, edge):       # a jittered grid: no two atoms close
        m = int(np.ceil(k ** (1 / 3) - 1e-9))
        g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[:k]
        pos.append((g + rng.uniform(-0.15, 0.15, g.shape)) * (e / m))
    # one atom of the second species, or none of it
    typ = rng.choice([1, 3], n).astype(np.int32)
    if not absent:
        typ[n // 2] = 2
    p = torch.tensor(np.concatenate(pos), device="cuda")
    t = torch.tensor(typ, device="cuda")
    E_t = torch.tensor(rng.normal(0, 1, len(sizes)), device="cuda")
    F_t = torch.tensor(rng.normal(0, 0.3, (n, 3)), device="cuda")
    nat = np.array(sizes)
    nw = [ann.nweights(x) for x in types]
    out = {}
    try:
        W0 = ann.get_weights()
        for prec in (FP64, MIXED):
            plan = Plan(sizes, cells, np.ones(len(sizes), np.int32), precision=prec)
            E = torch.empty(len(sizes), dtype=torch.float64, device="cuda")
            F = torch.empty((n, 3), dtype=torch.float64, device="cuda")

            def run(W):
                ann.set_weights(W)
                loss, g = plan.loss_gradient(p, t, E_t, F_t, w_E=1.0, w_F=0.1, E=E, F=F)
                return float(loss), g.cpu().numpy().copy()

            loss, g = run(W0)
            plan.check()
            # (forces: minus the gradient; the sums' rounding)
            want = float(((E - E_t).cpu().numpy() ** 2 / nat.astype(float) ** 2).sum()
                         + 0.1 * ((F - F_t) ** 2).sum())
            assert abs(loss - want) <= 1e-12 * want
            again = run(W0)[1] if prec == FP64 else g
            assert np.abs(again - g).max() <= 1e-12 * np.abs(g).max()
            out[prec] = g
            if prec == FP64:
                for _ in range(3):
                    d = rng.normal(0, 1, len(W0))
                    h = 1e-3 / np.linalg.norm(d)
                    f = {m: run(W0 + m * h * d)[0] for m in (-2, -1, 1, 2)}
                    fd = (8 * (f[1] - f[-1]) - (f[2] - f[-2])) / (12 * h)
                    assert abs(fd - g @ d) <= 1e-6 * np.abs(g * d).sum()
                ann.set_weights(W0)
            plan.close()
    finally:
        ann.release()
    second = slice(nw[0], nw[0] + nw[1])
    for g in out.values():
        assert np.isfinite(g).all()
        assert absent == (not g[second].any())
    assert np.linalg.norm(out[MIXED] - out[FP64]) <= 2e-3 * np.linalg.norm(out[FP64])
