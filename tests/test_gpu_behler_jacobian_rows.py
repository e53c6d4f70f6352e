"""Behler descriptor Jacobians of long neighbour rows (about 450 neighbours, a
capacity of 736) against the oracle at the tolerance of the suite's other
Jacobian test (1e-9 of the largest derivative)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_jacobian_of_long_rows(oracle, tmp_path):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from aenet_gb300 import nnfile, workloads
    from aenet_gb300.core import ANNPotentials, FP64
    from aenet_gb300.plan import Plan
    rng = np.random.default_rng(21)
    types = ["Ti", "O"]
    funcs = [{"G": 2, "type2": t, "Rc": 10.0, "Rs": 0.5, "eta": 0.02} for t in types]
    funcs += [{"G": 4, "type2": "Ti", "type3": "Ti", "Rc": 10.0, "lambda": lam, "zeta": 2.0,
               "eta": 0.01} for lam in (1.0, -1.0)]
    n = len(funcs)
    w = workloads.Workload("rows", types, {t: nnfile.behler_setup(t, types, funcs, 1.0)
                                           for t in types}, [n, 4, 1], [], 21)
    w.networks = workloads.glorot_networks(rng, types, w.arch)
    stats = {t: (np.zeros(n), np.zeros(n), np.zeros(n), np.full(n, 100.0)) for t in types}
    paths = workloads.write_potentials(w, str(tmp_path), stats=stats)
    g = np.stack(np.meshgrid(*[np.arange(5)] * 3, indexing="ij"), -1).reshape(-1, 3)
    pos = (g + rng.uniform(-0.1, 0.1, g.shape)) * 2.1
    cell = np.eye(3) * 10.5
    typ = (1 + (np.arange(len(pos)) % 9 > 0)).astype(np.int32)
    ann = ANNPotentials(paths, angular_domain="current")
    try:
        plan = Plan([len(pos)], cell[None], np.array([1]), precision=FP64)
        plan.run(torch.tensor(pos, device="cuda"), torch.tensor(typ, device="cuda"), forces=False)
        plan.check()
        cap, _, _, vec = plan.neighbors()
        assert cap == 736
        vec = vec.cpu().numpy()
        Ji, Jj, nbl, nnb = (x.cpu().numpy() for x in plan.jacobian(0, 3))
        plan.close()
    finally:
        ann.release()
    oracle.load(types, paths)
    _, centres, nb = oracle.neighbors(cell, pos, typ)
    for a in range(3):
        nbcoo, _, nblist, nbt = nb[a]
        _, di, dj = oracle.descriptor(centres[a], int(typ[a]), nbcoo, nbt, scaled=False, deriv=True)
        m = int(nnb[a])
        assert m == len(nblist) > 400
        scale = max(1.0, np.abs(dj).max())
        np.testing.assert_allclose(Ji[a, :n], di, rtol=0, atol=1e-9 * scale)
        R = nbcoo - centres[a]
        for q in range(m):
            k = int(np.argmin(np.abs(R - vec[a, q, :3]).sum(1)))
            assert nbl[a, q] + 1 == nblist[k]
            np.testing.assert_allclose(Jj[a, q, :n], dj[k], rtol=0, atol=1e-9 * scale)
