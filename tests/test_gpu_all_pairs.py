"""The search over all pairs of wide orthogonal structures against the cell
lists: boxes just below and above twice the cut-off, numbers of atoms around
a batch and around the kernel's limit, plans with wide and narrow structures
side by side, and recorded launches whose lattices become narrow or oblique
later."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RC = 4.001      # the cut-off of the potentials and its margin


def _potentials(tmp_path):
    from aenet_gb300 import nnfile, workloads
    from aenet_gb300.core import ANNPotentials
    rng = np.random.default_rng(3)
    types = ["Li", "Si"]
    setups = {t: nnfile.chebyshev_setup(t, types, 4.0, 4, 3.4, 2, 1.0) for t in types}
    w = workloads.Workload("wide", types, setups, [16, 8, 8, 1], [], 4)
    w.networks = workloads.glorot_networks(rng, types, w.arch)
    stats = {t: (np.zeros(16), np.zeros(16), np.zeros(16), np.full(16, 25.0)) for t in types}
    return ANNPotentials(workloads.write_potentials(w, str(tmp_path), stats=stats),
                         angular_domain="current")


def _rows(torch, plan):
    """counts, and per atom its neighbours' indices and vectors in the order
    of (index, vector): images of one atom are whole ångströms apart"""
    cap, cnt, jt, vec = plan.neighbors()
    k = torch.arange(cap, device="cuda")[None] < cnt[:, None]
    j = torch.where(k, jt & ((1 << 26) - 1), 1 << 26).cpu().numpy()
    v = torch.where(k[..., None], vec.double(), 0.0).cpu().numpy()
    r = np.rint(v[..., :3] / 0.5)       # ties are broken the same way below
    order = np.lexsort((r[..., 2], r[..., 1], r[..., 0], j), axis=1)
    return (cnt.cpu().numpy(), np.take_along_axis(j, order, 1),
            np.take_along_axis(v, order[..., None], 1))


def _same(a, b, tol):
    assert np.array_equal(a[0], b[0])
    assert np.array_equal(a[1], b[1])
    # rows with two images of one atom may come in either order of them
    once = np.ones(a[1].shape, bool)
    eq = (a[1][:, 1:] == a[1][:, :-1])
    once[:, 1:] &= ~eq
    once[:, :-1] &= ~eq
    assert np.abs(a[2] - b[2])[once].max(initial=0.0) <= tol
    assert np.abs(a[2].sum(1) - b[2].sum(1)).max() <= tol * a[2].shape[1]


@pytest.mark.parametrize("edges", [(2.0, 2.01, 2.5), (2.0019, 2.0019, 2.0019),
                                   (2.003, 2.003, 2.003), (2.003, 3.5, 2.7), (1.2, 0.9, 4.0)])
def test_all_pairs_against_cells(edges, tmp_path):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from aenet_gb300.core import FP64, MIXED, set_option
    from aenet_gb300.plan import Plan
    rng = np.random.default_rng(17)
    L = np.array(edges) * RC
    nat = [1, 2, 31, 32, 33, 64, 65, 767, 768, 769]
    if edges == (2.0, 2.01, 2.5):
        # a plan of one structure, and wide and narrow ones together
        sets = [([n], [L + 0.2]) for n in nat] + [(nat, [L + 0.2 * (k & 1) for k in range(len(nat))])]
    else:
        sets = [([n], [L]) for n in (33, 768)] + [(nat, [L] * len(nat))]
    ann = _potentials(tmp_path)
    try:
        for ns, Ls in sets:
            cells = np.array([np.diag(x) for x in Ls])
            # far outside the cell as well, and some exactly on its faces
            pos = np.concatenate([(rng.random((n, 3)) * 3 - 1) * x for n, x in zip(ns, Ls)])
            pos[::7, 1] = 0.0
            typ = rng.integers(1, 3, len(pos)).astype(np.int32)
            p, t = torch.tensor(pos, device="cuda"), torch.tensor(typ, device="cuda")
            # FP64 vectors: both searches evaluate the same expression; FP32:
            # two roundings of coordinates of up to 16 A
            for prec, tol in ((FP64, 1e-13), (MIXED, 4e-6)):
                got = {}
                for kern in ("cell", "atom", "struct", "struct_half"):
                    set_option("neighbour_kernel", kern)
                    plan = Plan(ns, cells, np.ones(len(ns), np.int32), precision=prec)
                    plan.run(p, t)
                    plan.check()
                    got[kern] = _rows(torch, plan)
                    plan.close()
                for kern in ("atom", "struct", "struct_half"):
                    _same(got["cell"], got[kern], tol)
    finally:
        set_option("neighbour_kernel", "atom")
        ann.release()


@pytest.mark.parametrize("fp64", [False, True])
def test_recorded_launches_after_new_lattices(fp64, tmp_path):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from aenet_gb300.core import FP64, MIXED
    from aenet_gb300.plan import Plan
    rng = np.random.default_rng(5)
    n = 90
    wide = np.diag([9.0, 10.0, 11.0])
    later = [np.diag([7.0, 10.0, 12.0]),
             np.array([[9.0, 1.0, 0.0], [0.5, 9.5, 1.0], [0.0, 2.0, 10.0]]), wide]
    s = rng.random((n, 3))
    t = torch.tensor(rng.integers(1, 3, n).astype(np.int32), device="cuda")
    p = torch.tensor(s @ wide, device="cuda")
    ann = _potentials(tmp_path)
    prec = FP64 if fp64 else MIXED
    try:
        plan = Plan([n], wide[None], np.array([1]), precision=prec)
        plan.run(p, t)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = plan.run(p, t)
        for cell in later:
            p.copy_(torch.tensor(s @ cell))
            plan.set_cells(cell[None])
            graph.replay()
            plan.check()
            rows = _rows(torch, plan)
            E = out["E"].clone()
            fresh = Plan([n], cell[None], np.array([1]), precision=prec)
            want = fresh.run(p, t)["E"]
            _same(_rows_to(_rows(torch, fresh), rows), rows, 1e-13 if fp64 else 4e-6)
            # sums of some thousand terms in another order
            assert abs(float(E - want)) <= (1e-9 if fp64 else 1e-3)
            fresh.close()
        plan.close()
    finally:
        ann.release()


def _rows_to(a, like):
    """a's rows cut or filled to the row length of `like`"""
    w = like[1].shape[1]
    assert a[0].max() <= w
    j = np.full((len(a[0]), w), 1 << 26)
    v = np.zeros((len(a[0]), w, 4))
    m = min(w, a[1].shape[1])
    j[:, :m], v[:, :m] = a[1][:, :m], a[2][:, :m]
    return a[0], j, v
