"""An atom's own image at the cut-off: a recorded pass of a wide cell replayed
after one edge has become as long as the cut-off with its margin, or longer or
shorter by a few units in the last place, against a new plan.  Whether an own
image is inside goes by the lattice vector alone (the same for every atom and
for both directions)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fp64", [False, True])
def test_own_image_at_the_cutoff(fp64, tmp_path):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from aenet_gb300.core import FP64, MIXED
    from aenet_gb300.plan import Plan
    from tests.test_gpu_all_pairs import RC, _potentials
    rng = np.random.default_rng(6)
    n = 16        # (rows of the narrow cell stay within the capacity of the wide one)
    wide = np.diag([9.0, 10.0, 11.0])
    s = rng.random((n, 3))
    t = torch.tensor(rng.integers(1, 3, n).astype(np.int32), device="cuda")
    p = torch.tensor(s @ wide, device="cuda")
    ann = _potentials(tmp_path)
    prec = FP64 if fp64 else MIXED
    own = torch.arange(n, device="cuda")[:, None]
    seen = set()
    try:
        plan = Plan([n], wide[None], np.array([1]), precision=prec)
        plan.run(p, t)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            plan.run(p, t)
        for ulps in (-3, -2, -1, 0, 1, 2, 3):
            cell = wide.copy()
            cell[1, 1] = RC + ulps * np.spacing(RC)
            p.copy_(torch.tensor(s @ cell))
            plan.set_cells(cell[None])
            graph.replay()
            plan.check()
            fresh = Plan([n], cell[None], np.array([1]), precision=prec)
            fresh.run(p, t)
            fresh.check()
            got = []
            for q in (plan, fresh):
                cap, cnt, jt, _ = q.neighbors()
                k = torch.arange(cap, device="cuda")[None] < cnt[:, None]
                images = (((jt & ((1 << 26) - 1)) == own) & k).sum(1).cpu().numpy()
                # both directions or neither, as the lattice vector decides
                assert np.all(images == images[0]) and images[0] in (0, 2)
                got.append((images, cnt.cpu().numpy()))
            assert np.array_equal(got[0][0], got[1][0])
            assert np.array_equal(got[0][1], got[1][1])
            seen.add(int(got[0][0][0]))
            fresh.close()
        plan.close()
        assert seen == {0, 2}
    finally:
        ann.release()
