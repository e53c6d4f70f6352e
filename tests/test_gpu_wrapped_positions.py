"""Wrapped positions and cell indices as the kernels compute them: pairs of an
atom at the origin and one on an axis, at the faces of the search cells, at the
doubles beside them and some lattice vectors outside, whose FP64 vector is the
wrapped position itself.  Bit for bit against the plain expressions (division
by 2 pi, floor), by the search over cells and by the one over all pairs; a
wrong cell would lose the pair."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("edges", [(7.9, 7.3, 6.1), (8.1, 9.7, 8.3), (30.3, 21.7, 17.9)])
@pytest.mark.parametrize("kernel", ["atom", "struct_half"])
def test_wrapped_bits(edges, kernel, tmp_path):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from aenet_gb300.core import FP64, set_option
    from aenet_gb300.plan import Plan
    from tests.test_gpu_all_pairs import _potentials
    L = np.array(edges)
    rng = np.random.default_rng(2)
    x = [rng.uniform(-2, 3, 200) * 1.0]
    for nc in range(1, 16):
        f = np.arange(0, nc) / nc
        x += [f, np.nextafter(f, -1), np.nextafter(f, 2)]
    f = np.concatenate(x)
    f = np.concatenate([f, f - 1.0, f + 2.0, f - 3.0])
    axis = np.arange(len(f)) % 3
    pos = np.zeros((len(f), 2, 3))
    pos[np.arange(len(f)), 1, axis] = f * L[axis]
    ann = _potentials(tmp_path)
    try:
        set_option("neighbour_kernel", kernel)
        plan = Plan([2] * len(f), np.array([np.diag(L)] * len(f)), np.ones(len(f), np.int32),
                    precision=FP64)
        plan.run(torch.tensor(pos.reshape(-1, 3), device="cuda"),
                 torch.ones(2 * len(f), dtype=torch.int32, device="cuda"), forces=False)
        plan.check()
        cap, cnt, jt, vec = (v.cpu().numpy() if hasattr(v, "cpu") else v for v in plan.neighbors())
        cnt, jt, vec = cnt.copy(), jt.copy(), vec.copy()
        plan.close()
    finally:
        set_option("neighbour_kernel", "atom")
        ann.release()
    # the reciprocal lattice as the plan forms it
    V = L[0] * L[1] * L[2]
    b = np.array([L[1] * L[2], L[0] * L[2], L[0] * L[1]])
    B = (b / V) * 2.0 * 3.141592653589793
    for k in range(len(f)):
        v, l = axis[k], L[axis[k]]
        s = (B[v] * pos[k, 1, v]) / 6.283185307179586
        w = s - np.floor(s)
        w = 0.0 if w == 1.0 else w
        want = [l * w if T == 0 else l * (w + T) for T in (-1, 0, 1)]
        if min(abs(abs(R) - 4.001) for R in want) < 1e-6:
            continue
        want = sorted(R for R in want if abs(R) < 4.001)
        i = 2 * k
        row = slice(0, cnt[i])
        other = (jt[i, row] & ((1 << 26) - 1)) == i + 1
        got = sorted(vec[i, row, v][other].tolist())
        assert got == want, (edges, k, f[k], got, want)
        # (square root of a square)
        assert np.all(np.abs(vec[i, row, 3][other] - np.abs(vec[i, row, v][other]))
                      <= np.spacing(4.0))
