"""Plans whose cell lists, grouping by species and energy sum take one block
each, at the edges of those kernels (a block's width, the tiles of the
grouping, a chunk of the energy sum, the largest plan and the first beyond):
neighbour counts against all pairs, energies against the sum of the atoms',
networks of both paths, and rows in the same order every time."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 1023, 1025, 2048, 2049, 4097, 8192, 12288, 12289])
def test_small_plan_edges(n, tmp_path):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from aenet_gb300 import nnfile, workloads
    from aenet_gb300.core import ANNPotentials, FP64, MIXED
    from aenet_gb300.plan import Plan
    rng = np.random.default_rng(n)
    m = int(np.ceil((n / 4) ** (1 / 3)))
    pos, cell = workloads.fcc_positions(max(2, m), 3.9)
    pos = pos[rng.permutation(len(pos))[:n]] + rng.normal(0, 0.1, (n, 3))
    typ = rng.integers(1, 4, n).astype(np.int32)
    types = ["Li", "Si", "O"]
    setups = {t: nnfile.chebyshev_setup(t, types, 4.0, 4, 3.4, 2, 1.0) for t in types}
    w = workloads.Workload("small", types, setups, [16, 8, 8, 1],
                           [workloads.Structure(pos, typ, cell)], n)
    w.networks = workloads.glorot_networks(rng, types, w.arch)
    stats = {t: (np.zeros(16), np.zeros(16), np.zeros(16), np.full(16, 25.0)) for t in types}
    ann = ANNPotentials(workloads.write_potentials(w, str(tmp_path), stats=stats),
                        angular_domain="current")
    p = torch.tensor(pos, device="cuda")
    t = torch.tensor(typ, device="cuda")
    try:
        out = {}
        for prec in (FP64, MIXED):
            plan = Plan([n], cell[None], np.array([1]), precision=prec)
            r = plan.run(p, t, atomic=True)
            first = [x.clone() for x in (r["E"], r["E_atoms"], r["F"])]
            cap, cnt, jt, _ = plan.neighbors()
            rows = jt.clone()
            again = plan.run(p, t, atomic=True)
            plan.check()
            cells = int(cell[0, 0] / (4.001 / 2)) ** 3
            if n <= 12288 and cells <= 16384:
                k = torch.arange(cap, device="cuda") < cnt[:, None]
                assert torch.equal(rows[k], plan.neighbors()[2][k])
                assert torch.equal(first[1], again["E_atoms"])
                assert torch.equal(first[0], again["E"])
            # rounding of a sum of n terms in tree order (at most 32 levels)
            e = first[1]
            assert abs(float(first[0] - e.sum())) <= 64 * 2.2e-16 * float(e.abs().sum())
            out[prec] = [x.cpu().numpy() for x in first] + [cnt.cpu().numpy().copy()]
            plan.close()
    finally:
        ann.release()
    # all pairs and the nearest images (cut-off 4.001 A, cells of 7.8 A and
    # more), away from the band that rounding decides
    L = float(cell[0, 0])
    count = np.zeros(n, dtype=int)
    images = [L * torch.tensor([a, b, c], dtype=torch.float64, device="cuda")
              for a in (-1, 0, 1) for b in (-1, 0, 1) for c in (-1, 0, 1)]
    q = p - torch.floor(p / L) * L
    for lo in range(0, n, 512):
        near = torch.zeros(min(512, n - lo), dtype=torch.long, device="cuda")
        for T in images:
            near += (torch.cdist(q[lo:lo + 512], q + T,
                                 compute_mode="donot_use_mm_for_euclid_dist") <= 4.001).sum(1)
        count[lo:lo + 512] = near.cpu().numpy() - 1      # the atom itself
    for prec in (FP64, MIXED):
        assert np.array_equal(out[prec][3], count)
    assert np.abs(out[MIXED][1] - out[FP64][1]).max() < 1e-3
    assert np.sqrt(np.mean((out[MIXED][2] - out[FP64][2]) ** 2)) < 2e-2
