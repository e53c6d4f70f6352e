"""FP64 pair-form adjoint with four, two and one blocks per atom (the launch
chooses by the number of atoms): one structure alone and many times in a plan,
one species and two, common orders and uncommon ones, legacy domain, rows from
none to several rounds.  The same sums in another order: 1e-11 of the largest
force, virials 1e-10."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("types,r_order,a_order,angular", [
    (["Cu"], 16, 8, "current"), (["Au", "Cu"], 12, 6, "current"), (["Au", "Cu"], 16, 8, "legacy"),
    (["Cu"], 9, 11, "legacy"), (["Li", "Si", "O"], 20, 7, "current"),
])
@pytest.mark.parametrize("scale", [0.85, 1.0, 1.9])
def test_parts_agree(types, r_order, a_order, angular, scale, tmp_path):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from aenet_gb300 import nnfile, workloads
    from aenet_gb300.core import ANNPotentials, FP64
    from aenet_gb300.plan import Plan
    rng = np.random.default_rng(r_order)
    setups = {t: nnfile.chebyshev_setup(t, types, 6.0, r_order, 4.2, a_order, 1.0) for t in types}
    nsf = setups[types[0]]["nsf"]
    w = workloads.Workload("parts", types, setups, [nsf, 12, 12, 1], [], 5)
    w.networks = workloads.glorot_networks(rng, types, w.arch)
    one = np.ones(nsf)
    stats = {t: (0 * one, 0 * one, 0 * one, 100.0 * one) for t in types}
    ann = ANNPotentials(workloads.write_potentials(w, str(tmp_path), stats=stats),
                        angular_domain=angular)
    # 32 atoms with periodic images: about 120, 75 and 10 neighbours
    pos, cell = workloads.fcc_positions(2, 3.65 * scale)
    pos = pos + rng.normal(0, 0.1, pos.shape)
    typ = rng.integers(1, len(types) + 1, len(pos)).astype(np.int32)
    n, ref = len(pos), None
    try:
        # 32, 128 | 160, 320, 352 | 384, 640 atoms on 152 SMs
        for copies in (1, 4, 5, 10, 11, 12, 20):
            p = torch.tensor(np.tile(pos, (copies, 1)), device="cuda")
            t = torch.tensor(np.tile(typ, copies), device="cuda")
            plan = Plan([n] * copies, np.array([cell] * copies), np.ones(copies, np.int32),
                        precision=FP64)
            r = plan.run(p, t, virial=True)
            plan.check()
            F = r["F"].reshape(copies, n, 3).cpu().numpy()
            W = r["virial"].reshape(copies, 9).cpu().numpy()
            plan.close()
            if ref is None:
                ref = (F[0], W[0])
            big = max(1e-3, np.abs(ref[0]).max())
            assert np.abs(F - ref[0]).max() <= 1e-11 * big
            assert np.abs(W - ref[1]).max() <= 1e-10 * max(1.0, np.abs(ref[1]).max())
    finally:
        ann.release()
