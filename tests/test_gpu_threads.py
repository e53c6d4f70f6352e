"""Plans of different sizes run by host threads at once, each on its own stream:
kernels whose shared memory goes by the size of the plan (the one-block cell
lists, the FP64 networks) are launched by several at the same time, and every
pass returns what it returns alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fp64", [False, True])
def test_threads_with_plans_of_different_sizes(fp64, tmp_path):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from aenet_gb300 import nnfile, workloads
    from aenet_gb300.core import ANNPotentials, FP64, MIXED
    from aenet_gb300.plan import Plan
    rng = np.random.default_rng(11)
    types = ["Li", "Si"]
    setups = {t: nnfile.chebyshev_setup(t, types, 4.0, 4, 3.4, 2, 1.0) for t in types}
    w = workloads.Workload("threads", types, setups, [16, 40, 40, 1], [], 5)
    w.networks = workloads.glorot_networks(rng, types, w.arch)
    stats = {t: (np.zeros(16), np.zeros(16), np.zeros(16), np.full(16, 25.0)) for t in types}
    ann = ANNPotentials(workloads.write_potentials(w, str(tmp_path), stats=stats),
                        angular_domain="current")
    work, errors = [], []
    try:
        # 98, 58 and 43 KB of cell lists; tiles of 4, 4 and 2 atoms in the networks
        for m in (13, 11, 10):
            pos, cell = workloads.fcc_positions(m, 3.9)
            pos = pos + rng.normal(0, 0.1, pos.shape)
            typ = rng.integers(1, 3, len(pos)).astype(np.int32)
            plan = Plan([len(pos)], cell[None], np.array([1]), precision=FP64 if fp64 else MIXED)
            p, t = torch.tensor(pos, device="cuda"), torch.tensor(typ, device="cuda")
            work.append((plan, p, t, plan.run(p, t)["E"].clone()))
            plan.check()
        torch.cuda.synchronize()

        def go(plan, p, t, E):
            try:
                with torch.cuda.stream(torch.cuda.Stream()):
                    out = {}
                    for _ in range(400):
                        plan.run(p, t, out=out)
                    plan.check()
                    assert torch.equal(out["E"], E)
            except Exception as e:
                errors.append(e)

        threads = [threading.Thread(target=go, args=a) for a in work]
        for th in threads:
            th.start()
        for th in threads:
            th.join()
        torch.cuda.synchronize()
        for plan, *_ in work:
            plan.close()
    finally:
        ann.release()
    assert not errors, errors
