"""Device memory of FP64 plans: the buffer of angular moments (400 bytes an atom
at angular order 4) belongs to the plans whose kernels use it, those of radial
order 10 or 16, and a basis of radial order 8 goes without."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bytes(torch, tmp_path, order, n):
    from aenet_gb300 import nnfile, workloads
    from aenet_gb300.core import ANNPotentials, FP64
    from aenet_gb300.plan import Plan
    setup = nnfile.chebyshev_setup("Cu", ["Cu"], 3.0, order, 2.9, 4, 1.0)
    nsf = setup["nsf"]
    w = workloads.Workload("memory", ["Cu"], {"Cu": setup}, [nsf, 4, 1], [], 1)
    w.networks = workloads.glorot_networks(np.random.default_rng(1), ["Cu"], w.arch)
    stats = {"Cu": (np.zeros(nsf), np.zeros(nsf), np.zeros(nsf), np.ones(nsf))}
    ann = ANNPotentials(workloads.write_potentials(w, str(tmp_path), stats=stats),
                        angular_domain="current")
    try:
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        plan = Plan([n], 400.0 * np.eye(3)[None], np.array([1]), precision=FP64)
        used = free - torch.cuda.mem_get_info()[0]
        plan.close()
    finally:
        ann.release()
    return used


def test_moment_buffers_only_where_used(tmp_path):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    n = 200000
    _bytes(torch, tmp_path, 8, n)       # (the first large allocations take more)
    pairs, moments = (_bytes(torch, tmp_path, order, n) for order in (8, 10))
    # two features more in two arrays of doubles, and the moments
    assert moments - pairs >= 400 * n
    assert pairs > 0
