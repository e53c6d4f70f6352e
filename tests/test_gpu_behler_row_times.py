"""Time of one-row Behler calls of five species: lists whose etas differ from each
other's take little longer than lists of the same etas (the factors of a list's
neighbours are filled once for both of its species)."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TYPES = ["H", "Li", "O", "Si", "Ti"]


def _call_us(tmp_path, own):
    from aenet_gb300 import nnfile, workloads
    from aenet_gb300.core import ANNPotentials
    rng = np.random.default_rng(4)
    funcs = [{"G": 2, "type2": t, "Rc": 6.0, "Rs": 0.0, "eta": e} for t in TYPES
             for e in (0.003, 0.03, 0.1)]
    for i, a in enumerate(TYPES):
        for b in TYPES[i:]:
            etas = rng.uniform(0.001, 0.1, 2) if own else (0.003, 0.03)
            funcs += [{"G": 4, "type2": a, "type3": b, "Rc": 6.0, "lambda": lam, "zeta": 1.0,
                       "eta": float(e)} for lam in (1.0, -1.0) for e in etas]
    n = len(funcs)
    w = workloads.Workload("rows", TYPES, {t: nnfile.behler_setup(t, TYPES, funcs, 1.0)
                                           for t in TYPES}, [n, 20, 20, 1], [], 4)
    w.networks = workloads.glorot_networks(rng, TYPES, w.arch)
    stats = {t: (np.zeros(n), np.zeros(n), np.zeros(n), np.full(n, 100.0)) for t in TYPES}
    ann = ANNPotentials(workloads.write_potentials(w, str(tmp_path), stats=stats),
                        angular_domain="current")
    x = rng.normal(size=(6, 3))
    x *= rng.uniform(2.0, 5.5, (6, 1)) / np.linalg.norm(x, axis=1)[:, None]
    symbols = [TYPES[k % 5] for k in range(6)]
    F, best = np.zeros((7, 3)), 1e9
    try:
        for _ in range(8):
            t0 = time.perf_counter()
            for _ in range(40):
                ann.atomic_energy_and_forces(np.zeros(3), "H", 1, x, symbols, np.arange(2, 8), F)
            best = min(best, (time.perf_counter() - t0) / 40e-6)
    finally:
        ann.release()
    return best


def test_lists_of_their_own_etas(tmp_path):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    same, own = (_call_us(tmp_path, o) for o in (False, True))
    # (filled bucket by bucket 1.2 times as long)
    assert own <= 1.1 * same, (same, own)
