"""Behler plans whose atoms take one block each or one per pair of species
(the launch chooses by the number of atoms): one structure alone and the same
structure many times in a plan, over the list forms of test_gpu_behler_pairs.
The lists' sums are the same, so that energies agree to FP64 rounding (1e-12
eV); forces differ by the order of their sums (FP64 1e-11, mixed 2e-5 of the
largest force); the FP64 exponential within an ulp of libm's by G2 sums."""
import numpy as np
import pytest

from tests.test_gpu_behler_pairs import LISTS, _workload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts", [(1, 2), (30, 34)])
@pytest.mark.parametrize("which", sorted(LISTS))
def test_split_lists_match_whole_atoms(tmp_path, which, counts):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from aenet_gb300 import workloads
    from aenet_gb300.core import ANNPotentials, FP64, MIXED
    from aenet_gb300.plan import Plan
    w = _workload(LISTS[which], counts, 7 + len(which))
    s = w.structures[0]
    n, nsf = s.natoms, w.arch[0]
    stats = {t: (np.zeros(nsf), np.zeros(nsf), np.zeros(nsf), np.full(nsf, 100.0))
             for t in w.types}
    ann = ANNPotentials(workloads.write_potentials(w, str(tmp_path), stats=stats),
                        angular_domain="current")
    try:
        for prec in (FP64, MIXED):
            ref = None
            # below and above the lines of either precision on 148 to 160 SMs
            for atoms in (0, 760, 1100, 1280, 1400):
                copies = max(1, atoms // n)
                p = torch.tensor(np.tile(s.positions, (copies, 1)), device="cuda")
                t = torch.tensor(np.tile(s.types, copies).astype(np.int32), device="cuda")
                plan = Plan([n] * copies, np.array([s.cell] * copies), np.ones(copies, np.int32),
                            precision=prec)
                r = plan.run(p, t, virial=True, atomic=True)
                plan.check()
                E = r["E_atoms"].reshape(copies, n).cpu().numpy()
                F = r["F"].reshape(copies, n, 3).cpu().numpy()
                W = r["virial"].reshape(copies, 9).cpu().numpy()
                plan.close()
                if ref is None:
                    ref = (E[0], F[0], W[0])
                big = max(1.0, np.abs(ref[1]).max())
                tol = (1e-11 if prec == FP64 else 2e-5) * big
                assert np.abs(E - ref[0]).max() <= 1e-12 * max(1.0, np.abs(ref[0]).max())
                assert np.abs(F - ref[1]).max() <= tol, atoms
                assert np.abs(W - ref[2]).max() <= 100 * tol, atoms
    finally:
        ann.release()


def test_exponentials_over_their_range(tmp_path):
    """One neighbour, G5 with eta from 0 to beyond the range of exp: E of a
    linear network is the sum of the functions."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from aenet_gb300 import nnfile, workloads
    from aenet_gb300.core import ANNPotentials, FP64
    etas = np.concatenate([[0.0], 10.0 ** np.linspace(-6, 3, 40), [35.0, 38.8, 39.0, 41.0]])
    funcs = [{"G": 5, "type2": "Ti", "type3": "Ti", "Rc": 8.0, "lambda": 1.0, "zeta": 1.0,
              "eta": float(e)} for e in etas]
    nsf = len(funcs)
    setup = nnfile.behler_setup("Ti", ["Ti"], funcs, 1.0)
    w = workloads.Workload("exp", ["Ti"], {"Ti": setup}, [nsf, 1], [], 1)
    stats = {"Ti": (np.zeros(nsf), np.zeros(nsf), np.zeros(nsf), np.ones(nsf))}
    pos = np.array([[0.0, 0, 0], [3.0, 0, 0], [0, 3.0, 0]])
    got = []
    W = np.zeros((1, nsf + 1))
    w.networks = {"Ti": nnfile.make_network([nsf, 1], W.ravel(order="F"))}
    ann = ANNPotentials(workloads.write_potentials(w, str(tmp_path), stats=stats),
                        angular_domain="current")
    try:
        base = ann.structure_energy_forces(pos, np.ones(3, np.int32), None, pbc=False,
                                           precision=FP64)["atomic_energies"][0]
        for k in range(nsf):
            W[:] = 0
            W[0, k] = 1.0
            ann.set_weights(W.ravel(order="F"))
            r = ann.structure_energy_forces(pos, np.ones(3, np.int32), None, pbc=False,
                                            precision=FP64)
            got.append(r["atomic_energies"][0] - base)
    finally:
        ann.release()
    got = np.array(got)
    fc = 0.5 * (np.cos(3.14159265358979 * 3.0 / 8.0) + 1.0)
    ref = 2.0 * 0.5 * np.exp(-etas * 18.0) * fc * fc
    # (E_scale multiplies all of them alike)
    scale = got[0] / ref[0]
    # a handful of roundings in each factor, and those of E_atom + E
    assert np.abs(got - scale * ref).max() <= 16 * 2.2e-16 * (abs(scale * ref[0]) + abs(base))
