"""Workloads of the evaluator: what its users have it do, through its public
entry points, from one atom per call to a quarter of a million per pass.

A case names a potential family (the seeded families of
``aenet_gb300/workloads.py``), a call, a size and a precision:

  atom       ANNPotentials.atomic_energy_and_forces, one atom and its
             neighbour list per call (libaenet's own interface)
  structure  ANNPotentials.structure_energy_forces, one structure from host
             arrays (what the ASE calculator and the predict driver call)
  list       ANNPotentials.neighbor_list_energy_forces, local and ghost atoms
             with the caller's lists (what an MD engine calls)
  plan       Plan.run on device tensors, one crystal: energies and forces,
             the virial on request (what a molecular-dynamics step evaluates)
  batch      Plan.run on device tensors, many small cells
  train      Plan.loss_gradient on many small cells: the loss on energies and
             forces and its gradient with respect to every weight

The whole trajectory of the MD object is left out: its runs change the state
that they start from, so that two passes are not the same work.

The mixed path computes in 32 bits, whatever the arrays that it fills, and its
results are taken on as 32-bit values here, as programs that ask for it do; the
FP64 path's stay as they are.

``exact`` is the same physics written with plain torch in 64 bits: all pairs
within the cut-off, the descriptors as sums over pairs and triples, and
derivatives by automatic differentiation.
"""
import math
import os
import tempfile

import numpy as np
import torch

from aenet_gb300 import core, nnfile, workloads
from aenet_gb300.core import FP64, MIXED, ANNPotentials
from aenet_gb300.plan import LOSS_ENERGY_FORCES, Plan

# -------------------------------------------------------------- families
# species, density of the setting, basis and network as in workloads.py
FAMILIES = {
    "cu": dict(types=["Cu"], frac=[1.0], r=(16, 6.0), a=(8, 4.0), arch=[26, 20, 20, 1],
               lattice=3.61, noise=0.05),
    "aucu": dict(types=["Au", "Cu"], frac=[0.5, 0.5], r=(12, 6.5), a=(6, 4.5),
                 arch=[40, 25, 25, 1], lattice=3.90, noise=0.08),
    "cuau": dict(types=["Cu", "Au"], frac=[0.75, 0.25], r=(16, 6.0), a=(8, 4.0),
                 arch=[52, 20, 20, 1], lattice=3.70, noise=0.1),
    "lisio": dict(types=["Li", "Si", "O"], frac=[0.3, 0.3, 0.4], r=(10, 6.0), a=(4, 4.0),
                  arch=[32, 32, 32, 1], density=0.08),
    "rutile": dict(types=["Ti", "O"], behler=6.5, arch=[64, 30, 30, 1], noise=0.1),
}
E_SCALE, E_SHIFT = 1.0 / workloads.TS_SCALE, workloads.TS_SHIFT
# the launch shape that aenet_gb300.autotune settles on for large batches of
# small cells, and the library's defaults
TUNED = {"neighbour_kernel": "struct_half", "cell_div": 2, "z_refine": 4, "lanes_per_atom": 8,
         "adjoint_lanes_per_atom": 0}
DEFAULT = {"neighbour_kernel": "atom", "cell_div": 2, "z_refine": 1, "lanes_per_atom": 16,
           "adjoint_lanes_per_atom": 0}


def listed():
    return [
        # libaenet's own call, one atom of a copper crystal with 78 neighbours
        dict(name="atom-cu-78", call="atom", family="cu", neighbours=78),
        # an ASE calculator on a small supercell, plain FP64
        dict(name="structure-cu-256-fp64", call="structure", family="cu", nx=4, ny=4, nz=4,
             vacancies=0, fp64=True, virial=True),
        # a short-latency step of a small supercell in mixed precision
        dict(name="plan-cu-256-mixed", call="plan", family="cu", nx=4, ny=4, nz=4, vacancies=0,
             fp64=False, virial=False),
        # an alloy supercell: the ordinary size of a molecular-dynamics cell
        dict(name="plan-aucu-4000-mixed", call="plan", family="aucu", nx=10, ny=10, nz=10,
             vacancies=0, fp64=False, virial=False),
        # the same in plain FP64, odd edges and vacancies
        dict(name="plan-aucu-2765-fp64", call="plan", family="aucu", nx=11, ny=9, nz=7,
             vacancies=7, fp64=True, virial=False),
        # an oxide with Behler functions, mixed, with the virial (constant pressure)
        dict(name="plan-rutile-9000-mixed", call="plan", family="rutile", nx=10, ny=10, nz=15,
             vacancies=0, fp64=False, virial=True),
        # the same basis in plain FP64 on a ragged smaller cell
        dict(name="plan-rutile-763-fp64", call="plan", family="rutile", nx=4, ny=4, nz=8,
             vacancies=5, fp64=True, virial=False),
        # screening: thousands of small cells per pass, mixed, tuned launch shape
        dict(name="batch-lisio-4096-mixed", call="batch", family="lisio", structures=4096,
             fp64=False, virial=False, tuned=True),
        # reference data for such a batch in plain FP64, default launch shape
        dict(name="batch-lisio-512-fp64", call="batch", family="lisio", structures=512, fp64=True,
             virial=False, tuned=False),
        # a training step on energies and forces
        dict(name="train-lisio-512-mixed", call="train", family="lisio", structures=512,
             fp64=False, tuned=False),
        # the energies and forces of one step of a large crystal
        dict(name="plan-cuau-256k-mixed", call="plan", family="cuau", nx=40, ny=40, nz=40,
             vacancies=0, fp64=False, virial=False),
        # an MD engine's local and ghost atoms with its own lists
        dict(name="list-cuau-2048-mixed", call="list", family="cuau", nx=8, ny=8, nz=8, fp64=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the listed ranges: sizes over the logarithm, uneven edges,
    vacancies, either precision (FP64 up to the sizes that it is used at)."""
    call = rng.choice(["atom", "structure", "plan", "plan", "plan", "batch", "batch", "train",
                       "list"])
    if call == "atom":
        return dict(call="atom", family=rng.choice(["cu", "aucu", "cuau", "lisio"]),
                    neighbours=_log(rng, 12, 400))
    if call in ("batch", "train"):
        fp64 = rng.random() < 0.4
        case = dict(call=call, family="lisio",
                    structures=_log(rng, 3, (200 if call == "train" else 512) if fp64 else
                                    (1024 if call == "train" else 4096)),
                    fp64=fp64, tuned=rng.random() < 0.5)
        if call == "batch":
            case["virial"] = rng.random() < 0.3
        return case
    family = rng.choice(["cu", "aucu", "cuau"] if call == "list" else
                        ["cu", "aucu", "cuau", "rutile"])
    fp64 = call == "structure" or rng.random() < 0.4
    top = {"structure": 2000, "list": 8000}.get(call, 4000 if fp64 else 150000)
    if family == "rutile":
        top = min(top, 700 if fp64 else 9000)
    per = 6 if family == "rutile" else 4
    edge = (_log(rng, 100, top) / per) ** (1.0 / 3.0)
    nx, ny, nz = (max(2, int(round(edge * rng.uniform(0.8, 1.2)))) for _ in range(3))
    while per * nx * ny * nz > 1.1 * top:
        nx, nz = max(2, nx - 1), max(2, nz - 1)
    case = dict(call=call, family=family, nx=nx, ny=ny, nz=nz, fp64=fp64)
    if call != "list":
        case["vacancies"] = rng.randrange(0, 1 + min(31, nx * ny * nz // 8))
        case["virial"] = rng.random() < 0.4
    return case


# ---------------------------------------------------------------- inputs
def _rng(seed, salt=0):
    return np.random.default_rng([int(seed), salt])


def _crystal(case, rng):
    """(sites, thermal displacements, 1-based types, box edges) of a crystal."""
    fam = FAMILIES[case["family"]]
    if case["family"] == "rutile":
        pos, typ, cell = workloads.rutile_positions(case["nx"], case["ny"], case["nz"], 4.59, 2.96,
                                                    0.305)
        box = np.diag(cell)
    else:
        a = fam["lattice"]
        n = np.array([case["nx"], case["ny"], case["nz"]])
        base = np.array([[0, 0, 0], [0, .5, .5], [.5, 0, .5], [.5, .5, 0]])
        grid = np.stack(np.meshgrid(*[np.arange(k) for k in n], indexing="ij"), -1).reshape(-1, 3)
        pos = (grid[:, None, :] + base).reshape(-1, 3) * a
        box = n * a
        typ = workloads.exact_species(rng, len(pos), fam["frac"])
    keep = np.ones(len(pos), dtype=bool)
    keep[rng.permutation(len(pos))[:case.get("vacancies", 0)]] = False
    pos, typ = pos[keep], typ[keep]
    return pos, rng.normal(0.0, fam["noise"], pos.shape), typ.astype(np.int32), box


def _cells(structures, rng):
    """Random cubic cells of 16 to 512 atoms at 0.08 atoms / A^3: jittered
    sites of a cubic grid, chosen at random, 1.6 A apart at least.  The sizes
    go with the number of cells, their order with the seed."""
    sizes = np.random.default_rng([13, structures]).uniform(np.log(16), np.log(512), structures)
    sizes = np.rint(np.exp(rng.permutation(sizes))).astype(int)
    pos, typ, edges = [], [], []
    for n in sizes:
        L = (n / FAMILIES["lisio"]["density"]) ** (1.0 / 3.0)
        m = math.ceil(n ** (1.0 / 3.0) - 1e-9)
        site = rng.permutation(m ** 3)[:n]
        grid = np.stack([site // (m * m), site // m % m, site % m], -1)
        jitter = 0.5 * max(0.0, L / m - 1.6)
        pos.append((grid + 0.5) * (L / m) + rng.uniform(-jitter, jitter, (n, 3)))
        typ.append(workloads.exact_species(rng, int(n), FAMILIES["lisio"]["frac"]))
        edges.append(L)
    return sizes.astype(np.int32), np.concatenate(pos), np.concatenate(typ), np.array(edges)


def _row(case, rng):
    """A central atom and its ``neighbours`` nearest atoms inside the cut-off,
    in a random order: a crystal compressed or stretched to hold that many."""
    fam = FAMILIES[case["family"]]
    n, rc = case["neighbours"], max(fam["r"][1], fam["a"][1])
    g = np.arange(-8, 9)
    base = np.array([[0, 0, 0], [0, .5, .5], [.5, 0, .5], [.5, .5, 0]])
    grid = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    pts = (grid[:, None, :] + base).reshape(-1, 3)
    d = np.sort(np.linalg.norm(pts, axis=1))
    a = rc * 0.985 / (0.5 * (d[n] + d[n + 1]))     # d[0] is the atom itself
    pts = pts[np.argsort(np.linalg.norm(pts, axis=1), kind="stable")][1:n + 1] * a
    pts = pts + rng.uniform(-0.012, 0.012, pts.shape) * rc * a / 3.61
    pts = pts[rng.permutation(n)]
    types = workloads.exact_species(rng, n + 1, fam["frac"])
    return rng.uniform(0.0, 5.0, 3), pts, types


def _ghosts(site, move, typ, box, rc):
    """The local atoms, their ghost images within ``rc`` of the box, and full
    neighbour lists (CSR) of the local atoms, as an MD engine holds them."""
    pos = site + move
    x, t = [pos], [typ]
    for i in (-1, 0, 1):
        for j in (-1, 0, 1):
            for k in (-1, 0, 1):
                if (i, j, k) != (0, 0, 0):
                    p = site + np.array([i, j, k]) * box
                    keep = np.all((p > -rc - 1.0) & (p < box + rc + 1.0), axis=1)
                    x.append((p + move)[keep])
                    t.append(typ[keep])
    x, t = np.concatenate(x), np.concatenate(t)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    X = torch.as_tensor(x, device=dev)
    offs, nbr = [0], []
    for lo in range(0, len(pos), 256):
        near = torch.cdist(X[lo:min(lo + 256, len(pos))], X,
                           compute_mode="donot_use_mm_for_euclid_dist") <= rc
        near[torch.arange(near.shape[0]), lo + torch.arange(near.shape[0])] = False
        nbr.append(near.nonzero()[:, 1].to(torch.int32).cpu().numpy())
        offs.extend((offs[-1] + near.sum(1).cumsum(0)).tolist())
    return x, t.astype(np.int32), np.array(offs, dtype=np.int32), np.concatenate(nbr)


def _targets(seed, natoms, sizes):
    """Reference energies and forces of a training batch."""
    rng = _rng(seed, 1)
    E = sizes * (E_SHIFT - 2.1) + rng.normal(0.0, 0.3, len(sizes)) * np.sqrt(sizes)
    return E, rng.normal(0.0, 1.5, (natoms, 3))


def _inputs(case, seed):
    rng = _rng(seed)
    if case["call"] in ("batch", "train"):
        sizes, pos, typ, edges = _cells(case["structures"], rng)
        return dict(sizes=sizes, pos=pos, typ=typ, box=np.repeat(edges[:, None], 3, 1))
    if case["call"] == "atom":
        centre, pts, types = _row(case, rng)
        return dict(centre=centre, pts=pts, types=types)
    site, move, typ, box = _crystal(case, rng)
    pos = site + move
    got = dict(sizes=np.array([len(pos)], dtype=np.int32), pos=pos, typ=typ, box=box[None])
    if case["call"] == "list":
        got["list"] = _ghosts(site, move, typ, box, _rc(case["family"]) + 0.5)
    return got


def _rc(family):
    fam = FAMILIES[family]
    return fam["behler"] if "behler" in fam else max(fam["r"][1], fam["a"][1])


# ------------------------------------------------------------ potentials
_STATS, _LOADED = {}, {}


def _networks(family):
    fam = FAMILIES[family]
    rng = np.random.default_rng([7, sorted(FAMILIES).index(family)])
    return workloads.glorot_networks(rng, fam["types"], fam["arch"])


def _statistics(family):
    """Per species the mean and mean square of every descriptor over a sample
    (the statistics that a potential file carries)."""
    if family not in _STATS:
        if family == "lisio":
            sizes, pos, typ, edges = _cells(6, np.random.default_rng(11))
            box = np.repeat(edges[:, None], 3, 1)
        else:
            n = dict(nx=3, ny=3, nz=4) if family == "rutile" else dict(nx=4, ny=4, nz=4)
            pos, move, typ, box = _crystal(dict(family=family, **n), np.random.default_rng(11))
            pos = pos + move
            sizes, box = np.array([len(pos)]), box[None]
        model = _Model(family, None, "cpu")
        G = model.descriptors(pos, typ, sizes, box).numpy()
        _STATS[family] = [
            [np.array([float("%.9g" % v) for v in f(G[typ == t + 1], axis=0)])
             for f in (lambda g, axis: g.mean(axis), lambda g, axis: (g * g).mean(axis))]
            for t in range(len(FAMILIES[family]["types"]))]
    return _STATS[family]


def _potentials(family):
    """The loaded potentials of a family (the library holds one set at a time)."""
    if _LOADED.get("family") != family:
        if _LOADED:
            _LOADED.pop("ann").release()
            _LOADED.clear()
        fam = FAMILIES[family]
        types, nets, stats = fam["types"], _networks(family), _statistics(family)
        ts = dict(scale=workloads.TS_SCALE, shift=E_SHIFT, typeName=types,
                  E_atom=[-float(k + 1) for k in range(len(types))])
        if "behler" in fam:
            functions = workloads.behler_functions(types, fam["behler"])
        with tempfile.TemporaryDirectory() as d:
            paths = {}
            for k, t in enumerate(types):
                if "behler" in fam:
                    setup = nnfile.behler_setup(t, types, functions, workloads.RC_MIN)
                else:
                    setup = nnfile.chebyshev_setup(t, types, fam["r"][1], fam["r"][0],
                                                   fam["a"][1], fam["a"][0], workloads.RC_MIN)
                avg, sq = stats[k]
                setup.update(sfval_min=avg - 1.0, sfval_max=avg + 1.0, sfval_avg=avg, sfval_cov=sq)
                paths[t] = os.path.join(d, t + ".nn")
                nnfile.write_nn(paths[t], nets[t], setup, ts)
            _LOADED.update(family=family, ann=ANNPotentials(paths, angular_domain="current"))
    return _LOADED["ann"]


def _options(case):
    want = TUNED if case.get("tuned") else DEFAULT
    if _LOADED.get("options") is not want:
        for key, value in want.items():
            core.set_option(key, value)
        _LOADED["options"] = want


# ------------------------------------------------------- prepare and run
def prepare(case, seed):
    ann = _potentials(case["family"])
    _options(case)
    got = _inputs(case, seed)
    precision = FP64 if case.get("fp64") else MIXED
    state = dict(case=case, ann=ann, precision=precision)
    call, names = case["call"], FAMILIES[case["family"]]["types"]
    if call == "atom":
        t = got["types"]
        state.update(centre=got["centre"], type_i=names[t[0] - 1],
                     coo=got["centre"] + got["pts"], type_j=[names[k - 1] for k in t[1:]],
                     index_j=np.arange(2, len(t) + 1, dtype=np.int32),
                     F=np.zeros((len(t), 3)))
    elif call == "structure":
        state.update(pos=got["pos"], typ=got["typ"], cell=np.diag(got["box"][0]))
    elif call == "list":
        x, t, offs, nbr = got["list"]
        state.update(x=x, typ=t, offs=offs, nbr=nbr, nlocal=len(got["pos"]))
    else:
        cells = np.stack([np.diag(b) for b in got["box"]])
        state.update(plan=Plan(got["sizes"], cells, precision=precision),
                     pos=torch.as_tensor(got["pos"], device="cuda").contiguous(),
                     typ=torch.as_tensor(got["typ"], device="cuda").contiguous())
        if call == "train":
            E, F = _targets(seed, len(got["pos"]), got["sizes"])
            state.update(E_t=torch.as_tensor(E, device="cuda"),
                         F_t=torch.as_tensor(F, device="cuda").contiguous(),
                         E=torch.empty(len(E), dtype=torch.float64, device="cuda"),
                         F=torch.empty((len(F), 3), dtype=torch.float64, device="cuda"),
                         grad=torch.empty(ann.nweights(), dtype=torch.float64, device="cuda"),
                         loss=torch.empty(1, dtype=torch.float64, device="cuda"))
        else:
            state["out"] = {}
    return state


def run(state):
    case, ann, precision = state["case"], state["ann"], state["precision"]
    call = case["call"]
    if call == "atom":
        F = state["F"]
        F.fill(0.0)
        E = ann.atomic_energy_and_forces(state["centre"], state["type_i"], 1, state["coo"],
                                         state["type_j"], state["index_j"], F)
        return {"E": E, "F": F}
    if call == "structure":
        r = ann.structure_energy_forces(state["pos"], state["typ"], state["cell"],
                                        precision=precision, virial=case["virial"])
        out = {"E": r["energy"], "E_atoms": r["atomic_energies"], "F": r["forces"]}
        if case["virial"]:
            out["virial"] = r["virial"]
        return out
    if call == "list":
        r = ann.neighbor_list_energy_forces(state["x"], state["typ"], state["offs"], state["nbr"],
                                            state["nlocal"], precision=precision)
        out = {"E_atoms": r["atomic_energies"], "F": r["forces"]}
    elif call == "train":
        state["plan"].loss_gradient(state["pos"], state["typ"], state["E_t"], state["F_t"],
                                    mode=LOSS_ENERGY_FORCES, w_E=1.0, w_F=0.1, grad=state["grad"],
                                    loss=state["loss"], E=state["E"], F=state["F"])
        out = {k: state[k] for k in ("loss", "grad", "E", "F")}
    else:
        out = state["plan"].run(state["pos"], state["typ"], virial=case["virial"],
                                out=state["out"])
    if precision == FP64:
        return dict(out)
    return {k: v.float() if isinstance(v, torch.Tensor) else v.astype(np.float32)
            for k, v in out.items()}


# ----------------------------------------------------------------- work
def work(case):
    """Positions and types in, energies and forces out; the operations of the
    cheapest known form of the descriptors: radial terms per neighbour,
    angular terms as moments of spherical harmonics (Chebyshev) or per triple
    (Behler), the network forwards and backwards."""
    fam = FAMILIES[case["family"]]
    if case["call"] == "atom":
        atoms, structures, density = 1, 1, None
    elif case["call"] in ("batch", "train"):
        atoms, structures, density = 144.0 * case["structures"], case["structures"], fam["density"]
    else:
        rutile = case["family"] == "rutile"
        atoms = (6 if rutile else 4) * case["nx"] * case["ny"] * case["nz"]
        atoms -= case.get("vacancies", 0)
        structures = 1
        density = 6 / (4.59 * 4.59 * 2.96) if rutile else 4 / fam["lattice"] ** 3
    rc = _rc(case["family"])
    n = case["neighbours"] if density is None else density * 4.189 * rc ** 3
    weights = sum((i + 1) * o for i, o in zip(fam["arch"], fam["arch"][1:]))
    flops = 4.0 * weights + 10.0 * n
    if "behler" in fam:
        triples = 0.47 * n * (n - 1) / 2
        flops += n * 2 * (30 + 8 * 6) + triples * 2 * (60 + 16 * 4)
    else:
        m = 2 if len(fam["types"]) > 1 else 1
        na = n * (fam["a"][1] / rc) ** 3
        flops += n * 2 * (30 + 4 * m * (fam["r"][0] + 1))
        flops += na * 2 * (30 + 4 * m * (fam["a"][0] + 1) ** 2)
    moved = 24 + 4 + 24
    if case["call"] == "train":
        flops, moved = 3.0 * flops, moved + 24
    if case["call"] == "atom":
        return {"bytes": 52.0 * (n + 1) + 8.0 * weights, "flops": flops}
    if case["call"] == "list":
        moved += 4 * n
    width = 8.0 if case.get("fp64") else 4.0
    return {"bytes": atoms * moved + 8.0 * structures + width * weights * len(fam["types"]),
            "flops": atoms * flops}


# ---------------------------------------------------------------- exact
class _Model:
    """Energies and their derivatives in plain torch, 64 bits.  Rows are
    padded neighbour vectors [atoms, slots, 3]; an empty slot lies beyond
    every cut-off."""

    def __init__(self, family, stats, device):
        self.fam, self.device = FAMILIES[family], device
        self.types = len(self.fam["types"])
        self.rc = _rc(family)
        # spins of the species: consecutive integers from -(n // 2), zero left
        # out for an even number of species
        m = self.types
        spin = [k for k in range(-(m // 2), m + 1) if k or m % 2][:m]
        self.spin = torch.tensor(spin, dtype=torch.float64, device=device)
        if stats is not None:
            f = lambda v: torch.as_tensor(np.stack(v), device=device)
            self.avg = f([s[0] for s in stats])
            var = f([s[1] for s in stats]) - self.avg * self.avg
            s = var.clamp_min(0.0).sqrt()
            self.scale = torch.where(s <= 1e-10, torch.zeros_like(s), 1.0 / s)
            nets = _networks(family)
            self.weights = []
            for t in self.fam["types"]:
                W, at, layers = nets[t]["W"], 0, []
                for i, o in zip(self.fam["arch"], self.fam["arch"][1:]):
                    layers.append(torch.as_tensor(
                        W[at:at + (i + 1) * o].reshape(i + 1, o).copy(), device=device))
                    at += (i + 1) * o
                self.weights.append(layers)

    @staticmethod
    def _cut(d, rc):
        return torch.where(d < rc, 0.5 * (torch.cos(math.pi * d / rc) + 1.0), torch.zeros_like(d))

    @staticmethod
    def _chebyshev(x, order):
        T = [torch.ones_like(x), x]
        while len(T) <= order:
            T.append(2.0 * x * T[-1] - T[-2])
        return T[:order + 1]

    def rows(self, v, s):
        """Raw descriptors of rows: vectors v [A, M, 3], species s [A, M]
        (0-based, -1 in an empty slot)."""
        full = s >= 0
        d = v.square().sum(-1).sqrt()
        if "behler" in self.fam:
            return self._behler(v, d, s, full)
        (ro, rrc), (ao, arc) = self.fam["r"], self.fam["a"]
        w = self._cut(d, rrc) * full
        spin = self.spin[s.clamp_min(0)]
        radial = torch.stack(self._chebyshev(2.0 * d / rrc - 1.0, ro), -1) * w[..., None]
        near = full & (d < arc)
        order = torch.argsort((~near).to(torch.int8), dim=1, stable=True)
        M = max(1, int(near.sum(1).max()))
        order = order[:, :M]
        va = torch.gather(v, 1, order[..., None].expand(-1, -1, 3))
        da, sa = torch.gather(d, 1, order), torch.gather(spin, 1, order)
        wa = self._cut(da, arc) * torch.gather(near, 1, order)
        u = va / da[..., None]
        T = self._chebyshev(torch.einsum("aic,ajc->aij", u, u), ao)
        upper = torch.triu(torch.ones(M, M, dtype=torch.float64, device=v.device), 1)
        out = [radial.sum(1)]
        pairs = [torch.einsum("aij,ai,aj->a", t * upper, wa, wa) for t in T]
        out.append(torch.stack(pairs, -1))
        if self.types > 1:
            ws = wa * sa
            out.append((radial * spin[..., None]).sum(1))
            out.append(torch.stack([torch.einsum("aij,ai,aj->a", t * upper, ws, ws) for t in T],
                                   -1))
        return torch.cat(out, -1)

    def _behler(self, v, d, s, full):
        rc = self.fam["behler"]
        w = self._cut(d, rc) * full
        m = [(s == t).to(torch.float64) for t in range(self.types)]
        radial = torch.stack([torch.exp(-float(e) * d * d) * w
                              for e in np.geomspace(0.003, 0.5, 8)], -1)
        u = v / d[..., None]
        c = torch.einsum("aic,ajc->aij", u, u).clamp(-1.0, 1.0)
        x = (v[:, :, None] - v[:, None]).square().sum(-1)
        x = x + torch.eye(v.shape[1], dtype=torch.float64, device=v.device) * (4.0 * rc * rc)
        cut = w[:, :, None] * w[:, None] * self._cut(x.sqrt(), rc)
        upper = torch.triu(torch.ones_like(cut[0]), 1)
        cut = cut * upper
        q = (d * d)[:, :, None] + (d * d)[:, None] + x
        gauss = [torch.exp(-eta * q) * cut for eta in (0.003, 0.03)]
        angular = []                                 # per function [types, types]
        for zeta in (1, 2, 4, 16):
            for lam in (1.0, -1.0):
                p = (0.5 * (1.0 + lam * c)) ** zeta
                for g in gauss:
                    f = 2.0 * p * g
                    rows = [torch.einsum("aij,ai->aj", f, mi) for mi in m]
                    angular.append([[(r * mj).sum(1) for mj in m] for r in rows])
        out = []
        for t2 in range(self.types):
            out.append((radial * m[t2][..., None]).sum(1))
            for t3 in range(t2, self.types):
                fs = [a[t2][t3] if t2 == t3 else a[t2][t3] + a[t3][t2] for a in angular]
                out.append(torch.stack(fs, -1))
        return torch.cat(out, -1)

    def atom_energies(self, G, t, weights=None):
        """Atomic energies from raw descriptors, species t (0-based)."""
        E = torch.zeros(G.shape[0], dtype=torch.float64, device=G.device)
        for k, layers in enumerate(weights or self.weights):
            at = (t == k).nonzero()[:, 0]
            if at.numel():
                x = (G[at] - self.avg[k]) * self.scale[k]
                for l, W in enumerate(layers):
                    x = x @ W[:-1] + W[-1]
                    if l + 1 < len(layers):
                        x = torch.tanh(x)
                E = E.index_copy(0, at, E_SCALE * x[:, 0] + E_SHIFT - float(k + 1))
        return E

    # ---- pairs of periodic orthorhombic cells -------------------------
    def pairs(self, pos, sizes, box):
        """Chunks of (first home atom, home atoms, i, j, image vector) with
        every pair inside the cut-off; pos is wrapped by the caller."""
        dev, start = self.device, 0
        grid = np.floor(box[0] / self.rc).astype(int) if len(sizes) == 1 else np.zeros(3)
        if grid.min() >= 3:
            yield from self._pairs_grid(pos, box[0], grid)
            return
        step = 0
        while start < len(sizes):
            # structures of one chunk, with the same images
            images = np.maximum(1, np.ceil(self.rc / box[start])).astype(int)
            stop, cost = start, 0
            while stop < len(sizes) and np.array_equal(
                    images, np.maximum(1, np.ceil(self.rc / box[stop])).astype(int)):
                cost += int(sizes[stop]) ** 2
                if stop > start and cost * np.prod(2 * images + 1) > 3e7:
                    break
                stop += 1
            n = torch.as_tensor(sizes[start:stop].astype(np.int64), device=dev)
            first = torch.cumsum(n, 0) - n + step
            m = int(n.max())
            k = torch.arange(m, device=dev)
            index = torch.where(k < n[:, None], first[:, None] + k, -torch.ones_like(k))
            L = torch.as_tensor(np.array(box[start:stop]), device=dev)
            p = pos[index.clamp_min(0)]
            got = []
            for i in range(-images[0], images[0] + 1):
                for j in range(-images[1], images[1] + 1):
                    for l in range(-images[2], images[2] + 1):
                        T = L * torch.tensor([i, j, l], dtype=torch.float64, device=dev)
                        d = (p[:, None] + T[:, None, None] - p[:, :, None]).square().sum(-1)
                        ok = (d < self.rc ** 2) & (index[:, :, None] >= 0) & (index[:, None] >= 0)
                        if (i, j, l) == (0, 0, 0):
                            ok = ok & (k[:, None] != k)
                        b, x, y = ok.nonzero(as_tuple=True)
                        got.append((index[b, x], index[b, y], T[b]))
            total = int(n.sum())
            yield step, total, *(torch.cat(c) for c in zip(*got))
            step += total
            start = stop

    def _pairs_grid(self, pos, box, grid):
        dev = self.device
        L = torch.as_tensor(np.array(box), device=dev)
        g = torch.as_tensor(grid, device=dev)
        c = torch.minimum((pos / L * g).floor().long(), g - 1)
        flat = (c[:, 0] * g[1] + c[:, 1]) * g[2] + c[:, 2]
        cells = int(np.prod(grid))
        order = torch.argsort(flat, stable=True)
        count = torch.bincount(flat, minlength=cells)
        first = torch.cumsum(count, 0) - count
        m = int(count.max())
        slot = torch.arange(m, device=dev)
        table = torch.where(slot < count[:, None],
                            order[(first[:, None] + slot).clamp_max(len(pos) - 1)],
                            -torch.ones_like(slot))
        off = torch.tensor([[i, j, k] for i in (-1, 0, 1) for j in (-1, 0, 1) for k in (-1, 0, 1)],
                           device=dev)
        for lo in range(0, len(pos), 8192):
            home = torch.arange(lo, min(lo + 8192, len(pos)), device=dev)
            other = c[home][:, None] + off
            T = torch.div(other, g, rounding_mode="floor")
            other = other - T * g
            near = table[(other[..., 0] * g[1] + other[..., 1]) * g[2] + other[..., 2]]
            shift = T * L
            d = (pos[near.clamp_min(0)] + shift[:, :, None] - pos[home][:, None, None])
            ok = (d.square().sum(-1) < self.rc ** 2) & (near >= 0) & (
                (near != home[:, None, None]) | (T != 0).any(-1)[:, :, None])
            a, b, s = ok.nonzero(as_tuple=True)
            yield lo, len(home), home[a], near[a, b, s], shift[a, b]

    def chunks(self, pos, typ, sizes, box, atoms=None):
        """Row chunks: (first atom, count, i, j, image vector, slot) by atom."""
        atoms = atoms or (96 if "behler" in self.fam else 2048)
        for first, count, i, j, T in self.pairs(pos, sizes, box):
            order = torch.argsort(i, stable=True)
            i, j, T = i[order], j[order], T[order]
            per = torch.bincount(i - first, minlength=count)
            ends = torch.cumsum(per, 0)
            begin = ends - per
            slot = torch.arange(len(i), device=i.device) - begin[i - first]
            for lo in range(0, count, atoms):
                hi = min(lo + atoms, count)
                a, b = int(begin[lo]), int(ends[hi - 1])
                yield first + lo, hi - lo, i[a:b], j[a:b], T[a:b], slot[a:b]

    def _fill(self, pos, typ, first, count, i, j, T, slot):
        M = int(slot.max()) + 1 if len(slot) else 1
        v = torch.full((count, M, 3), 4.0 * self.rc, dtype=torch.float64, device=pos.device)
        v = v + torch.arange(M, device=pos.device)[:, None] * 2.0 * self.rc
        v = v.index_put((i - first, slot), pos[j] + T - pos[i])
        s = torch.full((count, M), -1, dtype=torch.long, device=pos.device)
        s = s.index_put((i - first, slot), typ[j])
        return v, s

    def _wrap(self, pos, sizes, box):
        L = torch.as_tensor(np.repeat(box, sizes, axis=0), device=self.device)
        p = torch.as_tensor(pos, device=self.device)
        return p - torch.floor(p / L) * L

    def descriptors(self, pos, typ, sizes, box):
        p, t = self._wrap(pos, sizes, box), torch.as_tensor(typ, device=self.device).long() - 1
        return torch.cat([self.rows(*self._fill(p, t, *c)) for c in
                          self.chunks(p, t, sizes, box)])

    def evaluate(self, pos, typ, sizes, box):
        """(atomic energies, forces, virial per structure)"""
        p, t = self._wrap(pos, sizes, box), torch.as_tensor(typ, device=self.device).long() - 1
        owner = torch.repeat_interleave(torch.arange(len(sizes), device=self.device),
                                        torch.as_tensor(sizes.astype(np.int64),
                                                        device=self.device))
        E, F = torch.zeros_like(p[:, 0]), torch.zeros_like(p)
        W = torch.zeros((len(sizes), 3, 3), dtype=torch.float64, device=self.device)
        for first, count, i, j, T, slot in self.chunks(p, t, sizes, box):
            v, s = self._fill(p, t, first, count, i, j, T, slot)
            v.requires_grad_(True)
            e = self.atom_energies(self.rows(v, s), t[first:first + count])
            g, = torch.autograd.grad(e.sum(), v)
            E[first:first + count] = e.detach()
            g, r = g[i - first, slot], v.detach()[i - first, slot]
            F.index_add_(0, i, g)
            F.index_add_(0, j, -g)
            W.index_add_(0, owner[i], -r[:, :, None] * g[:, None, :])
        return E, F, W, owner

    def loss(self, pos, typ, sizes, box, E_t, F_t, w_E, w_F):
        """The training loss and its gradient with respect to the weights."""
        Ea, F, _, owner = self.evaluate(pos, typ, sizes, box)
        n = torch.as_tensor(sizes.astype(np.float64), device=self.device)
        E = torch.zeros_like(n).index_add_(0, owner, Ea)
        dE = E - torch.as_tensor(E_t, device=self.device)
        dF = F - torch.as_tensor(F_t, device=self.device)
        loss = w_E * (dE / n).square().sum() + w_F * dF.square().sum()
        cE = (2.0 * w_E * dE / (n * n))[owner]
        p, t = self._wrap(pos, sizes, box), torch.as_tensor(typ, device=self.device).long() - 1
        flat = [W.clone().requires_grad_(True) for layers in self.weights for W in layers]
        per = len(self.fam["arch"]) - 1
        weights = [flat[k * per:(k + 1) * per] for k in range(self.types)]
        total = [torch.zeros_like(W) for W in flat]
        for first, count, i, j, T, slot in self.chunks(p, t, sizes, box):
            v, s = self._fill(p, t, first, count, i, j, T, slot)
            v.requires_grad_(True)
            e = self.atom_energies(self.rows(v, s), t[first:first + count], weights)
            g, = torch.autograd.grad(e.sum(), v, create_graph=True)
            # F_i = sum of g over the row of i, minus g where i is the neighbour
            along = (g[i - first, slot] * (dF[i] - dF[j])).sum()
            part = (cE[first:first + count] * e).sum() + 2.0 * w_F * along
            got = torch.autograd.grad(part, flat, allow_unused=True)
            total = [a if b is None else a + b for a, b in zip(total, got)]
        return loss.reshape(1), torch.cat([W.reshape(-1) for W in total]), E, F


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    model = _Model(case["family"], _statistics(case["family"]), dev)
    got = _inputs(case, seed)
    if case["call"] in ("atom", "list"):
        if case["call"] == "atom":
            x = np.concatenate([np.zeros((1, 3)), got["pts"]])
            t, n = got["types"], 1
            j = torch.arange(1, len(x), device=dev)
            i = torch.zeros_like(j)
        else:
            x, t, offs, nbr = got["list"]
            n = len(got["pos"])
            j = torch.as_tensor(nbr, device=dev).long()
            i = torch.repeat_interleave(torch.arange(n, device=dev),
                                        torch.as_tensor(np.diff(offs), device=dev).long())
        x, t = torch.as_tensor(x, device=dev), torch.as_tensor(t, device=dev).long() - 1
        near = (x[j] - x[i]).square().sum(-1) < model.rc ** 2
        i, j = i[near], j[near]
        per = torch.bincount(i, minlength=n)
        slot = torch.arange(len(i), device=dev) - (torch.cumsum(per, 0) - per)[i]
        v, s = model._fill(x, t, 0, n, i, j, torch.zeros_like(x[i]), slot)
        v.requires_grad_(True)
        e = model.atom_energies(model.rows(v, s), t[:n])
        g, = torch.autograd.grad(e.sum(), v)
        g = g[i, slot]
        F = torch.zeros_like(x).index_add_(0, i, g).index_add_(0, j, -g)
        if case["call"] == "atom":
            return {"E": float(e[0]), "F": F}
        return {"E_atoms": e.detach(), "F": F}
    args = got["pos"], got["typ"], got["sizes"], got["box"]
    if case["call"] == "train":
        E_t, F_t = _targets(seed, len(got["pos"]), got["sizes"])
        return dict(zip(("loss", "grad", "E", "F"), model.loss(*args, E_t, F_t, 1.0, 0.1)))
    Ea, F, W, owner = model.evaluate(*args)
    if case["call"] == "structure":
        out = {"E": float(Ea.sum()), "E_atoms": Ea, "F": F}
    else:
        out = {"E": torch.zeros(len(W), dtype=torch.float64, device=dev).index_add_(0, owner, Ea),
               "F": F}
    if case["virial"]:
        out["virial"] = W[0] if case["call"] == "structure" else W
    return out
