"""Performance cases of the framework: what its users have it do, with sizes.

Each case is a dict of plain values. prepare() makes what a program has in hand
before the call (a resident batch, a captured step graph, a SNAP potential, host
arrays), run() is one pass through the public Python entry points, and exact()
is the same result from plain torch in FP64 where that is defined. Inputs are
FCC / BCC lattices with seeded noise and Maxwell-Boltzmann velocities in the
reduced Lennard-Jones units of the benchmark (rho* 0.8442, T* 1.44, rc 2.5,
skin 0.3, dt 0.005) or the units of the SNAP decks.

Kinds of case:
  md        velocity-Verlet steps of one resident system
  ensemble  the same for a ragged batch of independent systems in one graph
  force     lennard_jones_force on current lists
  build     chunk_neighbors on current positions
  snap      a SNAP velocity-Verlet step, or the SNAP force operator alone
  request   one served request: upload, init, steps, download, removal
"""
import math
import os

import numpy as np
import torch

from exanbody_gb300 import snap, xnb

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
RCUT, SKIN, DT = 2.5, 0.3, 0.005
PAIRS = 0.5 * 4.18879020478639 * RCUT**3  # pairs within rc per atom and unit density
FCC = ((0.0, 0.0, 0.0), (0.0, 0.5, 0.5), (0.5, 0.0, 0.5), (0.5, 0.5, 0.0))
BCC = ((0.0, 0.0, 0.0), (0.5, 0.5, 0.5))
# the systems of the SNAP decks: lattice, constant (angstrom), atomic mass, noise
SNAP = {"Ni": (FCC, 3.48, 58.693, 0.05), "Mo": (BCC, 3.15, 95.96, 0.1)}


def listed():
    return [
        # the benchmark system, in the mixed path, as the step loop of a long run replays it
        {"name": "md_mixed_4m", "kind": "md", "n": 100, "rho": 0.8442, "T": 1.44, "precision": "mixed", "steps": 25,
         "graph": True},
        # the 32,000-atom configuration of the benchmark's small end: a few short launches per step
        {"name": "md_mixed_32k", "kind": "md", "n": 20, "rho": 0.8442, "T": 1.44, "precision": "mixed", "steps": 50,
         "graph": True},
        # the smallest system a user steps (the smoke system, 864 atoms): launch latency
        {"name": "md_mixed_864", "kind": "md", "n": 6, "rho": 0.8442, "T": 1.44, "precision": "mixed", "steps": 50,
         "graph": True},
        # ragged batch as the ensemble and serving drivers run it: 4^3 to 25^3 unit cells, dense to dilute, cool to hot
        {"name": "ensemble_mixed_96", "kind": "ensemble", "systems": 96, "nmin": 4, "nmax": 25, "precision": "mixed",
         "steps": 20},
        # full double precision at its faster traversal (Newton half lists)
        {"name": "md_fp64_newton_256k", "kind": "md", "n": 40, "rho": 0.8442, "T": 1.44, "precision": "fp64_newton",
         "steps": 5, "graph": True},
        # step() as its defaults have it: the reference's arithmetic bit for bit, the trigger read on the host
        {"name": "md_exact_sync_9k", "kind": "md", "n": 13, "rho": 0.8442, "T": 1.44, "precision": "fp64_exact",
         "steps": 5, "graph": False},
        # a force evaluation with energies on resident lists, one million atoms, odd lattice
        {"name": "force_mixed_energy_1m", "kind": "force", "n": 63, "rho": 0.8442, "precision": "mixed",
         "energy": True},
        # the reproducible double-precision force operator (full lists), odd size, dense fluid
        {"name": "force_fp64_119k", "kind": "force", "n": 31, "rho": 0.95, "precision": "fp64", "energy": False},
        # the neighbour build alone, two million atoms, odd lattice
        {"name": "build_2m", "kind": "build", "n": 79, "rho": 0.8442},
        # the Ni SNAP deck: 16,384 atoms, twojmax 8, one velocity-Verlet step in FP64
        {"name": "snap_ni_md_16k", "kind": "snap", "element": "Ni", "n": 16, "mixed": False, "md": True,
         "energy": False},
        # the Mo SNAP deck: 8,192 atoms, twojmax 6, forces and energies in the mixed path
        {"name": "snap_mo_mixed_8k", "kind": "snap", "element": "Mo", "n": 16, "mixed": True, "md": False,
         "energy": True},
        # a request of the serving driver alone on the GPU: host arrays in, 200 steps, host arrays out
        {"name": "request_mixed_23k", "kind": "request", "n": 18, "rho": 0.90, "T": 1.0, "precision": "mixed",
         "steps": 200},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["md", "md", "md", "ensemble", "force", "force", "build", "snap", "request"])
    rho, temp = round(rng.uniform(0.70, 1.00), 4), round(rng.uniform(0.7, 1.5), 4)
    if kind == "md":
        precision = rng.choice(["mixed", "mixed", "mixed", "fp64_newton", "fp64", "fp64_exact"])
        graph = precision != "fp64_exact"
        n = _log_int(rng, 6, 90 if precision == "mixed" else (40 if graph else 20))
        steps = rng.randint(10, 25) if n > 40 or precision != "mixed" else rng.randint(10, 50)
        return {"kind": kind, "n": n, "rho": rho, "T": temp, "precision": precision, "steps": steps, "graph": graph}
    if kind == "ensemble":
        nmin = rng.randint(4, 8)
        return {"kind": kind, "systems": _log_int(rng, 8, 96), "nmin": nmin, "nmax": rng.randint(nmin + 4, 25),
                "precision": "mixed", "steps": rng.randint(5, 20)}
    if kind == "force":
        precision = rng.choice(["mixed", "mixed", "fp64", "fp64_exact"])
        return {"kind": kind, "n": _log_int(rng, 30, 63 if precision == "mixed" else 40), "rho": rho,
                "precision": precision, "energy": rng.random() < 0.5}
    if kind == "build":
        return {"kind": kind, "n": _log_int(rng, 16, 79), "rho": rho}
    if kind == "snap":
        return {"kind": kind, "element": rng.choice(["Ni", "Mo"]), "n": rng.randint(8, 15),
                "mixed": rng.random() < 0.5, "md": rng.random() < 0.5, "energy": rng.random() < 0.5}
    return {"kind": kind, "n": _log_int(rng, 5, 24), "rho": rho, "T": temp, "precision": "mixed",
            "steps": rng.randint(100, 200)}


# ---------------------------------------------------------------------------
# Inputs, on the GPU from the seed.
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _geometry(length, nbh):
    """Cubic box of the given edge in cells of at least nbh."""
    d = max(2, int(math.floor(length / nbh)))
    return {"origin": (0.0, 0.0, 0.0), "extent": (length,) * 3, "dims": (d,) * 3, "cell_size": length / d}


def _lattice(basis, n, a, noise, g):
    """Sites of an n^3 block of unit cells, (k, j, i, basis) order, with Gaussian noise, wrapped into the box."""
    ax = torch.arange(n, dtype=torch.float64, device="cuda")
    k, j, i = torch.meshgrid(ax, ax, ax, indexing="ij")
    cells = torch.stack([i, j, k], dim=-1).reshape(-1, 1, 3)
    r = ((cells + torch.tensor(basis, dtype=torch.float64, device="cuda")) * a).reshape(-1, 3)
    if noise > 0.0:
        r = r + noise * torch.randn(r.shape, dtype=torch.float64, device="cuda", generator=g)
        r = torch.remainder(r, n * a)
        r = torch.where(r >= n * a, torch.zeros_like(r), r)
    return r


def _velocities(count, kt_over_m, g):
    v = torch.randn((count, 3), dtype=torch.float64, device="cuda", generator=g)
    v -= v.mean(dim=0)
    return v * math.sqrt(kt_over_m * (3.0 * count - 3.0) / float((v * v).sum()))


def _cell_order(r, geom):
    d, cs = geom["dims"][0], geom["cell_size"]
    c = torch.clamp(torch.floor(r / cs).long(), 0, d - 1)
    return torch.argsort((c[:, 2] * d + c[:, 1]) * d + c[:, 0], stable=True)


def _columns(r, v):
    t = torch.cat([r, v], dim=1).t().contiguous().cpu().numpy()
    return dict(zip(("rx", "ry", "rz", "vx", "vy", "vz"), t))


def _lj_inputs(n, rho, temp, noise, g, sort=False):
    a = (4.0 / rho) ** (1.0 / 3.0)
    geom = _geometry(n * a, RCUT + SKIN)
    r = _lattice(FCC, n, a, noise, g)
    v = _velocities(len(r), temp, g)
    if sort:
        r = r[_cell_order(r, geom)].contiguous()
    return r, v, geom


def _cells(geom):
    return geom["dims"][0] * geom["dims"][1] * geom["dims"][2]


class _Device:
    """A device array of a batch as torch sees it (no copy); the tensor made from it keeps the batch."""

    def __init__(self, batch, pointer, count, typestr):
        self.batch = batch
        self.__cuda_array_interface__ = {"shape": (int(count),), "typestr": typestr, "data": (int(pointer), False),
                                         "version": 3, "strides": None}


def _tensor(batch, pointer, count, typestr):
    return torch.as_tensor(_Device(batch, pointer, count, typestr), device="cuda")


def _views(batch, s, names):
    """The system's resident arrays as tensors, in the library's storage order."""
    v = batch.pair_view(s)
    kinds = {"id": "<i8", "nbr_count": "<i4", "nbr_half": "<i4", "nbr_start": "<i4"}
    return {k: _tensor(batch, getattr(v, k), v.n_particles, kinds.get(k, "<f8")) for k in names}


STATE = ("rx", "ry", "rz", "vx", "vy", "vz", "fx", "fy", "fz", "id")


# ---------------------------------------------------------------------------
def prepare(case, seed):
    g = _generator(seed)
    kind = case["kind"]
    if kind in ("md", "request"):
        r, v, geom = _lj_inputs(case["n"], case["rho"], case["T"], 0.0, g)
        count = len(r)
        state = {"case": case, "cols": _columns(r, v), "ids": np.arange(count, dtype=np.uint64),
                 "params": xnb.lj_params(geom), "precision": xnb.PRECISIONS[case["precision"]]}
        stream = torch.cuda.Stream()
        state["stream"] = stream
        batch = xnb.Batch(count, _cells(geom), 200 * count + 64, stream=stream.cuda_stream)
        state["batch"] = batch
        if kind == "md":
            s = batch.add_system_soa(state["params"], state.pop("cols"), state.pop("ids"))
            batch.init_particles(s, state["precision"])
            state["out"] = _views(batch, s, STATE)
            state["graph"] = batch.graph(case["steps"], state["precision"]) if case["graph"] else None
        return state
    if kind == "ensemble":
        # sizes spread evenly over their range, in an order of their own; the state points from the seed
        ns = np.rint(np.linspace(case["nmin"], case["nmax"], case["systems"])).astype(int)
        ns = np.random.default_rng(case["systems"]).permutation(ns)
        rng = np.random.default_rng(int(seed))
        rhos, temps = rng.uniform(0.70, 1.00, len(ns)), rng.uniform(0.7, 1.5, len(ns))
        made = [_lj_inputs(int(n), float(rho), float(t), 0.0, g) for n, rho, t in zip(ns, rhos, temps)]
        total, cells = sum(len(r) for r, _, _ in made), sum(_cells(geom) for _, _, geom in made)
        stream = torch.cuda.Stream()
        batch = xnb.Batch(total, cells, 200 * total + 64 * len(made), max_systems=len(made), stream=stream.cuda_stream)
        systems = [batch.add_system_soa(xnb.lj_params(geom), _columns(r, v), np.arange(len(r), dtype=np.uint64))
                   for r, v, geom in made]
        batch.init_particles(-1, xnb.PRECISIONS[case["precision"]])
        first = batch.pair_view(systems[0])  # the systems lie one after the other in the batch's arrays
        out = {k: _tensor(batch, getattr(first, k), total, "<i8" if k == "id" else "<f8") for k in STATE}
        return {"case": case, "batch": batch, "stream": stream, "out": out,
                "graph": batch.graph(case["steps"], xnb.PRECISIONS[case["precision"]])}
    if kind in ("force", "build"):
        r, v, geom = _lj_inputs(case["n"], case["rho"], 1.0, 0.07, g, sort=True)
        count = len(r)
        batch = xnb.Batch(count, _cells(geom), 200 * count + 64)
        s = batch.add_system_soa(xnb.lj_params(geom), _columns(r, v), np.arange(count, dtype=np.uint64))
        state = {"case": case, "batch": batch, "s": s}
        if kind == "force":
            state["precision"] = xnb.PRECISIONS[case["precision"]]
            batch.init_particles(s, state["precision"])
            state["out"] = _views(batch, s, ("fx", "fy", "fz") + (("pe",) if case["energy"] else ()))
        else:
            batch.init_particles(s, xnb.PREC_MIXED)
            state["out"] = _views(batch, s, ("nbr_count", "nbr_half", "nbr_start"))
            # the whole list segment; what lies past a particle's count is not part of its list
            state["out"]["nbr"] = _tensor(batch, batch.pair_view(s).nbr, batch.info(s).list_cap, "<i4")
            state["out"]["nbr"].zero_()
        return state
    if kind == "snap":
        basis, a, mass, noise = SNAP[case["element"]]
        files = os.path.join(ROOT, "tests", "golden", "snap", case["element"] + "_Zuo_JPCA2020.snap")
        cfg = snap.read_lammps(files + "param", files + "coeff")
        r = _lattice(basis, case["n"], a, noise, g)
        kb = snap.energy_unit() * 8.617333262e-5
        v = _velocities(len(r), kb * 300.0 / mass, g)
        skin, d = 2.0, case["n"] // 4  # the decks' skin, and their cells of four unit cells
        geom = {"origin": (0.0, 0.0, 0.0), "extent": (case["n"] * a,) * 3, "dims": (d,) * 3,
                "cell_size": case["n"] * a / d}
        r = r[_cell_order(r, geom)].contiguous()
        batch = xnb.Batch(len(r), _cells(geom), 400 * len(r) + 64)
        s = batch.add_system_soa(xnb.lj_params(geom, rcut=cfg["rcutfac"], rcut_inc=skin, dt=2e-3, mass=mass,
                                               divide_by_mass=True),
                                 _columns(r, v), np.arange(len(r), dtype=np.uint64))
        batch.init_particles(s, xnb.PREC_FP64)
        pot = snap.Potential(cfg)
        pot.force(batch, s, energy=True, mixed=case["mixed"])
        names = STATE if case["md"] else ("fx", "fy", "fz")
        return {"case": case, "batch": batch, "s": s, "pot": pot,
                "out": _views(batch, s, names + (("pe",) if case["energy"] else ()))}
    raise ValueError("unknown kind of case: %s" % kind)


def run(state):
    case, batch = state["case"], state["batch"]
    kind = case["kind"]
    if kind in ("md", "ensemble"):
        if state["graph"] is not None:
            state["graph"].launch()
        else:
            batch.step(case["steps"], state["precision"])
    elif kind == "force":
        batch.lennard_jones_force(state["s"], state["precision"], energy=case["energy"])
    elif kind == "build":
        batch.chunk_neighbors(state["s"])
    elif kind == "snap":
        if case["md"]:
            snap.md_steps(batch, state["s"], state["pot"], 1, energy=case["energy"], mixed=case["mixed"])
        else:
            state["pot"].force(batch, state["s"], energy=case["energy"], mixed=case["mixed"])
    else:
        s = batch.add_system_soa(state["params"], state["cols"], state["ids"])
        batch.init_particles(s, state["precision"])
        batch.step(case["steps"], state["precision"], 0)
        batch.check_errors()
        out = batch.download(s)
        batch.remove_system(s)
        del out["pe"]  # written by steps that ask for energies only
        return out
    return state["out"]


# ---------------------------------------------------------------------------
def _atoms(case):
    if case["kind"] == "ensemble":
        sizes = np.arange(case["nmin"], case["nmax"] + 1, dtype=np.float64)
        return case["systems"] * 4.0 * float((sizes**3).mean())
    return float((2 if case.get("element") == "Mo" else 4) * case["n"] ** 3)


def _snap_flops(twojmax, neighbours):
    """Per atom: the U recursion and its adjoint on the unique half (64 flop per neighbour and element) and the
    Clebsch-Gordan contractions of the unique Z elements (12 flop per product)."""
    nu = sum(((j // 2) * (j + 1) + j // 2 + 1) if j % 2 == 0 else ((j + 1) // 2) * (j + 1) for j in range(twojmax + 1))
    terms = 0
    for j1 in range(twojmax + 1):
        for j2 in range(j1 + 1):
            for j in range(j1 - j2, min(twojmax, j1 + j2) + 1, 2):
                per = [min(j1, (2 * m - j + j2 + j1) // 2) - max(0, (2 * m - j - j2 + j1) // 2) + 1
                       for m in range(j + 1)]
                terms += sum(per[mb] * per[ma] for mb in range(j // 2 + 1) for ma in range(j + 1)
                             if 2 * mb < j or ma <= mb)
    return 64.0 * neighbours * nu + 12.0 * terms


def work(case):
    n, kind = _atoms(case), case["kind"]
    rho = case.get("rho", 0.85)
    steps = case.get("steps", 1)
    pair = 0.5 * 8.0 * PAIRS * 2.0 * 1.405 * rho + 24.0 * PAIRS * rho  # listed distances, then pairs within rc
    if kind in ("md", "ensemble", "request"):
        # state in and out once; each pair of every step
        return {"bytes": n * 8.0 * (6 + 9), "flops": n * steps * (pair + 18.0)}
    if kind == "force":
        lists = 4.0 * 2.0 * 1.405 * PAIRS * rho  # the neighbour list is an input of the operator
        return {"bytes": n * (24.0 + lists + 24.0 + (8.0 if case["energy"] else 0.0)), "flops": n * pair}
    if kind == "build":
        nbh = RCUT + SKIN
        return {"bytes": n * (24.0 + 12.0 + 4.0 * 4.18879020478639 * nbh**3 * rho),
                "flops": n * 8.0 * 27.0 * nbh**3 * rho}
    twojmax, neighbours = (8, 42) if case["element"] == "Ni" else (6, 58)
    return {"bytes": n * 8.0 * ((6 + 9) if case["md"] else (3 + 3)), "flops": n * _snap_flops(twojmax, neighbours)}


# ---------------------------------------------------------------------------
def exact(case, seed):
    """lennard_jones_force in plain FP64 torch: an exhaustive search of each particle's 27 cells."""
    if case["kind"] != "force":
        return None
    r, _, geom = _lj_inputs(case["n"], case["rho"], 1.0, 0.07, _generator(seed), sort=True)
    count, d, length = len(r), geom["dims"][0], geom["extent"][0]
    c = torch.clamp(torch.floor(r / geom["cell_size"]).long(), 0, d - 1)
    n_in = torch.bincount((c[:, 2] * d + c[:, 1]) * d + c[:, 0], minlength=d**3)
    start = torch.cumsum(n_in, 0) - n_in
    f = torch.zeros_like(r)
    pe = torch.zeros(count, dtype=torch.float64, device="cuda")
    shift6 = RCUT**-6
    e_cut = 4.0 * (shift6 * shift6 - shift6)
    for o in range(27):
        nb = c + torch.tensor([o % 3 - 1, (o // 3) % 3 - 1, o // 9 - 1], device="cuda")
        wrapped = torch.remainder(nb, d)
        shift = (nb - wrapped).double() * (length / d)
        cell = (wrapped[:, 2] * d + wrapped[:, 1]) * d + wrapped[:, 0]
        first, have = start[cell], n_in[cell]
        for m in range(int(n_in.max())):
            j = torch.where(m < have, first + m, 0)
            dr = r[j] + shift - r
            d2 = (dr * dr).sum(dim=1)
            ok = (m < have) & (d2 > 0.0) & (d2 <= RCUT * RCUT)
            inv = 1.0 / torch.where(ok, d2, 1.0)
            s6 = inv * inv * inv
            f += torch.where(ok, 24.0 * s6 * (1.0 - 2.0 * s6) * inv, 0.0)[:, None] * dr
            pe += torch.where(ok, 0.5 * (4.0 * s6 * (s6 - 1.0) - e_cut), 0.0)
    out = {"fx": f[:, 0].contiguous(), "fy": f[:, 1].contiguous(), "fz": f[:, 2].contiguous()}
    if case["energy"]:
        out["pe"] = pe
    return out
