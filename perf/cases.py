"""Performance cases of the tensormd force path, through its Python entry points.

A case is one of the calls that a user's program makes, over the potentials,
lattices and sizes of this repository's benchmark, tests and shipped examples:

  step    positions handed over, forces, energy and virial back: what LAMMPS
          does each MD step (set_positions + compute), periodic or, with
          `ghost`, a rank's local atoms plus the ghosts of its neighbours
  pair    a new configuration through the pair-style object (PairTensorMD
          .compute: atoms uploaded, list built, per-atom energies and virials)
  nve     a device-resident MD segment (set_atoms, nve_run, get)
  nvt     the same under fix nvt
  batch   many small periodic cells evaluated once (a data set of structures)
  bnve    an MD segment of many small periodic cells
  serve   a burst of single-point, NVE and FIRE jobs through the job server

run() returns what the calls return.  exact() is the same mathematics in plain
torch at 64 bits (neighbour search, descriptor, MLP, autograd forces, velocity
Verlet, Nose-Hoover chain).
"""
import math
import sys
import tempfile
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parent.parent
sys.path.insert(0, str(ROOT / "lammps-tensormd_b200"))

from tmd_b200 import (PairTensorMD, TensorMDBatch, TensorMDModel,  # noqa: E402
                      TensorMDServer, TensorMDSystem, synth)

GOLDEN = ROOT / "tests" / "golden"
SKIN = 1.0
DT = 0.001
BOLTZ, MVV2E = 8.617343e-5, 1.0364269e-4  # metal units

# potentials: the shipped trained ones (file, elements), and random-weight
# ones of the benchmark's and tests' shapes
SHIPPED = {"MoNi_m3": ("MoNi_m3.npz", "Mo Ni"),
           "MoNi_sp": ("MoNi_squareplus_500k.npz", "Mo Ni"),
           "AlMgSi": ("AlMgSi.24aug13.npz", "Al Mg Si"),
           "W_k32": ("W_k32_snapshot.npz", "W"),
           "W_k64": ("W_m3_k64_n128_squareplus.npz", "W")}
RANDOM = {"tanh16": dict(num_filters=16, rc=6.0, hidden=(64, 64), actfn=2),
          "soft32": dict(num_filters=32, rc=6.5, hidden=(128, 128, 128), actfn=1),
          "res8": dict(num_filters=8, rc=5.5, hidden=(32, 32, 32), actfn=1, resnet=1),
          "rank2": dict(num_filters=8, rc=5.5, hidden=(64, 64), actfn=2, max_moment=2)}
# structures of the shipped potentials and of the random-weight ones
CELL_FILES = {"MoNi_m3": "Mo8_Ni8_id3210.data", "MoNi_sp": "Mo8_Ni8_id3210.data",
              "AlMgSi": "AlMgSi.data"}
LATTICE = {"W_k32": ("bcc", 3.189), "W_k64": ("bcc", 3.189)}


def _case(name, kind, pot, **kw):
    c = dict(kind=kind, pot=pot, nelt=1, lattice="", nx=1, ny=1, nz=1, drop=0, sigma=0.05,
             T=300.0, steps=0, precision="fp32", ghost=False, ncells=0, nmin=0, nmax=0)
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: one 16-atom triclinic cell of the shipped MoNi
        # potential (its example's unit cell), where launches are the cost
        _case("step MoNi 16", "step", "MoNi_m3", nelt=2),
        # one configuration of a training or test set, shipped three-element
        # potential, 2 x 2 x 1 of its 108-atom cell with two vacancies
        _case("pair AlMgSi 430", "pair", "AlMgSi", nelt=3, nx=2, ny=2, drop=2),
        # the 4,000-atom FCC cell of the plain configuration, short MD
        _case("nve fcc 4k", "nve", "tanh16", lattice="fcc", nx=10, ny=10, nz=10, steps=50),
        # the reference's own speed benchmark: W_k32, 23,040 atoms, fix nvt 300 K
        _case("nvt W 23k", "nvt", "W_k32", lattice="bcc", nx=24, ny=24, nz=20, sigma=0.0,
              steps=50),
        # the headline BCC cell as LAMMPS drives it, one step
        _case("step bcc 128k", "step", "tanh16", lattice="bcc", nx=40, ny=40, nz=40,
              sigma=0.08),
        # the headline: the same cell, device-resident NVE at 600 K
        _case("nve bcc 128k", "nve", "tanh16", lattice="bcc", nx=40, ny=40, nz=40, sigma=0.08,
              T=600.0, steps=50),
        # one rank of a domain-decomposed LAMMPS run: half of a two-element
        # FCC cell and its ghosts
        _case("step ghost 16k", "step", "tanh16", nelt=2, lattice="fcc", nx=20, ny=20, nz=20,
              ghost=True),
        # a data set of 256 ragged small cells, forces and energies once
        _case("batch 256 cells", "batch", "tanh16", nelt=2, ncells=256, nmin=32, nmax=512),
        # the batch configuration: 4,096 cells of 256 atoms, NVE
        _case("bnve 4096 cells", "bnve", "tanh16", nelt=2, ncells=4096, nmin=256, nmax=256,
              steps=20),
        # the precision configuration in the plain form: a 4-element alloy of
        # 432,000 atoms, wide MLP
        _case("step alloy 432k", "step", "soft32", nelt=4, lattice="fcc", nx=60, ny=60, nz=30),
        # the same potential on 55,296 atoms with the split-BF16 tensor-core MLP
        _case("step alloy 55k x3", "step", "soft32", nelt=4, lattice="fcc", nx=24, ny=24, nz=24,
              precision="bf16x3"),
        # a burst of serving jobs: 60% single points, 25% NVE, 15% FIRE
        _case("serve 64 jobs", "serve", "tanh16", nelt=4, ncells=64, nmin=32, nmax=1024,
              steps=20),
    ]


def _logu(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "pair", "nve", "nvt", "batch", "bnve", "serve"])
    if kind in ("batch", "bnve", "serve"):
        nelt = rng.randint(1, 4) if kind != "serve" else 4
        ncells = int(_logu(rng, 16, 64 if kind == "serve" else 2048))
        nmin = rng.randint(24, 64)
        nmax = rng.randint(nmin + 8, 600)
        return _case("", kind, "tanh16", nelt=nelt, ncells=ncells, nmin=nmin, nmax=nmax,
                     precision=rng.choice(["fp32", "fp32", "bf16x3"]),
                     steps=0 if kind == "batch" else rng.randint(5, 20))
    pots = ["tanh16", "tanh16", "soft32", "res8", "rank2", "W_k32", "W_k64", "MoNi_m3",
            "MoNi_sp", "AlMgSi"]
    pot = rng.choice(pots)
    n = int(_logu(rng, 16, 200000 if kind == "step" or (kind, pot) == ("nve", "tanh16") else 20000))
    kw = dict(sigma=rng.choice([0.03, 0.05, 0.1]), T=rng.choice([300.0, 600.0]))
    if pot in CELL_FILES:
        per = 16 if pot.startswith("MoNi") else 108
        kw["nelt"] = 3 if pot == "AlMgSi" else 2
        side = (min(n, 40000) / per) ** (1 / 3)
    else:
        kw["lattice"] = "bcc" if pot in LATTICE else rng.choice(["fcc", "bcc"])
        if pot in RANDOM:
            kw["nelt"] = rng.choice([1, 2, 4] if pot == "tanh16" else [4] if pot == "soft32"
                                    else [2])
        per = 4 if kw["lattice"] == "fcc" else 2
        side = (min(n, 60000 if pot == "W_k64" else n) / per) ** (1 / 3)
    low = 1 if pot in CELL_FILES else 3
    kw["nx"] = max(low, round(side * rng.uniform(0.7, 1.0)))
    kw["ny"] = max(low, round(side * rng.uniform(0.8, 1.1)))
    kw["nz"] = max(low, round(side))
    kw["drop"] = rng.randint(0, 3) if per * kw["nx"] * kw["ny"] * kw["nz"] > 40 else 0
    if kind in ("nve", "nvt"):
        kw["steps"] = rng.randint(10, 50)
    if kind == "step":
        if pot in ("tanh16", "soft32"):
            kw["precision"] = rng.choice(["fp32", "fp32", "tf32x3", "bf16x3", "bf16"])
        if pot in RANDOM and min(kw["nx"], kw["ny"], kw["nz"]) >= 8 and rng.random() < 0.3:
            kw["ghost"] = True
    return _case("", kind, pot, **kw)


# ---------------------------------------------------------------- inputs

def _potential(case):
    """(npz path, pair_coeff arguments)."""
    if case["pot"] in SHIPPED:
        f, el = SHIPPED[case["pot"]]
        return GOLDEN / f, f"{GOLDEN / f} {el} interp 0.001"
    path = Path(tempfile.mkdtemp(prefix="tmdperf")) / f"{case['pot']}.npz"
    syms = synth.gaussian_potential(path, nelt=case["nelt"], seed=1234,
                                    **{"max_moment": 3, **RANDOM[case["pot"]]})
    args = f"{path} {' '.join(syms)}"
    return path, args if case["precision"] == "fp32" else args + f" precision {case['precision']}"


def _structure(case, seed):
    """x, types (1-based), box of one periodic cell."""
    rng = np.random.default_rng([seed, 1])
    rep = (case["nx"], case["ny"], case["nz"])
    if case["pot"] in CELL_FILES:
        x0, t0, b0 = synth.read_data(GOLDEN / CELL_FILES[case["pot"]])
        x0 = synth.frac_wrap(x0, b0)
        h = _cell(b0)
        g = np.stack(np.meshgrid(*(np.arange(k) for k in rep), indexing="ij"), -1).reshape(-1, 3)
        x = (x0[None] + (g @ h)[:, None]).reshape(-1, 3)
        t = np.tile(t0, len(g))
        box = b0.copy()
        box[3], box[4], box[5] = b0[3] * rep[0], b0[4] * rep[1], b0[5] * rep[2]
        box[6], box[7], box[8] = b0[6] * rep[1], b0[7] * rep[2], b0[8] * rep[2]
    else:
        kind = case["lattice"]
        a = LATTICE[case["pot"]][1] if case["pot"] in LATTICE else {"fcc": 3.6, "bcc": 2.87}[kind]
        x, box = synth.lattice(kind, a, *rep)
        t = np.arange(len(x)) % case["nelt"] + 1
        rng.shuffle(t)
    if case["drop"]:
        keep = np.sort(rng.permutation(len(x))[case["drop"]:])
        x, t = x[keep], t[keep]
    if case["sigma"] > 0:
        x = x + rng.normal(0.0, case["sigma"], size=x.shape)
    return synth.frac_wrap(x, box), t.astype(np.int32), box


def _ghosts(x, t, box, cut):
    """The local atoms of the lower half in x and every periodic image within
    `cut` of it (what LAMMPS's border exchange hands a rank)."""
    L, half = box[3:6], box[3] / 2
    loc = x[:, 0] < half
    gx, gt = [x[loc]], [t[loc]]
    for s in np.ndindex(3, 3, 3):
        sh = (np.array(s) - 1) * L
        p = x + sh
        ok = ((p >= -cut) & (p < np.array([half, L[1], L[2]]) + cut)).all(1)
        if not sh.any():
            ok &= ~loc
        gx.append(p[ok])
        gt.append(t[ok])
    return np.concatenate(gx), np.concatenate(gt), int(loc.sum())


def _jobs(case, seed):
    """Small cells: x, types, box, v and a job kind each.  A batch takes FCC
    and BCC cells; the server's burst random packings too."""
    rng = np.random.default_rng([seed, 2])
    shape = np.random.default_rng([case["ncells"], case["nmin"], case["nmax"]])
    nelt, out = case["nelt"], []
    for c in range(case["ncells"]):
        n = int(round(math.exp(shape.uniform(math.log(case["nmin"]), math.log(case["nmax"] + 1)))))
        form = int(shape.integers(3 if case["kind"] == "serve" else 2))
        kind = int(shape.choice([0, 1, 2], p=[0.6, 0.25, 0.15]))
        if case["nmin"] == case["nmax"] == 256:
            rep = (4, 4, 4) if c % 2 == 0 else (4, 4, 8)
            x, box = synth.lattice("fcc" if c % 2 == 0 else "bcc", 3.6 if c % 2 == 0 else 2.87,
                                   *rep)
        elif form == 2:
            x, box = synth.random_packing(min(n, 256), rng)
        else:
            per, a = (4, 3.6) if form == 0 else (2, 2.87)
            x, box = synth.lattice("fcc" if form == 0 else "bcc", a,
                                   *synth._near_cubic(max(n, 4 * per) / per))
        sig = 0.1 if case["kind"] == "bnve" else 0.05
        if form != 2:
            x = x + rng.normal(0.0, sig, size=x.shape)
        x = synth.frac_wrap(x, box)
        t = rng.integers(1, nelt + 1, size=len(x)).astype(np.int32)
        m = np.array([synth.MASSES[s] for s in synth.SYMBOLS[:nelt]])[t - 1]
        v = synth.maxwell(m, rng.uniform(300.0, 1200.0), rng)
        out.append((kind, x, t, box, v))
    return out


def _pinned(a):
    p = torch.empty(a.shape, dtype=torch.float64, pin_memory=True)
    p.copy_(torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)))
    return p


def prepare(case, seed):
    kind = case["kind"]
    _, args = _potential(case)
    s = {"case": case}
    if kind == "pair":
        s["x"], s["t"], s["box"] = _structure(case, seed)
        s["pair"] = PairTensorMD(skin=SKIN)
        s["pair"].settings()
        s["pair"].coeff("* * " + args)
        return s
    model = s["model"] = TensorMDModel(args)
    if kind in ("batch", "bnve", "serve"):
        jobs = _jobs(case, seed)
        if kind == "serve":
            s["jobs"] = jobs
            s["server"] = TensorMDServer(model, max_atoms=100000, max_cells=256, skin=SKIN,
                                         steps_per_tick=8)
            return s
        s["batch"] = TensorMDBatch(model, [len(j[1]) for j in jobs], SKIN)
        s["batch"].set_cells(np.stack([j[3] for j in jobs]))
        s["x"], s["t"], s["v"] = (np.concatenate([j[q] for j in jobs]) for q in (1, 2, 4))
        return s
    x, t, box = _structure(case, seed)
    if case["ghost"]:
        x, t, nloc = _ghosts(x, t, box, model.cutmax + SKIN)
        s["system"] = TensorMDSystem(model, len(x), SKIN)
        s["system"].set_atoms_ghost(nloc, x, t)
    else:
        s["system"] = TensorMDSystem(model, len(x), SKIN)
        s["system"].set_box(box)
    if kind == "step":
        if not case["ghost"]:
            s["system"].set_atoms(x, t)
        s["pin"] = _pinned(x)
        s["x"] = s["pin"].numpy()
        return s
    m = np.asarray(model.type_mass)[t]
    s["x"], s["t"] = x, t
    s["v"] = synth.maxwell(m, case["T"], np.random.default_rng([seed, 3]))
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "step":
        s["system"].set_positions(s["x"])
        return s["system"].compute(1, 1)
    if kind == "pair":
        p = s["pair"]
        f = p.compute(s["x"], s["t"], s["box"], eflag=1, vflag=1, eflag_atom=1, vflag_atom=1)
        return {"energy": p.eng_vdwl, "virial": p.virial, "f": f, "eatom": p.eatom,
                "vatom": p.vatom}
    if kind in ("nve", "nvt"):
        q = s["system"]
        q.set_atoms(s["x"], s["t"], s["v"])
        if kind == "nve":
            th = q.nve_run(case["steps"], DT, thermo_every=10)
        else:
            th = q.nvt_run(case["steps"], DT, case["T"], case["T"], 0.1, thermo_every=10)
        x, v, f, image = q.get()
        return {"thermo": th, "x": x, "v": v, "f": f, "image": image}
    if kind == "batch":
        s["batch"].set_atoms(s["x"], s["t"])
        return s["batch"].compute()
    if kind == "bnve":
        b = s["batch"]
        b.set_atoms(s["x"], s["t"], s["v"])
        th = b.nve_run(case["steps"], DT, thermo_every=case["steps"])
        x, v, f, image = b.get()
        return {"thermo": th, "x": x, "v": v, "f": f, "image": image}
    srv = s["server"]
    tickets = [srv.submit(k, x, t, box, v=v if k == 1 else None, nsteps=case["steps"], dt=DT,
                          fmax=1e-6) for k, x, t, box, v in s["jobs"]]
    done = [srv.wait(tk) for tk in tickets]
    out = {}
    for kind, name in enumerate(("single", "nve", "fire")):
        some = [d for (k, *_), d in zip(s["jobs"], done) if k == kind]
        if some:
            out[name] = {key: np.concatenate([np.atleast_1d(d[key]) for d in some])
                         for key in ("energy", "virial", "f", "x", "v", "steps")}
    return out


# ---------------------------------------------------------------- work

def _counts(case):
    """atoms, pairs inside the cutoff per atom, K, D, elements, MLP widths."""
    if case["pot"] in SHIPPED:
        k, hid = {"MoNi_m3": (64, [64] * 4), "MoNi_sp": (64, [64] * 4), "AlMgSi": (64, [64] * 3),
                  "W_k32": (32, [128] * 3), "W_k64": (64, [128] * 4)}[case["pot"]]
        mm, rc = 3, 6.0
    else:
        p = RANDOM[case["pot"]]
        k, hid, mm, rc = p["num_filters"], list(p["hidden"]), p.get("max_moment", 3), p["rc"]
    rep = case["nx"] * case["ny"] * case["nz"]
    if case["kind"] in ("batch", "bnve", "serve"):
        lo, hi = case["nmin"], case["nmax"] + 1
        n = case["ncells"] * (hi - lo) / math.log(hi / lo)
        dens = 0.085
    elif case["pot"] in CELL_FILES:
        _, t, b = synth.read_data(GOLDEN / CELL_FILES[case["pot"]])
        n, dens = len(t) * rep - case["drop"], len(t) / (b[3] * b[4] * b[5])
    else:
        per = 4 if case["lattice"] == "fcc" else 2
        a = LATTICE[case["pot"]][1] if case["pot"] in LATTICE else (3.6 if per == 4 else 2.87)
        n, dens = per * rep - case["drop"], per / a ** 3
        if case["ghost"]:
            n = n / 2
    d = {1: 4, 2: 10, 3: 20}[mm]
    return n, dens * 4 / 3 * math.pi * rc ** 3, k, d, case["nelt"], [case["nelt"] * k * (mm + 1)] + hid


def work(case):
    n, pairs, k, d, nelt, net = _counts(case)
    evals = 1 + case["steps"] if case["kind"] in ("nve", "nvt", "bnve") else \
        1 + 0.4 * case["steps"] if case["kind"] == "serve" else 1
    # per pair: P, V and W contractions, radial basis and angular terms; per
    # atom: the MLP forward and backward
    mlp = 4 * sum(a * b for a, b in zip(net, net[1:])) + 4 * net[-1]
    flops = evals * n * (pairs * (6 * k * d + 14 * k + 11 * d) + mlp)
    # positions and types in, forces out; in MD positions and velocities are
    # read and written every step
    bytes_ = n * 52 + (evals - 1) * n * 120
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    # four times the largest distance from exact() over 60 cases of the
    # ranges: FP32 arithmetic 4.6e-5 (forces of barely displaced shipped
    # cells, where FP32 terms of eV/A cancel) and 6.1e-5 (virials of nearly
    # perfect lattices), the split tensor-core forms no more; plain BF16
    # 4e-3 in forces, 8e-3 in virials
    rel = 2.5e-2 if case["precision"] == "bf16" else 2.5e-4
    return {"rel": rel, "max": min(0.9, 60 * rel)}


# ---------------------------------------------------------------- 64-bit reference

def _cell(box):
    return np.array([[box[3], 0, 0], [box[6], box[4], 0], [box[7], box[8], box[5]]], dtype=float)


def _pairs(x, box, rc, periodic=True, rows=None):
    """(i, j, x_j + image - x_i) of every pair inside rc, sorted by i."""
    dev = x.device
    n = len(x)
    rows = n if rows is None else rows
    if periodic:
        h = torch.tensor(_cell(box), device=dev)
        lo = torch.tensor(np.asarray(box[:3], dtype=float), device=dev)
        hn = _cell(box)
    else:
        lo = x.min(0).values - 1.0
        hn = np.diag((x.max(0).values - lo + 1.0).cpu().numpy())
        h = torch.tensor(hn, device=dev)
    vol = abs(np.linalg.det(hn))
    w = [vol / np.linalg.norm(np.cross(hn[(a + 1) % 3], hn[(a + 2) % 3])) for a in range(3)]
    nb = [max(1, int(v / rc)) for v in w]
    ns = [math.ceil(rc / (v / b) - 1e-12) for v, b in zip(w, nb)]
    frac = (x - lo) @ torch.linalg.inv(h)
    wrap = torch.floor(frac) if periodic else torch.zeros_like(frac)
    xw = x - wrap @ h
    nbt = torch.tensor(nb, device=dev)
    b3 = torch.minimum(((frac - wrap) * nbt).long().clamp_(min=0), nbt - 1)
    flat = (b3[:, 0] * nb[1] + b3[:, 1]) * nb[2] + b3[:, 2]
    order = torch.argsort(flat)
    count = torch.bincount(flat, minlength=nb[0] * nb[1] * nb[2])
    start = torch.cumsum(count, 0) - count
    m = int(count.max())
    lane = torch.arange(m, device=dev)
    offs = [(a, b, c) for a in range(-ns[0], ns[0] + 1) for b in range(-ns[1], ns[1] + 1)
            for c in range(-ns[2], ns[2] + 1)]
    got = []
    step = max(1, 20_000_000 // m)
    for r0 in range(0, rows, step):
        r1 = min(rows, r0 + step)
        for o in offs:
            tb = b3[r0:r1] + torch.tensor(o, device=dev)
            sh = torch.div(tb, nbt, rounding_mode="floor")
            inside = torch.ones(r1 - r0, dtype=torch.bool, device=dev) if periodic else \
                (sh == 0).all(1)
            wb = tb - sh * nbt
            fb = (wb[:, 0] * nb[1] + wb[:, 1]) * nb[2] + wb[:, 2]
            slot = start[fb][:, None] + lane
            ok = (lane < count[fb][:, None]) & inside[:, None]
            j = order[slot.clamp_(max=n - 1)]
            d = xw[j] + (sh.double() @ h)[:, None] - xw[r0:r1, None]
            r2 = (d * d).sum(-1)
            ok &= (r2 < rc * rc) & (r2 > 1e-10)
            k = ok.nonzero(as_tuple=True)
            got.append((k[0] + r0, j[k], d[k]))
    i, j, d = (torch.cat([g[q] for g in got]) for q in range(3))
    o = torch.argsort(i, stable=True)
    return i[o], j[o], d[o]


class _Exact:
    """Energy, forces and virial of a potential file in 64 bits."""

    MONO = [(), (0,), (1,), (2,), (0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2),
            (0, 0, 0), (0, 0, 1), (0, 0, 2), (0, 1, 1), (0, 1, 2), (0, 2, 2), (1, 1, 1),
            (1, 1, 2), (1, 2, 2), (2, 2, 2)]

    def __init__(self, path):
        with np.load(path) as z:
            self.z = {k: z[k] for k in z.files}
        g = lambda k: int(np.asarray(self.z[k]).ravel()[0])  # noqa: E731
        self.rc = float(np.asarray(self.z["rmax"]).ravel()[0])
        self.nelt, self.mm, self.nl, self.act = g("nelt"), g("max_moment"), g("nlayers"), g("actfn")
        self.res, self.outb, self.fnn = g("use_resnet_dt"), g("apply_output_bias"), g("use_fnn")
        self.mass = np.asarray(self.z["masses"], dtype=float)
        self.D = {1: 4, 2: 10, 3: 20}[self.mm]
        # multiplicity of each monomial in the full tensor of its rank
        mult = [math.factorial(len(q)) // math.prod(math.factorial(q.count(a)) for a in range(3))
                for q in self.MONO]
        self.T = torch.zeros(self.mm + 1, self.D, dtype=torch.float64, device="cuda")
        for d in range(self.D):
            self.T[len(self.MONO[d]), d] = mult[d]

    def w(self, key):
        return torch.tensor(np.asarray(self.z[key], dtype=float), device="cuda")

    @staticmethod
    def phi(kind, y):
        if kind == 1:
            return torch.nn.functional.softplus(y, threshold=34.0)
        if kind == 2:
            return torch.tanh(y)
        return 0.5 * (y + torch.sqrt(y * y + 4.0))

    def radial(self, r):
        fc = 0.5 + 0.5 * torch.cos(math.pi * torch.clamp(r / self.rc, max=1.0))
        if not self.fnn:
            eta, om = self.w("descriptor::eta"), self.w("descriptor::omega")
            return fc[..., None] * torch.exp(-eta * (r[..., None] - om) ** 2 / self.rc ** 2)
        y, nl = r[..., None], int(self.z["fnn::nlayers"])
        act = int(self.z["fnn::actfn"])
        for q in range(nl):
            wt = self.w(f"fnn::weights_0_{q}")
            y = y @ wt.reshape(y.shape[-1], -1)
            if q < nl - 1:
                y = self.phi(act, y + self.w(f"fnn::biases_0_{q}"))
            elif int(self.z["fnn::apply_output_bias"]):
                y = y + self.w(f"fnn::biases_0_{q}")
        return fc[..., None] * y

    def net(self, g, e):
        for q in range(self.nl):
            w = self.w(f"weights_{e}_{q}").reshape(g.shape[-1], -1)
            y = g @ w
            if q < self.nl - 1 or self.outb:
                y = y + self.w(f"biases_{e}_{q}").reshape(-1)
            if q < self.nl - 1:
                y = self.phi(self.act, y)
                if q > 0 and self.res and w.shape[0] == w.shape[1]:
                    y = y + g
            g = y
        return g.sum(-1)

    def rows(self, d, mask, ei, ej):
        """Atomic energies of padded rows d[A, C, 3] (elements ei[A], ej[A, C])."""
        r = torch.sqrt((d * d).sum(-1))
        u = d / r[..., None]
        hk = self.radial(r) * mask[..., None]
        mono = torch.stack([u[..., list(q)].prod(-1) if q else torch.ones_like(r)
                            for q in self.MONO[:self.D]], -1)
        blocks = []
        for b in range(self.nelt):
            # block 0 is the atom's own element, then the others in order
            eb = ei if b == 0 else torch.where(ei >= b, torch.full_like(ei, b - 1),
                                               torch.full_like(ei, b))
            p = (hk * (ej == eb[:, None])[..., None]).transpose(1, 2) @ mono
            g = (p * p) @ self.T.T
            blocks.append(torch.cat([p[..., :1], g[..., 1:]], -1))
        feat = torch.stack(blocks, 1).flatten(1)
        e = torch.zeros(len(d), dtype=torch.float64, device="cuda")
        for el in range(self.nelt):
            k = (ei == el).nonzero()[:, 0]
            if len(k):
                e = e.index_copy(0, k, self.net(feat[k], el))
        return e

    def forces(self, elem, i, j, d, n, rows=None):
        """(atomic energies, forces, virial rows per atom) from a pair list."""
        rows = n if rows is None else rows
        f = torch.zeros(n, 3, dtype=torch.float64, device="cuda")
        vir = torch.zeros(rows, 6, dtype=torch.float64, device="cuda")
        ea = torch.zeros(rows, dtype=torch.float64, device="cuda")
        cnt = torch.bincount(i, minlength=rows)
        off = torch.cumsum(cnt, 0) - cnt
        c = max(1, int(cnt.max()))
        step = max(1, 400_000 // c)
        ends = torch.cumsum(cnt, 0).cpu().numpy()
        for r0 in range(0, rows, step):
            r1 = min(rows, r0 + step)
            q0, q1 = (int(ends[r0 - 1]) if r0 else 0), int(ends[r1 - 1])
            ii, jj, dd = i[q0:q1], j[q0:q1], d[q0:q1]
            at = (ii - r0, torch.arange(q0, q1, device="cuda") - off[ii])
            pad = torch.ones(r1 - r0, c, 3, dtype=torch.float64, device="cuda")
            mask = torch.zeros(r1 - r0, c, dtype=torch.float64, device="cuda")
            ej = torch.zeros(r1 - r0, c, dtype=torch.long, device="cuda")
            pad[at], mask[at], ej[at] = dd, 1.0, elem[jj]
            pad.requires_grad_(True)
            e = self.rows(pad, mask, elem[r0:r1], ej)
            g = torch.autograd.grad(e.sum(), pad)[0][at]
            ea[r0:r1] = e.detach()
            f.index_add_(0, ii, g)
            f.index_add_(0, jj, -g)
            six = torch.stack([dd[:, a] * g[:, b] for a, b in
                               ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))], -1)
            vir.index_add_(0, ii, -six)
        return ea, f, vir

    def at(self, x, elem, box):
        i, j, d = _pairs(x, box, self.rc)
        return self.forces(elem, i, j, d, len(x))

    def md(self, x, v, types, box, steps, every, nvt=None):
        """Velocity Verlet (with a Nose-Hoover chain of three for nvt = (T,
        damping time)): thermo rows, v, f at the end."""
        elem = torch.tensor(types.astype(np.int64) - 1, device="cuda")
        m = torch.tensor(self.mass, device="cuda")[elem][:, None]
        x, v = torch.tensor(x, device="cuda"), torch.tensor(v, device="cuda")
        dtf = 0.5 * DT / MVV2E / m
        ea, f, _ = self.at(x, elem, box)
        dof = 3.0 * len(x) - 3.0
        two_ke = lambda: float((m * v * v).sum()) * MVV2E  # noqa: E731
        th = [(float(ea.sum()), 0.5 * two_ke())]
        if nvt:
            kt, q1 = BOLTZ * nvt[0], BOLTZ * nvt[0] * nvt[1] ** 2
            mass, vel, acc = [dof * q1, q1, q1], [0.0] * 4, [0.0] * 3
            for k in (1, 2):
                acc[k] = (mass[k - 1] * vel[k - 1] ** 2 - kt) / mass[k]

            def chain(k2):
                """Half a step of the chain; the factor of the velocities."""
                acc[0] = (k2 - dof * kt) / mass[0]
                for k in (2, 1, 0):
                    s = math.exp(-DT / 8 * vel[k + 1])
                    vel[k] = (vel[k] * s + acc[k] * DT / 4) * s
                fac = math.exp(-DT / 2 * vel[0])
                acc[0] = (k2 * fac * fac - dof * kt) / mass[0]
                s = math.exp(-DT / 8 * vel[1])
                vel[0] = vel[0] * s + acc[0] * DT / 4
                vel[0] *= s
                for k in (1, 2):
                    s = math.exp(-DT / 8 * vel[k + 1])
                    vel[k] *= s
                    acc[k] = (mass[k - 1] * vel[k - 1] ** 2 - kt) / mass[k]
                    vel[k] = (vel[k] + acc[k] * DT / 4) * s
                return fac
        for step in range(1, steps + 1):
            if nvt:
                v = v * chain(two_ke())
            v = v + dtf * f
            x = x + DT * v
            ea, f, _ = self.at(x, elem, box)
            v = v + dtf * f
            if nvt:
                v = v * chain(two_ke())
            if step % every == 0 or step == steps:
                th.append((float(ea.sum()), 0.5 * two_ke()))
        return np.array(th), v.cpu().numpy(), f.cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    w = work(case)["flops"]
    if kind == "bnve" or w > (4e12 if case["steps"] else 4e11):
        return None
    path, _ = _potential(case)
    ex = _Exact(path)
    cuda = lambda a: torch.tensor(a, device="cuda")  # noqa: E731
    if kind in ("batch", "serve"):
        jobs = _jobs(case, seed)

        def single(some):
            e, vir, f = [], [], []
            for _, x, t, box, _ in some:
                ea, fx, vx = ex.at(cuda(x), cuda(t.astype(np.int64) - 1), box)
                e.append(float(ea.sum()))
                vir.append(vx.sum(0).cpu().numpy())
                f.append(fx.cpu().numpy())
            return {"energy": np.array(e), "virial": np.stack(vir), "f": np.concatenate(f)}

        if kind == "batch":
            return single(jobs)
        # FIRE's end state has no 64-bit value here (its branches depend on
        # the sign of a power), nor the periodic image a moved atom is in
        out = {}
        if any(k == 0 for k, *_ in jobs):
            sp = single([q for q in jobs if q[0] == 0])
            sp["virial"] = sp["virial"].reshape(-1)
            out["single"] = {**sp, "x": None, "v": None, "steps": None}
        md = [ex.md(x, v, t, box, case["steps"], case["steps"])
              for k, x, t, box, v in jobs if k == 1]
        if md:
            out["nve"] = {"energy": np.array([q[0][-1, 0] for q in md]),
                          "v": np.concatenate([q[1] for q in md]),
                          "f": np.concatenate([q[2] for q in md])}
        return out
    x, t, box = _structure(case, seed)
    elem = cuda(t.astype(np.int64) - 1)
    if kind in ("nve", "nvt"):
        m = ex.mass[t - 1]
        v = synth.maxwell(m, case["T"], np.random.default_rng([seed, 3]))
        th, v, f = ex.md(x, v, t, box, case["steps"], 10,
                         nvt=(case["T"], 0.1) if kind == "nvt" else None)
        return {"thermo": th, "x": None, "v": v, "f": f, "image": None}
    if case["ghost"]:
        xa, ta, nloc = _ghosts(x, t, box, ex.rc + SKIN)
        xa, elem = cuda(xa), cuda(ta.astype(np.int64) - 1)
        i, j, d = _pairs(xa, box, ex.rc, periodic=False, rows=nloc)
        ea, f, vir = ex.forces(elem, i, j, d, len(xa), rows=nloc)
    else:
        ea, f, vir = ex.at(cuda(x), elem, box)
    out = {"energy": float(ea.sum()), "virial": vir.sum(0).cpu().numpy(), "f": f.cpu().numpy()}
    if kind == "pair":
        out.update(eatom=ea.cpu().numpy(), vatom=None)
    return out
