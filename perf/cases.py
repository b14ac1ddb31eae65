"""Workloads whose speed is measured: the calls that users of this package make, with their sizes.

A case is a dict of plain values; ``prepare`` builds the loaded and uploaded system (what a
program holds before the call), ``run`` makes one call through the public entry points and
returns what the program gets back, ``exact`` computes the same numbers in FP64 with plain
torch.  The kinds:

  md        a state from the host, SingleStep(steps), the state at the end back on the host
            (a segment of dynamics; every call starts at the same state, so results of two
            programs can be compared before chaos has taken over)
  print     SingleStep(steps) and EvalProps (a short print interval)
  forces    new positions, ComputeAccelGPU, forces (an external integrator's force engine)
  props     new positions, EvalProps, forces (energies, virial and pressure of a frame)
  npt       SingleStep(steps) under the Andersen barostat
  minimize  new positions, Minimize(steps)
  batch     Batch.step(steps) over boxes of several sizes, and their states
  pme       pme_reciprocal_static on device tensors (no allocation)

Systems are TIP3P boxes, with or without a slab of linear united-atom chains (the geometry of
the lipid membranes that FEN ZI was written for).  Positions come from a short relaxation in
plain torch, so that pair distances, temperatures and list lifetimes are those of a liquid;
a seed gives another translation, other velocities.
"""
from __future__ import annotations

import atexit
import math
import os
import shutil
import tempfile

import numpy as np
import torch

import fenzi_b200 as fz
from fenzi_b200 import gen_system

DEV = "cuda" if torch.cuda.is_available() else "cpu"
F64 = torch.float64

CC, TU, RC_K = 332.0716, 20.4548, 0.001987
P_ATM = 68558.64100846418  # kcal/mol/A^3 -> atm
P_PU = 1.4586e-5           # atm -> kcal/mol/A^3
ROH, RHH, M_O, M_H = 0.9572, 1.5139, 15.9994, 1.008
CHAIN_LEN = 30
E_KEYS = ["bond", "angle", "ureyb", "dihed", "impr", "vdw", "elec", "pme", "ewexcl", "ewself", "potential"]
# cost limit of exact(): atoms x force evaluations that take about 20 s
EXACT_WORK = 3.0e7
# boxes of a batch whose outputs are returned (and computed in FP64) one by one
SINGLED = 6


# ------------------------------------------------------------------ cases
def listed():
    return [
        # the smallest system of a screening set: one 648-atom box, bound by launches
        dict(name="md_648", kind="md", nw=216, chains=0, rc=9.0, steps=100),
        # one ordinary water box over a print interval
        dict(name="md_9000", kind="md", nw=3000, chains=0, rc=10.0, steps=100),
        # the small membrane system
        dict(name="md_17280", kind="md", nw=5360, chains=40, rc=10.0, steps=100),
        # the large membrane system, the headline size
        dict(name="md_230400", kind="md", nw=72000, chains=480, rc=10.0, steps=100),
        # no rigid bonds, 0.5 fs, a box with three different edges, grid edges that are not
        # powers of two, Urey-Bradley, impropers and two-fold dihedrals
        dict(name="md_flexible_ragged", kind="md", nw=3517, chains=23, rc=9.5, steps=50, flexible=True, ragged=True),
        # energies printed every 10 steps
        dict(name="print_9000", kind="print", nw=3000, chains=0, rc=10.0, steps=10),
        # one force call per new set of positions
        dict(name="forces_17280", kind="forces", nw=5360, chains=40, rc=10.0),
        # energies, virial and forces of one large frame
        dict(name="props_230400", kind="props", nw=72000, chains=480, rc=10.0),
        # constant pressure
        dict(name="npt_17280", kind="npt", nw=5360, chains=40, rc=10.0, steps=20),
        # the moves made before dynamics
        dict(name="minimize_9000", kind="minimize", nw=3000, chains=0, rc=10.0, steps=20),
        # a screening set: 128 boxes of 216 to 2,000 waters advanced together
        dict(name="batch_128", kind="batch", boxes=128, nw=216, nw_max=2000, rc=9.0, steps=100),
        # reciprocal sum for a host program that owns the memory
        dict(name="pme_static_21k", kind="pme", nw=7001, chains=0, rc=10.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["md", "md", "md", "print", "forces", "props", "npt", "minimize", "batch", "pme"])
    c = dict(kind=kind, chains=0, rc=rng.choice([9.0, 9.5, 10.0]))
    if kind == "batch":
        lo = _log_int(rng, 216, 1000)
        c.update(boxes=_log_int(rng, 4, 120), nw=lo, nw_max=_log_int(rng, lo + 1, 2000), rc=9.0, steps=rng.choice([20, 50, 100]))
        del c["chains"]
        return c
    hi = {"md": 60000, "print": 60000, "forces": 60000, "props": 60000, "npt": 12000, "minimize": 12000, "pme": 12000}[kind]
    c["nw"] = _log_int(rng, 350, hi)
    if kind != "pme" and rng.random() < 0.5 and c["nw"] >= 2500:
        c["chains"] = max(1, int(c["nw"] * rng.uniform(0.002, 0.007)))
    if kind in ("md", "print"):
        c["steps"] = rng.choice([7, 20, 50, 100, 100] if kind == "md" else [5, 10, 20])
        if rng.random() < 0.25:
            c["flexible"] = True
        if rng.random() < 0.3 and c["nw"] >= 1000:
            c["ragged"] = True
    elif kind in ("npt", "minimize"):
        c["steps"] = rng.randint(5, 25)
    return c


def _natom(c):
    return 3 * c["nw"] + CHAIN_LEN * c.get("chains", 0)


def _box_waters(c):
    """Waters of each box of a batch: up to 24 sizes, the boxes of one size differing in positions and velocities."""
    sizes = np.random.default_rng(c["boxes"]).integers(c["nw"], c["nw_max"] + 1, size=min(24, c["boxes"]))
    return np.resize(sizes, c["boxes"])


def _members(c):
    """The single systems of a case, as cases."""
    if c["kind"] != "batch":
        return [c]
    return [dict(kind="md", nw=int(k), chains=0, rc=c["rc"], steps=c["steps"], member=i) for i, k in enumerate(_box_waters(c))]


def _geometry(c):
    """(box edges, PME grid) of a single system: the packaged sizes for theirs, else liquid density."""
    n = c["nw"], c.get("chains", 0)
    if n == (3000, 0):
        return np.full(3, 44.8), (48,) * 3
    if n == (5360, 40):
        return np.full(3, 56.0), (64,) * 3
    if n == (72000, 480):
        return np.full(3, 130.0), (128,) * 3
    v = c["nw"] / 0.0334 + c.get("chains", 0) * CHAIN_LEN * 29.0
    a = v ** (1.0 / 3.0)
    box = np.round(a * np.array([1.12, 0.97, 1.0 / (1.12 * 0.97)]), 3) if c.get("ragged") else np.full(3, a)
    if c.get("chains"):  # chains stand along z
        short = 41.0 / box[2]
        if short > 1.0:
            box = np.array([box[0] / math.sqrt(short), box[1] / math.sqrt(short), 41.0])
    if c["kind"] == "pme":
        return box, tuple(min(64, gen_system.fft_friendly(x)) for x in box)
    return box, tuple(gen_system.fft_friendly(x / 1.1) for x in box)


def work(c):
    """Bytes and operations of one pass: 60 per pair within rc; per step and atom 56 bytes of positions, charges,
    types and forces and 120 bytes of integration, per grid point 24 bytes; the state or forces handed over."""
    nbytes = flops = 0.0
    for m in _members(c):
        box, k = _geometry(m)
        n, grid = _natom(m), float(k[0] * k[1] * k[2])
        pairs = 0.5 * n * (n / box.prod()) * 4.0 / 3.0 * math.pi * m["rc"] ** 3
        fft = 2 * 2.5 * grid * math.log2(grid)
        evals = {"md": c.get("steps", 0), "print": c.get("steps", 0) + 1, "forces": 1, "props": 1, "npt": c.get("steps", 0),
                 "minimize": c.get("steps", 0) + 1, "batch": c.get("steps", 0), "pme": 1}[c["kind"]]
        if c["kind"] == "pme":
            nbytes += 40.0 * n + 24.0 * grid
            flops += 1000.0 * n + fft
            continue
        step = 120.0 * n if c["kind"] in ("md", "print", "npt", "minimize", "batch") else 24.0 * n
        nbytes += evals * (56.0 * n + 24.0 * grid + step)
        flops += evals * (60.0 * pairs + 1000.0 * n + fft)
    return {"bytes": nbytes, "flops": flops}


def tolerance(c):
    # Measured as the change that other partial sums of the pair forces make, and the distance from FP64, times four;
    # "max" is of the result's root mean square (a few atoms in close contact differ most).
    k = c["kind"]
    if k == "batch":  # its calls go on from one another: 1.6e-3 (max 0.11) after 300 steps
        return {"rel": 7e-3, "max": 0.5}
    if k in ("md", "npt"):  # FP32 states of a chaotic system: velocities 5e-5 (max 1.2e-3) after 100 steps
        return {"rel": 2e-4, "max": 1e-2}
    if k == "print":  # the virial after a few calls: 5e-6 to 3e-5
        return {"rel": 1e-4, "max": 1e-2}
    if k == "pme":  # 1.3e-5 from FP64
        return {"rel": 5e-5, "max": 5e-4}
    return {"rel": 1e-5, "max": 4e-4}  # forces 2.7e-6 (max 9e-5) from FP64


# ------------------------------------------------------------------ inputs
def _min_image(d, box):
    return d - box * torch.round(d / box)


def _chains(c, box, rng):
    """All-trans chains along z on an x-y lattice, a slab around z = 0."""
    nc = c.get("chains", 0)
    if not nc:
        return np.zeros((0, 3))
    half = math.radians(111.0) / 2
    k = np.arange(CHAIN_LEN)
    zig = np.stack([(k % 2) * 1.53 * math.cos(half), np.zeros(CHAIN_LEN), (k - (CHAIN_LEN - 1) / 2) * 1.53 * math.sin(half)], 1)
    nx = max(1, int(math.ceil(math.sqrt(nc * box[0] / box[1]))))
    ny = int(math.ceil(nc / nx))
    out = []
    for i in range(nc):
        a = rng.uniform(0, 2 * math.pi)
        r = np.array([[math.cos(a), -math.sin(a), 0], [math.sin(a), math.cos(a), 0], [0, 0, 1]])
        at = np.array([(i % nx + 0.5) / nx * box[0] - box[0] / 2, (i // nx + 0.5) / ny * box[1] - box[1] / 2, rng.uniform(-1, 1)])
        out.append(zig @ r.T + at)
    return np.concatenate(out) + rng.normal(scale=0.02, size=(nc * CHAIN_LEN, 3))


def _lattice(nw, box, chain, rng):
    """Oxygen sites: the coarsest lattice that leaves nw sites clear of the chains, a random choice of them."""
    ch = torch.tensor(chain, device=DEV, dtype=torch.float32)
    bx = torch.tensor(box, device=DEV, dtype=torch.float32)
    a = (box.prod() / nw) ** (1.0 / 3.0)
    while True:
        m = np.maximum(1, np.ceil(box / a - 1e-6).astype(int))
        g = [(np.arange(k) + 0.5) / k * e - e / 2 for k, e in zip(m, box)]
        s = np.stack(np.meshgrid(*g, indexing="ij"), -1).reshape(-1, 3)
        if len(s) >= nw and len(chain):
            t = torch.tensor(s, device=DEV, dtype=torch.float32)
            near = torch.cat([(_min_image(x[:, None] - ch[None], bx).square().sum(-1).min(1).values < 2.6 ** 2) for x in t.split(4096)])
            s = s[~near.cpu().numpy()]
        if len(s) >= nw:
            pick = np.sort(rng.choice(len(s), nw, replace=False))
            return s[pick] + rng.uniform(-0.1, 0.1, size=(nw, 3))
        a *= 0.985


def _nearest(x, y, k, box, own):
    """Indices of the k sites of y nearest to each x (own: x is y, itself left out)."""
    out = []
    for b in range(0, len(x), 2048):
        d2 = sum((_min_image(x[b:b + 2048, None, c] - y[None, :, c], box[c])).square() for c in range(3))
        i = torch.topk(d2, min(k + own, len(y)), dim=1, largest=False).indices
        out.append(i[:, own:])
    return torch.cat(out)


def _relax(ow, chain, box, rng):
    """Waters near 300 K around the fixed chains: 240 Langevin steps of 2 fs with the 32 nearest waters of each (dense
    sums, the same on every run), then each water put back on its rigid shape.  Returns (nw, 3, 3)."""
    g = torch.Generator(device="cpu").manual_seed(int(rng.integers(1 << 30)))
    f32 = dict(device=DEV, dtype=torch.float32)
    nw, bx = len(ow), torch.tensor(box, **f32)
    ch = torch.tensor(chain, **f32)
    q = torch.tensor([-0.834, 0.417, 0.417], **f32)
    qq = CC * q[:, None] * q[None, :]
    shape = torch.tensor([[0.0, 0, 0], [RHH / 2, 0, math.sqrt(ROH ** 2 - RHH ** 2 / 4)], [-RHH / 2, 0, math.sqrt(ROH ** 2 - RHH ** 2 / 4)]], **f32)
    w = torch.linalg.qr(torch.randn(nw, 3, 3, generator=g)).Q.to(DEV)
    x = torch.tensor(ow, **f32)[:, None] + shape @ w
    mass, kt, dt = 10.0, RC_K * 300.0, 0.002 * TU
    keep = math.exp(-0.08)
    v = torch.randn(nw, 3, 3, generator=g).to(DEV) * math.sqrt(kt / mass)
    rcut = 6.5
    for step in range(240):
        if step % 40 == 0:
            nb = _nearest(x[:, 0], x[:, 0], 32, bx, 1)
            nc = _nearest(x[:, 0], ch, 12, bx, 0) if len(ch) else None
        oo = _min_image(x[:, None, 0] - x[nb, 0], bx)
        off = x - x[:, :1]
        d = oo[:, :, None, None] + off[:, None, :, None] - off[nb][:, :, None, :]
        r2 = d.square().sum(-1).clamp(min=0.8)
        s = qq * (r2 < rcut ** 2) * (r2 ** -1.5 - rcut ** -3)
        f = (s[..., None] * d).sum((1, 3))
        o2 = oo.square().sum(-1).clamp(min=4.0)
        s6 = (3.1506 ** 2 / o2) ** 3
        f[:, 0] += ((24 * 0.1521 * s6 * (2 * s6 - 1) / o2)[..., None] * oo).sum(1)
        if nc is not None:
            cd = _min_image(x[:, None, 0] - ch[nc], bx)
            c2 = cd.square().sum(-1).clamp(min=4.0)
            s6 = (3.40 ** 2 / c2) ** 3
            f[:, 0] += ((24 * 0.109 * s6 * (2 * s6 - 1) / c2)[..., None] * cd).sum(1)
        for a, b, r0 in ((0, 1, ROH), (0, 2, ROH), (1, 2, RHH)):
            e = x[:, a] - x[:, b]
            r = e.square().sum(-1, keepdim=True).sqrt()
            h = 500.0 * (r0 / r - 1.0) * e
            f[:, a] += h
            f[:, b] -= h
        v = (v + dt / mass * f).clamp(-1.2, 1.2)
        v = keep * v + math.sqrt((1 - keep ** 2) * kt / mass) * torch.randn(nw, 3, 3, generator=g).to(DEV)
        x = x + dt * v
    o = x[:, 0].double()
    b = (x[:, 1] + x[:, 2]).double() / 2 - o
    b = b / b.norm(dim=1, keepdim=True)
    p = (x[:, 1] - x[:, 2]).double()
    p = p - (p * b).sum(1, keepdim=True) * b
    p = p / p.norm(dim=1, keepdim=True)
    h = math.sqrt(ROH ** 2 - RHH ** 2 / 4)
    return torch.stack([o, o + h * b + RHH / 2 * p, o + h * b - RHH / 2 * p], 1).cpu().numpy()


_base = {}   # relaxed positions of the sizes met so far in this process
_files = {}  # their input files


def _base_of(c):
    key = (c["nw"], c.get("chains", 0), bool(c.get("ragged")), c["kind"] == "pme")
    if key not in _base:
        rng = np.random.default_rng([c["nw"], c.get("chains", 0)])
        box, grid = _geometry(c)
        chain = _chains(c, box, rng)
        wat = _relax(_lattice(c["nw"], box, chain, rng), chain, box, rng)
        _base[key] = box, grid, np.concatenate([chain, wat.reshape(-1, 3)])
    return key, _base[key]


def _wrap(x, box):
    return x - box * np.floor(x / box + 0.5)


def _masses(c):
    return np.concatenate([np.full(CHAIN_LEN * c.get("chains", 0), 14.027), np.tile([M_O, M_H, M_H], c["nw"])])


def _charges(c):
    return np.concatenate([np.tile([0.09, -0.09], CHAIN_LEN * c.get("chains", 0) // 2), np.tile([-0.834, 0.417, 0.417], c["nw"])])


def _state(c, seed):
    """Positions and velocities (FP32) of one seed: the relaxed system moved by a random vector, and 300 K velocities
    that keep every water rigid."""
    key, (box, grid, base) = _base_of(c)
    rng = np.random.default_rng([seed, c.get("member") or 0])
    nca = CHAIN_LEN * c.get("chains", 0)
    w = base[nca:].reshape(-1, 3, 3)
    mw = np.array([M_O, M_H, M_H])
    com = (w * mw[:, None]).sum(1, keepdims=True) / mw.sum()
    r = w - com
    b = (r[:, 1] + r[:, 2]) - 2 * r[:, 0]
    p = r[:, 1] - r[:, 2]
    b, p = b / np.linalg.norm(b, axis=1, keepdims=True), p / np.linalg.norm(p, axis=1, keepdims=True)
    omega = 0.0
    kt = RC_K * 300.0
    for axis in (b, p, np.cross(b, p)):
        inertia = (mw * (np.cross(r, axis[:, None]) ** 2).sum(-1)).sum(1)
        omega = omega + (rng.normal(size=len(w)) * np.sqrt(kt / inertia))[:, None] * axis
    vw = rng.normal(size=(len(w), 1, 3)) * math.sqrt(kt / mw.sum()) + np.cross(omega[:, None], r)
    vel = np.concatenate([rng.normal(size=(nca, 3)) * math.sqrt(kt / 14.027), vw.reshape(-1, 3)])
    m = _masses(c)[:, None]
    vel -= (m * vel).sum(0) / m.sum()
    pos = _wrap(base + rng.uniform(-0.5, 0.5, 3) * box, box)
    return pos.astype(np.float32), vel.astype(np.float32)


def _topology(c):
    """Bonds, angles, dihedrals, impropers (0-based)."""
    nc = c.get("chains", 0)
    first = CHAIN_LEN * np.arange(nc)[:, None]
    run = lambda k: (first + np.arange(CHAIN_LEN - k + 1)).reshape(-1, 1) + np.arange(k)  # noqa: E731
    o = CHAIN_LEN * nc + 3 * np.arange(c["nw"])[:, None]
    bonds = np.concatenate([run(2), (o[:, None] + np.array([[0, 1], [0, 2], [1, 2]])).reshape(-1, 2)])
    angles = np.concatenate([run(3), o + np.array([1, 0, 2])])
    dihedrals = run(4)
    extras = bool(c.get("ragged")) and nc > 0
    impropers = (first + np.arange(0, CHAIN_LEN - 3, 4)).reshape(-1, 1) + np.arange(4) if extras else np.zeros((0, 4), int)
    return bonds.astype(np.int64), angles.astype(np.int64), dihedrals.astype(np.int64), impropers.astype(np.int64), extras


def _input_file(c):
    key, (box, grid, base) = _base_of(c)
    key = key + (c["rc"], c["kind"])
    if key not in _files:
        nc, nw = c.get("chains", 0), c["nw"]
        bonds, angles, dihedrals, impropers, extras = _topology(c)
        nca = CHAIN_LEN * nc
        s = gen_system.System(
            name="case", box=box, pos=_wrap(base, box), types=["CTU"] * nca + ["OT", "HT", "HT"] * nw, charge=_charges(c), mass=_masses(c),
            atom_names=[f"C{j + 1}" for j in range(CHAIN_LEN)] * nc + ["OH2", "H1", "H2"] * nw,
            resnames=["CHN"] * nca + ["TIP3"] * (3 * nw), segids=["CHN"] * nca + ["WAT"] * (3 * nw),
            resids=np.concatenate([np.repeat(np.arange(1, nc + 1), CHAIN_LEN), 1 + np.repeat(np.arange(nw), 3) % 9999]).astype(np.int64),
            bonds=bonds, angles=angles, dihedrals=dihedrals, impropers=impropers, extras=extras, kgrid=grid, rc=c["rc"], ron=c["rc"] - 2.0,
            pairlist=c["rc"] + 1.0)
        folder = tempfile.mkdtemp(prefix="fz_cases_")
        atexit.register(shutil.rmtree, folder, True)
        _files[key] = gen_system.write(s, folder)
    return _files[key]


def _load(c, seed):
    s = fz.FenZi.ReadInput(_input_file(c))
    if c.get("flexible"):
        s.cfg.shake, s.cfg.timestep_ps = 0, 0.0005
    if c["kind"] == "minimize":
        s.cfg.conjgradfac = s.cfg.steepdesfac = 1e-5
    s.LoadSystem()
    s.InitMem(0)
    pos, vel = _state(c, seed)
    box = torch.tensor(_base_of(c)[1][0], dtype=torch.float32)
    pin = lambda a: torch.from_numpy(a).pin_memory()  # noqa: E731
    st = dict(sys=s, start=pin(pos), vel0=pin(vel), pos=pin(pos.copy()), vel=pin(vel.copy()), box=box)
    s.set_state_f32(st["start"].numpy(), st["vel0"].numpy())
    s.sync()
    return st


def prepare(case, seed):
    k = case["kind"]
    if k == "batch":
        members = [_load(m, seed) for m in _members(case)]
        return dict(kind=k, members=members, batch=fz.Batch([m["sys"] for m in members]), steps=case["steps"])
    if k == "pme":
        pos, _ = _state(case, seed)
        box, grid = _geometry(case)
        xyzq = np.concatenate([pos, _charges(case)[:, None].astype(np.float32)], 1)
        return dict(kind=k, xyzq=torch.from_numpy(xyzq).to(DEV), box=box, grid=grid,
                    facc=torch.empty(3, len(pos), dtype=torch.int64, device=DEV))
    st = _load(case, seed)
    if k == "npt":
        st["sys"].set_barostat(True, pref_atm=1.0)
    st.update(kind=k, steps=case.get("steps"))
    return st


# ------------------------------------------------------------------ the measured calls
def _frame(st):
    """Positions (followed across the box edges) and velocities, as an analysis program keeps them."""
    s = st["sys"]
    s.get_state_f32(st["pos"].numpy(), st["vel"].numpy())
    d = st["pos"] - st["start"]
    d -= st["box"] * torch.round(d / st["box"])
    return {"pos": d.add_(st["start"]), "vel": st["vel"]}


def _props(e):
    return {"energies": np.array([e[k] for k in E_KEYS]), "kinetic": e["kinetic"], "temperature": e["temperature"],
            "virial": np.array(e["virial"])}


def _by_box(frames):
    """(positions, velocities) of the first boxes one by one, of the others in one piece."""
    rest = frames[SINGLED:]
    return {"boxes": frames[:SINGLED], "rest": [torch.cat([f[i] for f in rest]) for i in (0, 1)] if rest else None}


def run(st):
    k = st["kind"]
    if k == "pme":
        e = fz.pme_reciprocal_static(0, st["xyzq"].data_ptr(), st["xyzq"].shape[0], st["box"], st["grid"], 0.34, st["facc"].data_ptr(),
                                     stream=torch.cuda.current_stream().cuda_stream)
        return {"forces": st["facc"].double().mul_(2.0 ** -32), "energy": e}
    if k == "batch":
        st["batch"].step(st["steps"])
        frames = [_frame(m) for m in st["members"]]
        return _by_box([(f["pos"], f["vel"]) for f in frames])
    s = st["sys"]
    if k == "md":
        s.set_state_f32(st["start"].numpy(), st["vel0"].numpy())
        s.SingleStep(st["steps"])
        return _frame(st)
    if k == "npt":
        s.SingleStep(st["steps"])
        e = s.EvalProps()
        st["box"] = torch.tensor(e["box"], dtype=torch.float32)
        return dict(_props(e), box=np.array(e["box"]), **_frame(st))
    if k == "print":
        s.SingleStep(st["steps"])
        return _props(s.EvalProps())
    s.set_state_f32(st["start"].numpy(), None)
    if k == "forces":
        s.ComputeAccelGPU()
        return {"forces": s.forces()}
    if k == "props":
        return dict(_props(s.EvalProps()), forces=s.forces())
    moves, energy = s.Minimize(st["steps"])
    s.get_state_f32(st["pos"].numpy(), None)
    return {"moves": moves, "energy": energy, "pos": st["pos"]}


# ------------------------------------------------------------------ FP64 reference
class _Model:
    """Energies and forces of one system in FP64: exact erfc, order-4 smooth PME, CHARMM terms."""

    def __init__(self, c):
        box, self.K = _geometry(c)
        t = lambda a: torch.tensor(np.asarray(a), device=DEV)  # noqa: E731
        self.box, self.n, self.nw, self.nca = t(box).to(F64), _natom(c), c["nw"], CHAIN_LEN * c.get("chains", 0)
        self.rc, self.ron, self.beta = c["rc"], c["rc"] - 2.0, 0.34
        self.q, self.m = t(_charges(c)).to(F64), t(_masses(c)).to(F64)
        typ = np.where(np.arange(self.n) < self.nca, 2, np.where((np.arange(self.n) - self.nca) % 3 == 0, 0, 1))  # O, H, C
        self.typ = t(typ)
        eps, rmh = np.array([0.1521, 0.046, 0.078]), np.array([1.7682, 0.2245, 2.05])
        bonds, angles, dihedrals, impropers, extras = _topology(c)
        e4, s2 = 4 * np.sqrt(np.outer(eps, eps)), ((rmh[:, None] + rmh) / 2 ** (1 / 6)) ** 2
        e14, r14 = eps.copy(), rmh.copy()
        if extras:
            e4[0, 2] = e4[2, 0] = 4 * 0.12
            s2[0, 2] = s2[2, 0] = (3.7 / 2 ** (1 / 6)) ** 2
            e14[2], r14[2] = 0.05, 1.9
        self.e4, self.s2 = t(e4), t(s2)
        self.e4_14, self.s2_14 = t(4 * np.sqrt(np.outer(e14, e14))), t(((r14[:, None] + r14) / 2 ** (1 / 6)) ** 2)
        wb, wa = bonds[:, 0] >= self.nca, angles[:, 0] >= self.nca
        hh = wb & ((bonds[:, 0] - self.nca) % 3 == 1)
        self.bonds, self.bk = t(bonds), t(np.where(hh, 0.0, np.where(wb, 450.0, 222.5)))
        self.br = t(np.where(hh, RHH, np.where(wb, ROH, 1.53)))
        self.angles, self.ak = t(angles), t(np.where(wa, 55.0, 58.35))
        self.at = t(np.radians(np.where(wa, 104.52, 111.0)))
        self.dihe, self.impr = t(dihedrals), t(impropers)
        self.folds = [(0.16, 3, 0.0)] + ([(0.05, 1, math.radians(30.0))] if extras else [])
        self.ub = self.angles[~t(wa)][:, [0, 2]] if extras else self.angles[:0, :2]
        order = lambda p: np.unique(np.sort(p, 1), axis=0)  # noqa: E731
        ew = order(np.concatenate([bonds, angles[:, [0, 2]]]))
        p14 = order(dihedrals[:, [0, 3]]) if len(dihedrals) else np.zeros((0, 2), np.int64)
        self.ew, self.p14 = t(ew), t(p14)
        self.excl = torch.sort(t(np.concatenate([ew, p14]) @ np.array([self.n, 1]))).values
        self.wat = self.nca + 3 * torch.arange(self.nw, device=DEV)[:, None] + torch.arange(3, device=DEV)
        self.listed = None

    def pairs(self, x):
        """Unexcluded pairs within rc + 1.5, kept until an atom has moved 0.7 (the box may breathe by 0.05)."""
        if self.listed is not None and (x - self.listed).norm(dim=1).max() < 0.7:
            return self.pair
        self.listed = x.clone()
        y, b32 = _min_image(x, self.box).float(), self.box.float()
        got, rows = [], max(16, int(1.5e8 / self.n))
        for a in range(0, self.n, rows):
            d2 = sum(_min_image(y[a:a + rows, None, c] - y[None, a:, c], b32[c]).square_() for c in range(3))
            i, j = torch.nonzero(d2 < (self.rc + 1.51) ** 2, as_tuple=True)
            up = j > i
            got.append(torch.stack([i[up] + a, j[up] + a]))
        p = torch.cat(got, 1)
        k = p[0] * self.n + p[1]
        if len(self.excl):
            at = torch.searchsorted(self.excl, k).clamp(max=len(self.excl) - 1)
            p = p[:, self.excl[at] != k]
        self.pair = p
        return p

    def _lj_elec(self, r2, ij, e4, s2):
        r, ir2 = r2.sqrt(), 1.0 / r2
        ti, tj = self.typ[ij[0]], self.typ[ij[1]]
        s6 = (s2[ti, tj] * ir2) ** 3
        rc2, ron2 = self.rc ** 2, self.ron ** 2
        sw = torch.where(r2 > ron2, (rc2 - r2) ** 2 * (rc2 + 2 * r2 - 3 * ron2) / (rc2 - ron2) ** 3, torch.ones_like(r2))
        return (e4[ti, tj] * s6 * (s6 - 1) * sw).sum(), (CC * self.q[ij[0]] * self.q[ij[1]] * torch.erfc(self.beta * r) / r).sum()

    def _dihedral(self, x, box, q):
        f, g, h = (_min_image(x[q[:, a]] - x[q[:, b]], box) for a, b in ((0, 1), (1, 2), (3, 2)))
        a, b = torch.linalg.cross(f, g), torch.linalg.cross(h, g)
        return torch.atan2((torch.linalg.cross(b, a) * g).sum(1) / g.norm(dim=1), (a * b).sum(1))

    def pme(self, x, box):
        K = torch.tensor(self.K, device=DEV)
        u = x / box * K
        k0 = torch.floor(u.detach())
        t = u - k0
        w = torch.stack([t ** 3 / 6, (1 + 3 * t + 3 * t ** 2 - 3 * t ** 3) / 6, (4 - 6 * t ** 2 + 3 * t ** 3) / 6, (1 - t) ** 3 / 6])
        g = [torch.remainder(k0[:, c].long()[:, None] - torch.arange(4, device=DEV), K[c]) for c in range(3)]
        flat = ((g[2][:, :, None, None] * K[1] + g[1][:, None, :, None]) * K[0] + g[0][:, None, None, :]).reshape(-1)
        val = self.q[:, None, None, None] * w[:, :, 2].T[:, :, None, None] * w[:, :, 1].T[:, None, :, None] * w[:, :, 0].T[:, None, None, :]
        Q = torch.zeros(int(K.prod()), device=DEV, dtype=F64).index_add(0, flat, val.reshape(-1))
        S = torch.fft.fftn(Q.reshape(self.K[2], self.K[1], self.K[0]))
        m2, c = 0.0, 1.0
        for d in range(3):
            kd = self.K[d]
            m = torch.arange(kd, device=DEV, dtype=F64)
            a = 2 * math.pi * m / kd
            bm = 1.0 / ((1 + 4 * torch.cos(a) + torch.cos(2 * a)) ** 2 + (4 * torch.sin(a) + torch.sin(2 * a)) ** 2) * 36.0
            f2 = (torch.where(m <= kd // 2, m, m - kd) / box[d]) ** 2
            shape = [1, 1, 1]
            shape[2 - d] = kd
            m2, c = m2 + f2.reshape(shape), c * bm.reshape(shape)
        m2 = m2 + torch.zeros_like(S.real)
        on = torch.ones_like(m2)
        on[0, 0, 0] = 0.0
        m2 = m2 + (1.0 - on)
        c = on * c * torch.exp(-(math.pi / self.beta) ** 2 * m2) / m2
        return CC / (2 * math.pi * box.prod()) * (c * (S.real ** 2 + S.imag ** 2)).sum()

    def energies(self, x, lam, pair):
        """The E_KEYS energies; lam scales coordinates and box per axis (its gradient is minus the virial)."""
        box, x = self.box * lam, x * lam
        dist = lambda ij: _min_image(x[ij[0]] - x[ij[1]], box)  # noqa: E731
        with torch.no_grad():
            pair = pair[:, dist(pair).square().sum(1) < self.rc ** 2]
        vdw, elec = self._lj_elec(dist(pair).square().sum(1), pair, self.e4, self.s2)
        p = self.p14.T
        if len(self.p14):
            v14, e14 = self._lj_elec(dist(p).square().sum(1), p, self.e4_14, self.s2_14)
            vdw, elec = vdw + v14, elec + e14
        r = dist(self.ew.T).norm(dim=1)
        ex = -(CC * self.q[self.ew[:, 0]] * self.q[self.ew[:, 1]] * torch.erf(self.beta * r) / r).sum()
        bond = (self.bk * (dist(self.bonds.T).norm(dim=1) - self.br) ** 2).sum()
        u, v = dist(self.angles[:, [0, 1]].T), dist(self.angles[:, [2, 1]].T)
        th = torch.atan2(torch.linalg.cross(u, v).norm(dim=1), (u * v).sum(1))
        angle = (self.ak * (th - self.at) ** 2).sum()
        zero = x.new_zeros(())
        ub = (12.0 * (dist(self.ub.T).norm(dim=1) - 2.52) ** 2).sum() if len(self.ub) else zero
        dih = imp = zero
        if len(self.dihe):
            phi = self._dihedral(x, box, self.dihe)
            dih = sum((k * (1 + torch.cos(n * phi - d))).sum() for k, n, d in self.folds)
        if len(self.impr):
            imp = (1.5 * self._dihedral(x, box, self.impr) ** 2).sum()
        own = zero - CC * self.beta / math.sqrt(math.pi) * self.q.square().sum()
        e = [bond, angle, ub, dih, imp, vdw, elec, self.pme(x, box), ex, own]
        return torch.stack(e + [sum(e)])

    def forces(self, x, virial=False):
        """(forces, energies[, force virial per axis])"""
        pair = self.pairs(x)
        y = x.detach().requires_grad_()
        lam = torch.ones(3, device=DEV, dtype=F64, requires_grad=virial)
        e = self.energies(y, lam, pair)
        g = torch.autograd.grad(e[-1], [y, lam] if virial else [y])
        return (-g[0], e.detach(), -g[1]) if virial else (-g[0], e.detach())

    # waters: constraints (O,H1), (O,H2), (H1,H2)
    def _bond3(self, x):
        w = x[self.wat]
        return _min_image(torch.stack([w[:, 0] - w[:, 1], w[:, 0] - w[:, 2], w[:, 1] - w[:, 2]], 1), self.box)

    SIGN = [[1.0, 1.0, 0.0], [-1.0, 0.0, 1.0], [0.0, -1.0, -1.0]]  # atom x constraint

    def _coupling(self):
        s = torch.tensor(self.SIGN, device=DEV, dtype=F64)
        im = 1.0 / torch.tensor([M_O, M_H, M_H], device=DEV, dtype=F64)
        return s, im, (s.T * im) @ s

    def shake(self, x0, x):
        s, im, cf = self._coupling()
        rd, c0 = self._bond3(x0), self._bond3(x)
        d2 = torch.tensor([ROH, ROH, RHH], device=DEV, dtype=F64) ** 2
        lam = torch.zeros(self.nw, 3, device=DEV, dtype=F64)
        for _ in range(12):
            c = c0 + torch.einsum("kl,wl,wld->wkd", cf, lam, rd)
            J = 2.0 * cf * torch.einsum("wkd,wld->wkl", c, rd)
            lam = lam - torch.linalg.solve(J, (c.square().sum(-1) - d2)[..., None])[..., 0]
        y = x.clone()
        y[self.wat] += torch.einsum("ak,a,wk,wkd->wad", s, im, lam, rd)
        return y

    def rattle(self, x, v):
        s, im, cf = self._coupling()
        rd = self._bond3(x)
        vd = torch.einsum("ak,wad->wkd", s, v[self.wat])
        mu = torch.linalg.solve(cf * torch.einsum("wkd,wld->wkl", rd, rd), (vd * rd).sum(-1)[..., None])[..., 0]
        u = v.clone()
        u[self.wat] -= torch.einsum("ak,a,wk,wkd->wad", s, im, mu, rd)
        return u

    def constraint_virial(self, x, v, f):
        s, _, cf = self._coupling()
        rd = self._bond3(x)
        vd = torch.einsum("ak,wad->wkd", s, v[self.wat])
        ad = torch.einsum("ak,wad->wkd", s, (f / self.m[:, None])[self.wat])
        rhs = -vd.square().sum(-1) - (rd * ad).sum(-1)
        lam = torch.linalg.solve(cf * torch.einsum("wkd,wld->wkl", rd, rd), rhs[..., None])[..., 0]
        return (lam[..., None] * rd ** 2).sum((0, 1))

    def groups(self, x):
        """Offsets of the atoms of a water from its mass centre (0 for chain atoms)."""
        w = x[self.wat]
        d = _min_image(w - w[:, :1], self.box)
        m = self.m[self.wat][..., None]
        off = torch.zeros_like(x)
        off[self.wat] = d - (m * d).sum(1, keepdim=True) / m.sum(1, keepdim=True)
        return off

    def group_velocity(self, v):
        u, m = v.clone(), self.m[self.wat][..., None]
        u[self.wat] = ((m * v[self.wat]).sum(1, keepdim=True) / m.sum(1, keepdim=True)).expand(-1, 3, -1)
        return u

    def group_pressure(self, x, v, f, w):
        k = 0.5 * (self.m[:, None] * self.group_velocity(v) ** 2).sum()
        return float((2 * k + w.sum() - (self.groups(x) * f).sum()) / (3 * self.box.prod()))


def _dynamics(M, x, v, dt, steps, rigid):
    f = M.forces(x)[0]
    h = 0.5 * dt / M.m[:, None]
    for _ in range(steps):
        v = v + h * f
        y = x + dt * v
        if rigid:
            y = M.shake(x, y)
            v = (y - x) / dt
        x = y
        f = M.forces(x)[0]
        v = v + h * f
        if rigid:
            v = M.rattle(x, v)
    return x, v


def _constant_pressure(M, x, v, dt, steps, pmass=1e-5, pref=1.0):
    """Andersen's barostat with the waters as rigid scaling groups."""
    h = 0.5 * dt / M.m[:, None]
    f, _, w = M.forces(x, True)
    ldot = 0.0
    acc = lambda: (M.group_pressure(x, v, f, w) - pref * P_PU) / (3 * pmass * float(M.box[0]) ** 2) - 2 * ldot ** 2 / float(M.box[0])  # noqa: E731
    lacc = acc()
    for _ in range(steps):
        L = float(M.box[0])
        ldot += 0.5 * dt * lacc
        lam = (L + dt * ldot) / L
        v = v + (math.exp(-0.5 * dt * ldot / L) - 1) * M.group_velocity(v)
        v = v + h * f
        x = x + (lam - 1) * (x - M.groups(x))
        M.box = M.box * lam
        y = M.shake(x, x + dt * v)
        v = (y - x) / dt
        x = y
        f, _, w = M.forces(x, True)
        lacc = acc()
        ldot += 0.5 * dt * lacc
        v = v + h * f
        v = v + (math.exp(-0.5 * dt * ldot / (L * lam)) - 1) * M.group_velocity(v)
        v = M.rattle(x, v)
    return x, v


def _exact_props(M, x, v, rigid):
    """What _props() returns, and the forces."""
    f, e, w = M.forces(x, True)
    kin = float(0.5 * (M.m[:, None] * v ** 2).sum())
    if rigid:
        w = w + M.constraint_virial(x, v, f)
    dof = 3 * M.n - 6 - (3 * M.nw if rigid else 0)
    return {"energies": e, "kinetic": kin, "temperature": 2 * kin / (RC_K * dof), "virial": w}, f


def _minimised(M, x, steps, fac=1e-5):
    f, e = M.forces(x)
    prev, way = f, torch.zeros_like(x)
    for _ in range(steps):
        ff, pp = f.square().sum(1, keepdim=True), prev.square().sum(1, keepdim=True)
        pp = torch.where(pp < 1e-8, ff, pp)
        way = (f + way * (ff / pp)) * fac
        prev = f
        x = M.shake(x, x + way)
        f, e = M.forces(x)
    return x, float(e[-1])


def exact(case, seed):
    k, steps = case["kind"], case.get("steps", 1)
    members = _members(case)
    if max(_natom(m) for m in members) * (steps + 1) > EXACT_WORK:
        return None
    got = []
    for c in members[:SINGLED]:
        pos, vel = _state(c, seed)
        M = _Model(c)
        x, v = (torch.tensor(a, device=DEV, dtype=F64) for a in (pos, vel))
        dt = (0.0005 if c.get("flexible") else 0.001) * TU
        if k in ("md", "batch"):
            got.append(_dynamics(M, x, v, dt, steps, not c.get("flexible")))
        elif k == "npt":
            x, v = _constant_pressure(M, x, v, dt, steps)
            return dict(_exact_props(M, x, v, True)[0], box=M.box.cpu(), pos=x, vel=v)
        elif k == "minimize":
            x, e = _minimised(M, x, steps)
            return {"moves": steps, "energy": e, "pos": x}
        elif k == "pme":
            y = x.requires_grad_()
            e = M.pme(y, M.box)
            return {"forces": -torch.autograd.grad(e, y)[0].T.contiguous(), "energy": float(e.detach())}
        elif k == "forces":
            return {"forces": M.forces(x)[0]}
        else:
            if k == "print":
                x, v = _dynamics(M, x, v, dt, steps, not c.get("flexible"))
            out, f = _exact_props(M, x, v, not c.get("flexible"))
            return out if k == "print" else dict(out, forces=f)
    return {"boxes": got, "rest": None} if k == "batch" else dict(zip(("pos", "vel"), got[0]))
