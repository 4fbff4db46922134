"""The time loop of a granular run, measured through the public entry points.

A case is a bed of spheres, the calls that a program makes on it and how many
steps it makes per pass; every pass ends with positions, velocities and
angular velocities in the program's own host arrays, as a program has them
that saves or looks at the state every so many steps.

Beds
  packing   radii U[0.4, 0.6] in a fully periodic cube at a volume fraction
            ``phi``: 0.55 (a dense gas, few contacts) to 0.65 (jammed, about
            six contacts per sphere)
  floor     spheres of diameter 1 lying on a frictional floor, x and y periodic
  box       a bidisperse bed (diameters 1 and 3, 20:1) between a floor and four
            side walls, no periodic axis
  hopper    spheres of diameter 1 in a conic hopper over a floor, both shaken
  ensemble  independent floor beds of uneven size (radii U[0.45, 0.55], a
            friction coefficient and a restitution each) in one context
Calls
  run       ``run(first, last)``: the library's own time loop
  steps     one ``move_particles`` per step: the program's own time loop
  coupled   per step the program hands over its positions and velocities,
            advances them and takes them back (a solver that couples the
            spheres with something else)
"""
import math

import numpy as np
import torch

from dem3d_b200 import params as P
from dem3d_b200.system import DEMSystem

KN, KT = 1.0e5, 2.0e5 / 7.0      # pair springs; wall springs are the same
DENSITY = 6.0 / math.pi          # a sphere of diameter 1 has mass 1
EULER_INTERVALS = 10             # sub-steps of each of the three start-up steps
ORDER = 4


def listed():
    return [
        # the smallest runs: 2,000 spheres on a floor, stepped by the library
        # and one call at a time (the start of every study; launches count)
        dict(name="floor_2k_fp64", bed="floor", n=2000, prec="fp64", calls="run", steps=40),
        dict(name="floor_2k_calls_fp64", bed="floor", n=2000, prec="fp64", calls="steps", steps=10),
        # cone and rectangle walls in motion: a small vibrated hopper
        dict(name="hopper_600_fp64", bed="hopper", n=600, prec="fp64", calls="run", steps=40),
        # parameter studies: many independent systems in one context
        dict(name="ensemble_16_mixed", bed="ensemble", systems=16, nmin=200, nmax=2000,
             prec="mixed", calls="run", steps=40),
        dict(name="ensemble_64_mixed", bed="ensemble", systems=64, nmin=200, nmax=20000,
             prec="mixed", calls="run", steps=20),
        # a solver that exchanges the state with the library every step
        dict(name="coupled_250k_mixed", bed="packing", phi=0.55, n=250_001, prec="mixed",
             calls="coupled", steps=2),
        # compressed packings, six contacts per sphere
        dict(name="jammed_216k_fp64", bed="packing", phi=0.65, n=216_000, prec="fp64",
             calls="run", steps=20),
        dict(name="jammed_1m_mixed", bed="packing", phi=0.65, n=1_000_000, prec="mixed",
             calls="run", steps=20),
        # the benchmark's size in both precisions
        dict(name="dense_1m_fp64", bed="packing", phi=0.55, n=1_000_000, prec="fp64",
             calls="run", steps=40),
        dict(name="dense_1m_mixed", bed="packing", phi=0.55, n=1_000_000, prec="mixed",
             calls="run", steps=40),
        # two sizes of spheres between walls, an odd count
        dict(name="box_1m_mixed", bed="box", n=1_000_003, prec="mixed", calls="run", steps=20),
        # a large production run
        dict(name="dense_4m_mixed", bed="packing", phi=0.60, n=4_000_000, prec="mixed",
             calls="run", steps=20),
    ]


def _between(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    bed = rng.choice(["packing", "packing", "packing", "floor", "box", "hopper", "ensemble"])
    case = dict(bed=bed, prec=rng.choice(["fp64", "mixed"]))
    if bed == "ensemble":
        case.update(systems=_between(rng, 4, 80), nmin=200, nmax=_between(rng, 1000, 20000),
                    calls="run", steps=rng.randint(8, 40))
        return case
    lo, hi = {"packing": (2000, 2_000_000), "floor": (300, 200_000), "box": (3000, 1_000_000),
              "hopper": (200, 2000)}[bed]
    case["n"] = _between(rng, lo, hi)
    if bed == "packing":
        case["phi"] = rng.choice([0.55, 0.60, 0.65])
    case["calls"] = rng.choice(["run", "run", "run", "steps", "coupled"])
    case["steps"] = rng.randint(8, 40) if case["calls"] == "run" else rng.randint(1, 4)
    return case


# ---------------------------------------------------------------------------
# beds

def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _generator(seed):
    g = torch.Generator(device=_device())
    g.manual_seed(int(seed))
    return g


def _uniform(g, shape, lo=0.0, hi=1.0):
    return lo + (hi - lo) * torch.rand(shape, generator=g, device=_device(), dtype=torch.float64)


def _relaxed(radius, box, g, rounds, swell=1.0, layer=False):
    """Centres of spheres in a periodic box, moved apart until only the
    overlaps that their volume makes are left (a jittered lattice, then steps
    along the sum of each sphere's overlaps).  ``swell``: moved apart as
    spheres that much larger; ``layer``: between two planes in z, on which
    the lowest and the highest spheres lie."""
    n = radius.numel()
    L = torch.tensor(box, device=radius.device)
    cells = [max(1, round((n * b ** 3 / (box[0] * box[1] * box[2])) ** (1 / 3))) for b in box]
    while cells[0] * cells[1] * cells[2] < n:
        k = min(range(3), key=lambda d: cells[d] / box[d])
        cells[k] += 1
    site = torch.randperm(cells[0] * cells[1] * cells[2], generator=g, device=radius.device)[:n]
    idx = torch.stack([site % cells[0], site // cells[0] % cells[1],
                       site // (cells[0] * cells[1])], 1).double()
    a = L / torch.tensor(cells, device=radius.device, dtype=torch.float64)
    x = (idx + 0.5 + _uniform(g, (n, 3), -0.2, 0.2)) * a
    x, r, Lf = x.float(), (radius * swell).float(), L.float()
    per = torch.tensor([1.0, 1.0, 0.0 if layer else 1.0], device=x.device)
    k = min(24, n - 1)
    for it in range(rounds):
        if it % 20 == 0:
            near = []
            for lo in range(0, n, 2048):
                d = x[lo:lo + 2048, None, :] - x[None, :, :]
                d -= per * Lf * torch.round(d / Lf)
                near.append(torch.topk(d.square().sum(2), k + 1, dim=1, largest=False)[1][:, 1:])
            near = torch.cat(near)
        d = x[:, None, :] - x[near]
        d -= per * Lf * torch.round(d / Lf)
        dist = d.square().sum(2).sqrt().clamp_min(1e-3)
        push = (r[:, None] + r[near] - dist).clamp_min(0.0) / dist
        x = x + 0.3 * (push[:, :, None] * d).sum(1)
        if layer:
            x[:, 2] = torch.minimum(torch.maximum(x[:, 2], r), Lf[2] - r)
        x = torch.remainder(x, Lf)
    return x.double()


def _cell_order(pos, box, cutoff):
    """Numbers the spheres cell by cell (x fastest), as the generators do."""
    key = torch.zeros(pos.shape[0], dtype=torch.int64, device=pos.device)
    for d in (2, 1, 0):
        m = max(1, int(box[d] / cutoff))
        c = ((pos[:, d] / box[d] + 0.5) * m).long().clamp(0, m - 1)
        key = key * m + c
    return torch.sort(key, stable=True)[1]


def _rect(center, half_u, half_w, u, w, n):
    return dict(kind="rect", center=center, half=(half_u, half_w), u=u, w=w, n=n)


def _floor(width, depth, z):
    return _rect((0.0, 0.0, z), width, depth, (1.0, 0.0, 0.0), (0.0, 1.0, 0.0), (0.0, 0.0, 1.0))


def _packing(case, seed):
    n, phi = case["n"], case["phi"]
    g = _generator(seed)
    k = max(1, math.ceil((n / 6000.0) ** (1 / 3) - 1e-9))
    tile = -(-n // k ** 3)
    radius = _uniform(g, (tile,), 0.4, 0.6)
    side = float((4.0 / 3.0 * math.pi * radius.pow(3).sum() / phi) ** (1 / 3))
    gas = phi < 0.62                     # below jamming: spheres about to touch
    x = _relaxed(radius, [side] * 3, g, 240 if phi < 0.58 else 600 if gas else 400,
                 1.001 + 0.06 * max(phi - 0.55, 0.0) if gas else 1.0)
    at = torch.arange(k, device=x.device, dtype=torch.float64)
    at = torch.stack(torch.meshgrid(at, at, at, indexing="ij"), -1).reshape(-1, 3)
    pos = (x[None] + (at * side)[:, None]).reshape(-1, 3)[:n] - 0.5 * k * side
    radius = radius.repeat(k ** 3)[:n]
    box = [k * side] * 3
    order = _cell_order(pos, box, 1.2)
    return dict(pos=pos[order], radius=radius[order], box=box, pbc=(True,) * 3, gravity=0.0,
                walls=[], dt=1e-4, e=0.8, mu=0.5, rmax=0.6, g=g)


def _column(radius, width, g):
    """A column of touching spheres, ``width`` x ``width`` periodic, lying on
    height 0, and its height."""
    height = float(4.0 / 3.0 * math.pi * radius.pow(3).sum() / 0.56) / width ** 2
    x = _relaxed(radius, [width, width, height], g, 240, layer=True)
    x[:, :2] -= 0.5 * width
    return x, height


def _floor_bed(case, seed):
    n = case["n"]
    g = _generator(seed)
    width = 10.0
    while n * 0.9 / width ** 2 > 4.0 * width:      # wide beds, not towers
        width += 10.0
    k = int(width / 10.0)
    tile = min(-(-n // k ** 2), 4000)
    radius = torch.full((tile,), 0.5, device=_device(), dtype=torch.float64)
    x, height = _column(radius, 10.0, g)
    layers = -(-n // (k * k * tile))
    at = torch.tensor([(10.0 * (i + 0.5) - 0.5 * width, 10.0 * (j + 0.5) - 0.5 * width, l * height)
                       for l in range(layers) for j in range(k) for i in range(k)],
                      device=x.device, dtype=torch.float64)
    pos = (x[None] + at[:, None]).reshape(-1, 3)
    pos = pos[torch.sort(pos[:, 2], stable=True)[1][:n]]
    lz = float(pos[:, 2].max()) + 20.0
    pos[:, 2] -= 0.5 * lz + 1e-4
    box = [width, width, lz]
    pos = pos[_cell_order(pos, box, 1.0)]
    return dict(pos=pos, radius=torch.full((n,), 0.5, device=pos.device, dtype=torch.float64),
                comp=[1.0], box=box, pbc=(True, True, False), gravity=1.0,
                walls=[_floor(width, width, -0.5 * lz)], dt=1e-4, e=0.8, mu=0.5, g=g)


def _box_bed(case, seed):
    n = case["n"]
    g = _generator(seed)
    a, b = 2.9997, 0.9999                          # sites of the two sizes, just touching
    n_large = max(1, round(n / 21))
    n_small = n - n_large
    blocks = -(-n_small // 27)
    sites = n_large + blocks
    m = max(3, round((2.0 * sites) ** (1 / 3)))    # a bed half as high as it is wide
    kind = torch.zeros(sites, dtype=torch.bool, device=_device())
    kind[torch.randperm(sites, generator=g, device=_device())[:n_large]] = True
    s = torch.arange(sites, device=_device())
    width = m * a
    layers = -(-sites // (m * m))
    lz = layers * a + 10.0
    c = torch.stack([(s % m + 0.5) * a - 0.5 * width, (s // m % m + 0.5) * a - 0.5 * width,
                     (s // (m * m) + 0.5) * a - 0.5 * lz], 1).double()
    o = torch.arange(3, device=_device(), dtype=torch.float64) - 1.0
    o = torch.stack(torch.meshgrid(o, o, o, indexing="ij"), -1).reshape(-1, 3) * b
    small = (c[~kind][:, None] + o[None]).reshape(-1, 3)[:n_small]
    pos = torch.cat([small, c[kind]])
    radius = torch.full((n,), 0.5, device=pos.device, dtype=torch.float64)
    radius[n_small:] = 1.5
    box = [width, width, lz]
    order = _cell_order(pos, box, 3.0)
    h, hz = 0.5 * width, 0.5 * lz
    X, Y, Z = (1.0, 0.0, 0.0), (0.0, 1.0, 0.0), (0.0, 0.0, 1.0)
    walls = [_floor(h + 1.0, h + 1.0, -hz),
             _rect((-h, 0.0, 0.0), h + 1.0, hz, Y, Z, X), _rect((h, 0.0, 0.0), h + 1.0, hz, Y, Z, X),
             _rect((0.0, -h, 0.0), h + 1.0, hz, X, Z, (0.0, -1.0, 0.0)),
             _rect((0.0, h, 0.0), h + 1.0, hz, X, Z, (0.0, -1.0, 0.0))]
    return dict(pos=pos[order], radius=radius[order], comp=[1.0, 3.0], box=box, pbc=(False,) * 3,
                gravity=1.0, walls=walls, dt=5e-5, e=0.7, mu=0.5, g=g)


def _hopper_bed(case, seed):
    n = case["n"]
    g = _generator(seed)
    slope, outlet = 0.55, 1.5                      # radius of the cone: outlet + slope * height
    pts, z = [], 0.7
    while len(pts) < n:
        room = outlet + slope * z - 0.5707
        m = int(room / 0.9999) + 1
        pts += [(i * 0.9999, j * 0.9999, z) for j in range(-m, m + 1) for i in range(-m, m + 1)
                if math.hypot(i, j) * 0.9999 < room]
        z += 0.9999
    pos = torch.tensor(pts[:n], device=_device(), dtype=torch.float64)
    height = z + 1.0
    top = outlet + slope * height
    width, lz = 2.0 * top + 12.0, height + 16.0
    pos[:, 2] += 6.0 - 0.5 * lz
    shake = dict(amplitude=(0.0, 0.0, 0.05), frequency=(0.0, 0.0, 4.0), phase=(0.0, 0.0, 0.25))
    cone = dict(kind="cone", center=(0.0, 0.0, 6.0 + 0.5 * height - 0.5 * lz), length=height,
                ends=(outlet, top), u=(0.0, 0.0, 1.0), w=(1.0, 0.0, 0.0), **shake)
    floor = dict(_floor(0.5 * width, 0.5 * width, 1.0 - 0.5 * lz), **shake)
    return dict(pos=pos, radius=torch.full((n,), 0.5, device=pos.device, dtype=torch.float64),
                comp=[1.0], box=[width, width, lz], pbc=(False,) * 3, gravity=10.0,
                walls=[cone, floor], dt=1e-4, e=0.7, mu=0.5, g=g)


def _ensemble(case, seed):
    g = _generator(seed)
    width = 10.0
    lo, hi = math.log(case["nmin"]), math.log(case["nmax"])
    draws = _uniform(g, (case["systems"], 2)).tolist()
    radius = _uniform(g, (2000,), 0.45, 0.55)
    x, height = _column(radius, width, g)
    beds = []
    sizes = torch.randperm(case["systems"], generator=g, device=x.device).tolist()
    for k, (e, mu) in zip(sizes, draws):          # sizes spread evenly over their logarithm
        n = round(math.exp(lo + (k + 0.5) / case["systems"] * (hi - lo)))
        layers = -(-n // 2000)
        up = torch.arange(layers, device=x.device, dtype=torch.float64) * height
        pos = x.repeat(layers, 1)
        pos[:, 2] += up.repeat_interleave(2000)
        order = torch.sort(pos[:, 2], stable=True)[1][:n]
        pos, r = pos[order], radius.repeat(layers)[order]
        lz = float(pos[:, 2].max()) + 20.0
        pos[:, 2] -= 0.5 * lz + 1e-4
        box = [width, width, lz]
        order = _cell_order(pos, box, 1.1)
        beds.append(dict(pos=pos[order], radius=r[order], box=box, pbc=(True, True, False),
                         gravity=1.0, walls=[_floor(width, width, -0.5 * lz)], dt=1e-4,
                         e=0.5 + 0.45 * e, mu=0.2 + 0.6 * mu, rmax=0.55, g=g))
    return beds


def _beds(case, seed):
    """The case's systems: geometry, materials, velocities N(0, 0.1^2)."""
    make = {"packing": _packing, "floor": _floor_bed, "box": _box_bed, "hopper": _hopper_bed}
    beds = _ensemble(case, seed) if case["bed"] == "ensemble" else [make[case["bed"]](case, seed)]
    for b in beds:
        b["vel"] = 0.1 * torch.randn(b["pos"].shape, generator=b.pop("g"), device=b["pos"].device,
                                     dtype=torch.float64)
    return beds


# ---------------------------------------------------------------------------
# the program

def _params(bed, prec):
    walls = []
    for w in bed["walls"]:
        if w["kind"] == "rect":
            walls.append(P.rectangle(w["center"], w["half"][0], w["half"][1], w["u"], w["w"],
                                     2.0 * KN, 2.0 * KT))
        else:
            walls.append(P.cone(w["center"], w["length"], 2.0 * w["ends"][0], 2.0 * w["ends"][1],
                                w["u"], w["w"], 2.0 * KN, 2.0 * KT))
    nw = len(walls)
    e, mu = bed["e"], bed["mu"]
    common = dict(lbox=bed["box"], pbc=bed["pbc"], gravity=(0.0, 0.0, -bed["gravity"]),
                  time_step=bed["dt"], method_order=ORDER, euler_intervals=EULER_INTERVALS,
                  max_ncell=1 << 30,
                  precision=P.PREC_MIXED if prec == "mixed" else P.PREC_FP64)
    if "comp" not in bed:
        return P.per_particle_params(density=DENSITY, kn=KN, kt=KT, en=e, et=e, mu=mu,
                                     rmax=bed["rmax"], walls=walls, knw=[KN] * nw, ktw=[KT] * nw,
                                     enw=[e] * nw, etw=[e] * nw, muw=[mu] * nw, hist_capacity=4,
                                     **common)
    k = len(bed["comp"])
    comps = [P.Component(0, d, DENSITY, 2.0 * KN, 2.0 * KT) for d in bed["comp"]]
    full, wide = lambda v: np.full((k, k), v), lambda v: np.full((k, nw), v)  # noqa: E731
    return P.component_params(comps, walls, full(e), full(e), full(mu), wide(e), wide(e), wide(mu),
                              **common)[0]


def _motions(bed):
    return [P.wall_motion(w["center"], w["amplitude"], w["frequency"], w["phase"])
            for w in bed["walls"]] if any("amplitude" in w for w in bed["walls"]) else None


def prepare(case, seed):
    """A system past its start-up steps, and the program's own host arrays."""
    beds = _beds(case, seed)
    host = {k: torch.cat([b[k] for b in beds]).cpu().numpy() for k in ("pos", "vel", "radius")}
    n = host["pos"].shape[0]
    prm = [_params(b, case["prec"]) for b in beds]
    if len(beds) > 1:
        s = DEMSystem.ensemble(prm, [b["pos"].shape[0] for b in beds])
    else:
        s = DEMSystem(prm[0])
    comp = None
    if "comp" in beds[0]:
        comp = (host["radius"] > 1.0).astype(np.int32)
    s.set_state(host["pos"], host["vel"], np.zeros((n, 3)), comp=comp,
                radius=None if comp is not None else host["radius"])
    motions = _motions(beds[0])
    if motions:
        s.set_wall_motion(motions)
    s.initialize_cell_distribution()
    s.run(1, ORDER - 1)
    pin = _device().type == "cuda"
    out = {k: torch.empty((n, 3), dtype=torch.float64, pin_memory=pin)
           for k in ("pos", "vel", "omega")}
    from dem3d_b200.system import _dptr
    state = dict(sys=s, out=out, ptr=[_dptr(out[k].numpy()) for k in ("pos", "vel", "omega")],
                 calls=case["calls"], steps=case["steps"], next=ORDER)
    _read(state)
    return state


def _read(st):
    st["sys"]._call("get_state", *st["ptr"], None, None)


def run(st):
    """``steps`` steps, then the state in the program's arrays."""
    s, first, k = st["sys"], st["next"], st["steps"]
    st["next"] = first + k
    if st["calls"] == "run":
        s.run(first, first + k - 1)
    for step in range(first, first + k) if st["calls"] != "run" else ():
        if st["calls"] == "coupled":
            if step > first:
                _read(st)
            s._call("update_state", *st["ptr"], None, None)
        s.move_particles(step)
    _read(st)
    return st["out"]


def _spheres(case):
    if case["bed"] != "ensemble":
        return float(case["n"])
    lo, hi = case["nmin"], case["nmax"]
    return case["systems"] * (hi - lo) / math.log(hi / lo)   # mean of a log-uniform size


def work(case):
    """One pass: per sphere and step the state and the ring of the integrator
    read and written once by two force passes (and the records of its
    contacts); per coupled step, and at the end, the state to the program."""
    z = {"packing": {0.55: 0.2, 0.60: 0.4, 0.65: 6.3}.get(case.get("phi"), 0.0), "floor": 4.0,
         "ensemble": 4.0, "box": 3.0, "hopper": 3.0}[case["bed"]]
    fp64 = case["prec"] == "fp64"
    per = 656.0 + 84.0 * z if fp64 else 608.0 + 48.0 * z
    flops = 300.0 + 2.0 * (6.0 * 15.0 + 0.5 * z * 250.0)
    copies = 2.0 * case["steps"] if case["calls"] == "coupled" else 1.0
    n = _spheres(case)
    return {"bytes": n * (case["steps"] * per + 72.0 * copies), "flops": n * case["steps"] * flops}


# ---------------------------------------------------------------------------
# the same steps in plain torch, 64 bits

def _damping(e):
    le = math.log(e)
    return -2.0 * le / math.sqrt(le * le + math.pi ** 2)


def _dot(a, b):
    return (a * b).sum(1, keepdim=True)


def _on_plane(v, n):
    """``v`` turned into the plane normal to ``n``, its length kept."""
    p = v - _dot(v, n) * n
    s = _dot(p, p)
    f = torch.where(s > 0, torch.sqrt(_dot(v, v) / torch.where(s > 0, s, torch.ones_like(s))),
                    torch.zeros_like(s))
    return f * p


class _Plain:
    """Linear springs and dashpots with Coulomb friction and remembered
    tangential springs; Adams-Bashforth-Moulton steps of order 4."""

    def __init__(self, bed):
        self.bed = bed
        self.x, self.v = bed["pos"].clone(), bed["vel"].clone()
        self.R = bed["radius"][:, None]
        self.n, self.dev = self.x.shape[0], self.x.device
        t = lambda *a: torch.tensor(a, device=self.dev, dtype=torch.float64)  # noqa: E731
        self.t = t
        self.w = torch.zeros_like(self.x)
        self.a, self.al = torch.zeros_like(self.x), torch.zeros_like(self.x)
        self.m = 4.0 * math.pi / 3.0 * DENSITY * self.R ** 3
        self.I = 0.4 * self.m * self.R ** 2
        self.L = t(*bed["box"])
        self.per = t(*[1.0 if p else 0.0 for p in bed["pbc"]])
        self.cut = 2.0 * (bed["rmax"] if "rmax" in bed else 0.5 * max(bed["comp"]))
        self.N = [int(b / self.cut) for b in bed["box"]]
        self.skin = 0.1
        self.x0 = None
        self.key = torch.zeros(0, dtype=torch.int64, device=self.dev)
        self.ft = self.vt = torch.zeros((0, 3), device=self.dev, dtype=torch.float64)
        self.wrec = [None] * len(bed["walls"])
        self.cell = self._cells(self.x)[3]
        self.entered = torch.zeros(self.n, dtype=torch.int64, device=self.dev)
        self.passes, self.time = 0, 0.0
        self.ring = []

    def _image(self, d):
        return d - self.per * self.L * torch.round(d / self.L)

    def _cells(self, x):
        c = [(x[:, k] * (self.N[k] / self.bed["box"][k]) + 0.5 * self.N[k]).long()
             .clamp(0, self.N[k] - 1) for k in range(3)]
        return c + [c[0] + self.N[0] * (c[1] + self.N[1] * c[2])]

    def _find_pairs(self, x):
        """All pairs nearer than contact plus a skin, in the order of their keys."""
        cx, cy, cz, c = self._cells(x)
        total = self.N[0] * self.N[1] * self.N[2]
        order = torch.sort(c)[1]
        count = torch.bincount(c, minlength=total)
        start = torch.cumsum(count, 0) - count
        found = []
        for o in range(14):
            d = (o % 3 - 1, o // 3 % 3 - 1, o // 9 - 1)
            ok = torch.ones(self.n, dtype=torch.bool, device=self.dev)
            q = []
            for k, ck in enumerate((cx, cy, cz)):
                j = ck + d[k]
                if not self.bed["pbc"][k]:
                    ok &= (j >= 0) & (j < self.N[k])
                q.append(j % self.N[k])
            other = q[0] + self.N[0] * (q[1] + self.N[1] * q[2])
            most = int(count.max())
            for k in range(most):
                i = torch.nonzero(ok & (count[other] > k))[:, 0]
                if not i.numel():
                    continue
                j = order[start[other[i]] + k]
                keep = i > j if o == 13 else i != j
                i, j = i[keep], j[keep]
                r = self._image(x[j] - x[i])
                near = (r * r).sum(1) < ((self.R[i] + self.R[j])[:, 0] + self.skin) ** 2
                found.append(torch.stack([torch.minimum(i[near], j[near]),
                                          torch.maximum(i[near], j[near])], 1))
        pairs = torch.cat(found) if found else torch.zeros((0, 2), dtype=torch.int64, device=self.dev)
        self.pairs = pairs[torch.sort(pairs[:, 0] * self.n + pairs[:, 1])[1]]
        self.x0 = x.clone()

    def _orient(self, a, b, cells):
        """The sphere that the sweep meets first comes first: by cell, within a
        cell the one that entered it last, then the higher index."""
        lex = torch.zeros_like(a)
        for k, f in ((0, 1), (1, 3), (2, 9)):
            d = cells[k][b] - cells[k][a]
            if self.bed["pbc"][k]:
                d = torch.where(d > 1, d - self.N[k], torch.where(d < -1, d + self.N[k], d))
            lex += f * d
        late = self.entered[b] - self.entered[a]
        swap = (lex < 0) | ((lex == 0) & ((late > 0) | ((late == 0) & (b > a))))
        return torch.where(swap, b, a), torch.where(swap, a, b)

    def _contact(self, N, disp, V, Vc, rv, gap2, half_dt, known, ft, vt, meff):
        e, mu = self.bed["e"], self.bed["mu"]
        yn, yt = _damping(e) * torch.sqrt(meff * KN), _damping(e) * torch.sqrt(meff * KT)
        vn = _dot(Vc, N) * N
        VT = Vc - vn
        FN = KN * disp + yn * vn
        vt0 = _on_plane(vt, N)
        old = _on_plane(ft, N) + KT * half_dt * (vt0 + VT) + yt * (VT - vt0)
        v2 = _dot(V, V)
        safe = torch.where(v2 > 0, v2, torch.ones_like(v2))
        part = torch.minimum((rv + torch.sqrt(rv * rv + v2 * gap2)) / safe,
                             torch.full_like(v2, 2.0 * half_dt))
        part = torch.where(v2 > 0, part, torch.zeros_like(v2))
        FT = torch.where(known[:, None], old, (KT * part + yt) * VT)
        top, t2 = mu * mu * _dot(FN, FN), _dot(FT, FT)
        FT = torch.where(t2 > top, torch.sqrt(top / t2.clamp_min(1e-300)) * FT, FT)
        return FN, FT, VT

    def _walls_now(self):
        for w in self.bed["walls"]:
            pos, vel = list(w["center"]), [0.0] * 3
            if "amplitude" in w:
                for k in range(3):
                    A, om, ph = (w["amplitude"][k], 2 * math.pi * w["frequency"][k],
                                 2 * math.pi * w["phase"][k])
                    pos[k] += A * (math.cos(om * self.time + ph) - math.cos(ph))
                    vel[k] = -A * om * math.sin(om * self.time + ph)
            if self.time == 0.0:
                vel = [0.0] * 3
            yield w, self.t(*pos)[None], self.t(*vel)[None]

    def _wall_geometry(self, w, pos, x):
        """Which spheres overlap the wall, their distance, normal and nearest point."""
        r = self._image(pos - x)
        u = self.t(*w["u"])[None]
        if w["kind"] == "rect":              # (faces only: no bed reaches an edge)
            n = self.t(*w["n"])[None]
            an = _dot(r, n)
            inside = an.abs() < self.R
            return inside[:, 0], an.abs(), torch.sign(an) * n, an * n - r
        ra, rp = w["ends"]
        half = 0.5 * w["length"]
        slant = math.hypot(w["length"], rp - ra)
        sn, cs = w["length"] / slant, (rp - ra) / slant
        au = _dot(r, u)
        rw = r - au * u
        aw = torch.sqrt(_dot(rw, rw))
        lam = (half - au) * sn - (ra - aw) * cs
        W = rw / aw.clamp_min(1e-300)
        face = (lam >= 0) & (lam <= slant)
        sd = -((half - au) * cs + (ra - aw) * sn)
        nf = torch.sign(sd) * (sn * W + cs * u)
        lc = lam.clamp(0.0, slant)
        edge = (sn * lc - (half - au)) * u - (cs * lc + (ra - aw)) * W
        de = torch.sqrt(_dot(edge, edge))
        D = torch.where(face, sd.abs(), de)
        N = torch.where(face, nf, edge / de.clamp_min(1e-300))
        return (D < self.R)[:, 0], D, N, D * N - r

    def force(self, x, v, w, half_dt, update):
        if self.x0 is None or float(self._image(x - self.x0).square().sum(1).max()) > (0.4 * self.skin) ** 2:
            self._find_pairs(x)
        self.passes += 1
        cells = self._cells(x)
        moved = cells[3] != self.cell
        self.entered = torch.where(moved, torch.full_like(self.entered, self.passes), self.entered)
        self.cell = cells[3]
        F = torch.zeros_like(x)
        F[:, 2] -= self.m[:, 0] * self.bed["gravity"]
        T = torch.zeros_like(x)
        a, b = self.pairs[:, 0], self.pairs[:, 1]
        r = self._image(x[b] - x[a])
        md = self.R[a] + self.R[b]
        near = (md * md - _dot(r, r))[:, 0] > 0
        a, b = a[near], b[near]
        key = a * self.n + b
        i, j = self._orient(a, b, cells)
        r = self._image(x[j] - x[i])
        md = self.R[i] + self.R[j]
        D = torch.sqrt(_dot(r, r))
        N = r / D
        V = v[j] - v[i]
        Vc = V - torch.cross(self.R[i] * w[i] + self.R[j] * w[j], N, dim=1)
        at = torch.searchsorted(self.key, key).clamp_max(max(self.key.numel() - 1, 0))
        if self.key.numel():
            known = self.key[at] == key
            ft, vt = self.ft[at], self.vt[at]
        else:
            known = torch.zeros_like(key, dtype=torch.bool)
            ft = vt = torch.zeros_like(r)
        meff = self.m[i] * self.m[j] / (self.m[i] + self.m[j])
        FN, FT, VT = self._contact(N, (D - md) * N, V, Vc, _dot(r, V), md * md - D * D, half_dt,
                                   known, ft, vt, meff)
        turn = torch.cross(N, FT, dim=1)
        F.index_add_(0, i, FN + FT)
        F.index_add_(0, j, FN + FT, alpha=-1.0)
        T.index_add_(0, i, self.R[i] * turn)
        T.index_add_(0, j, self.R[j] * turn)
        if update:
            self.key, self.ft, self.vt = key, FT, VT
        for k, (wall, pos, vel) in enumerate(self._walls_now()):
            hit, D, N, Q = self._wall_geometry(wall, pos, x)
            s = torch.nonzero(hit)[:, 0]
            D, N, Q, R = D[s], N[s], Q[s], self.R[s]
            V = vel - v[s]
            Vc = V - torch.cross(R * w[s], N, dim=1)
            rec = self.wrec[k]
            if rec is None:
                known = torch.zeros_like(s, dtype=torch.bool)
                ft = vt = torch.zeros_like(V)
            else:
                known, ft, vt = rec[0][s], rec[1][s], rec[2][s]
            FN, FT, VT = self._contact(N, (D - R) * N, V, Vc, _dot(pos + Q - x[s], V),
                                       R * R - D * D, half_dt, known, ft, vt, self.m[s])
            F[s] += FN + FT
            T[s] += torch.cross(R * N, FT, dim=1)
            if update:
                rec = [torch.zeros(self.n, dtype=torch.bool, device=self.dev),
                       torch.zeros_like(x), torch.zeros_like(x)]
                rec[0][s], rec[1][s], rec[2][s] = True, FT, VT
                self.wrec[k] = rec
        return F / self.m, T / self.I

    def start(self):
        for _ in range(ORDER - 1):
            self.ring.insert(0, (self.v.clone(), self.a.clone(), self.al.clone()))
            h = self.bed["dt"] / EULER_INTERVALS
            for _ in range(EULER_INTERVALS):
                self.a, self.al = self.force(self.x, self.v, self.w, 0.5 * h, True)
                self.x = self.x + self.v * h + self.a * (0.5 * h * h)
                self.v = self.v + self.a * h
                self.w = self.w + self.al * h
                self.time += h
            self.x = self._image(self.x)

    def step(self, number):
        c = self.bed["dt"] / 24.0
        ab, am = (55 * c, -59 * c, 37 * c, -9 * c), (9 * c, 19 * c, -5 * c, 1 * c)
        self.a, self.al = self.force(self.x, self.v, self.w, 0.5 * self.bed["dt"], True)
        now = (self.v, self.a, self.al)
        old = self.ring[:3]
        go = lambda y, C, rates: y + sum(f * q for f, q in zip(C, rates))  # noqa: E731
        xp = self._image(go(self.x, ab, [now[0]] + [q[0] for q in old]))
        vp = go(self.v, ab, [now[1]] + [q[1] for q in old])
        wp = go(self.w, ab, [now[2]] + [q[2] for q in old])
        self.time = number * self.bed["dt"]
        self.ring = [now] + old[:2]
        a2, al2 = self.force(xp, vp, wp, 0.5 * self.bed["dt"], False)
        old = self.ring
        self.x = self._image(go(self.x, am, [vp] + [q[0] for q in old]))
        self.v = go(self.v, am, [a2] + [q[1] for q in old])
        self.w = go(self.w, am, [al2] + [q[2] for q in old])


def exact(case, seed):
    out = []
    for bed in _beds(case, seed):
        s = _Plain(bed)
        s.start()
        for k in range(case["steps"]):
            s.step(ORDER + k)
        out.append((s.x, s.v, s.w))
    return {k: torch.cat([o[i] for o in out]) for i, k in enumerate(("pos", "vel", "omega"))}
