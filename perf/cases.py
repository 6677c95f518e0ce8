"""Timed work of the DEM step as its users run it, through the public entry points.

A case is a running simulation (or one call of it) of a kind that the workloads,
decks and tests of this repository hold: spheres in a box, settled cohesive beds,
batched rotating drums, spheres in a mesh mixer, falling, piled and densely packed
polyhedra, bonded blocks.  ``prepare`` builds the simulation from the seed, settled
where a user's run is settled, with the optimised switches on (graph step for
spheres), and ``run`` advances it (``dem_step``), calls the operators of a step one
by one, runs ``first_iteration``, or restarts it from particles on the device and
runs from there; each pass ends with the particles' state in device tensors, in id
order.  ``exact`` runs the same simulation in plain torch FP64 for the cases without
meshes and bonds.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from exadem_gb300 import _abi as A
from exadem_gb300 import workloads as W
from exadem_gb300.system import System

SPHERES = dict(fp32_broad_phase=1, fp32_contact_screen=1, fused_step=1, graph_step=1)
POLY = dict(fp32_broad_phase=1, fp32_contact_screen=1, fused_step=1)
GROUPS = {"r": ("rx", "ry", "rz"), "v": ("vx", "vy", "vz"), "a": ("fx", "fy", "fz"),
          "vrot": ("vrotx", "vroty", "vrotz"), "arot": ("arotx", "aroty", "arotz"),
          "mom": ("momx", "momy", "momz"), "quat": ("qw", "qx", "qy", "qz")}
FIELDS = [f for g in GROUPS.values() for f in g]


def listed():
    return [
        # a small box advanced one step per call, as a coupled code does it: latency
        {"name": "box 1k, one step a call", "kind": "box", "n": 1000, "steps": 1},
        # the CPU-runnable box of the repository's first configuration
        {"name": "box 10k", "kind": "box", "n": 10000, "steps": 50},
        # beds of polydisperse cohesive spheres with rolling, periodic in x and y
        {"name": "cohesive bed 125k", "kind": "bed", "n": 125000, "law": "cohesive", "steps": 20},
        {"name": "cohesive bed 2M", "kind": "bed", "n": 2000000, "law": "cohesive", "steps": 5},
        # uneven rotating drums in one context
        {"name": "drums 40 x 1k-20k", "kind": "drums", "systems": 40, "nmin": 1000, "nmax": 20000, "steps": 20},
        # the operators of one step called one by one, as a deck's graph engine does it
        {"name": "bed 53k, operators", "kind": "bed", "n": 53000, "law": "none", "steps": 2, "operators": True},
        # polyhedra let fall: a run started from particles on the device
        {"name": "falling polyhedra 200k", "kind": "fall", "n": 200000, "steps": 100},
        # a small pile of polyhedra, many contacts per particle
        {"name": "pile of polyhedra 1.5k", "kind": "pile", "nx": 11, "ny": 11, "nz": 12, "steps": 20},
        # neighbour build and first forces of densely packed polyhedra: every rebuild does this
        {"name": "dense polyhedra 27k, forces", "kind": "forces", "nx": 30, "ny": 30, "nz": 30},
        # spheres at rest and moving in a triangle mesh
        {"name": "mixer mesh 50k", "kind": "mixer", "n": 50000, "steps": 20},
        # bonded blocks of cubes: steps between two breaks, and the build that a break forces
        {"name": "bonded cubes 16k", "kind": "bonded", "blocks": 128, "steps": 10},
        {"name": "bonded cubes 8k, forces", "kind": "bonded", "blocks": 64, "steps": 0},
    ]


def draw(rng):
    def log(lo, hi):
        return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))

    kind = rng.choice(["box", "bed", "bed", "operators", "drums", "fall", "pile", "forces", "mixer", "bonded"])
    if kind == "box":
        n = log(1000, 40000)
        return {"kind": "box", "n": n, "steps": rng.choice([1, log(2, 60)])}
    if kind == "bed":
        n = log(10000, 1500000)
        return {"kind": "bed", "n": n, "law": rng.choice(["cohesive", "none"]), "steps": max(2, min(40, 3000000 // n))}
    if kind == "operators":
        return {"kind": "bed", "n": log(5000, 300000), "law": "none", "steps": rng.randint(1, 3), "operators": True}
    if kind == "drums":
        return {"kind": "drums", "systems": rng.randint(3, 60), "nmin": 1000, "nmax": log(4000, 30000),
                "steps": rng.randint(5, 25)}
    if kind == "fall":
        return {"kind": "fall", "n": log(5000, 190000), "steps": rng.randint(20, 100)}
    if kind == "pile":
        return {"kind": "pile", "nx": rng.randint(4, 16), "ny": rng.randint(4, 16), "nz": rng.randint(3, 12),
                "steps": rng.randint(5, 25)}
    if kind == "forces":
        return {"kind": "forces", "nx": rng.randint(6, 32), "ny": rng.randint(6, 30), "nz": rng.randint(6, 28)}
    if kind == "mixer":
        return {"kind": "mixer", "n": log(4000, 50000), "steps": rng.randint(5, 25)}
    return {"kind": "bonded", "blocks": rng.randint(4, 120), "steps": rng.choice([0, rng.randint(2, 12)])}


def work(case):
    n, s = _count(case), max(1, case.get("steps", 1))
    # listed pairs per particle; 344 bytes a particle and step (19 doubles read and
    # written, 5 read), 104 a pair and step (history read and written, two indices)
    per = {"box": 1.0, "bed": 3.3, "drums": 2.5, "fall": 0.1, "pile": 12.0, "forces": 14.0, "mixer": 2.0, "bonded": 26.0}
    pairs = per[case["kind"]] * n
    if case["kind"] == "forces" or (case["kind"] == "bonded" and not case["steps"]):
        return {"bytes": n * 250.0 + pairs * (76.0 + 104.0), "flops": n * 150.0 + pairs * 150.0}
    return {"bytes": s * (n * 344.0 + pairs * 104.0), "flops": s * (n * 280.0 + pairs * 150.0)}


def _count(case):
    k = case["kind"]
    if k in ("pile", "forces"):
        return case["nx"] * case["ny"] * case["nz"]
    if k == "bonded":
        return case["blocks"] * 125
    if k == "drums":
        return int(case["systems"] * (case["nmax"] - case["nmin"]) / math.log(case["nmax"] / case["nmin"]))
    return case["n"]


# ------------------------------------------------------------------ inputs
def _bed(case, seed):
    """A settled bed about 12 deep: one periodic patch of at most about 20,000 spheres is
    deposited, and its copies side by side, each with velocities of its own, are the bed."""
    tiles = max(1, round(math.sqrt(case["n"] / 20000)))
    npatch = case["n"] // (tiles * tiles)
    side = 400.0 * math.sqrt(npatch / 2_000_000)
    w = W.spheres_floor(n=npatch, side=side, seed=seed, rsa_attempts=64, **SPHERES)
    if case["law"] == "none":
        cfg = dict(kn=1e4, kt=8e3, kr=0.0, mu=0.3, damp_rate=0.9)
        w.params.law = A.LAW_HOOKE_NONE
        w.params.config = w.params.config_driver = W.contact_params(**cfg)
    s = w.build()
    s.first_iteration()
    s.step(3000)
    p = s.particles()
    s.close()
    lo, hi = list(w.params.bounds_lo), list(w.params.bounds_hi)
    rng = np.random.default_rng(seed)
    m = tiles * tiles
    q = {k: np.tile(v, m) for k, v in p.items()}
    t = np.repeat(np.arange(m), npatch)
    q["rx"] = np.minimum(np.maximum(q["rx"], lo[0]), np.nextafter(hi[0], lo[0])) + (t % tiles) * side
    q["ry"] = np.minimum(np.maximum(q["ry"], lo[1]), np.nextafter(hi[1], lo[1])) + (t // tiles) * side
    for k in ("vx", "vy", "vz"):
        q[k] = q[k] + rng.uniform(-0.01, 0.01, m * npatch)
    q["id"] = p["id"][np.tile(np.arange(npatch), m)] * np.uint64(m) + t.astype(np.uint64)
    o = np.argsort(q["id"])
    w.particles = {k: np.ascontiguousarray(v[o]) for k, v in q.items()}
    w.particles["id"] = np.arange(m * npatch, dtype=np.uint64)
    w.params.bounds_hi[0] = side * tiles
    w.params.bounds_hi[1] = side * tiles
    return w


def _drums(case, seed):
    """Drums of log-uniform sizes (the case's, not the seed's), as workloads.drums_batch lays them out."""
    rng = np.random.default_rng(5)
    lo, hi = math.log(case["nmin"]), math.log(case["nmax"])
    counts = np.exp(rng.uniform(lo, hi, case["systems"])).astype(np.int64)
    first = np.concatenate([[0], np.cumsum(counts)[:-1]])

    def drum(k, again=0):  # a random placement that jams is drawn again
        try:
            return W.spheres_drum(n=int(counts[k]), seed=seed * 1000 + k + again * 7919, id_offset=int(first[k]), **SPHERES)
        except A.DemError:
            if again == 9:
                raise
            return drum(k, again + 1)

    members = [drum(k) for k in range(case["systems"])]
    return W.BatchWorkload("drums", members[0].params, members)


def _fall(case, seed):
    """Cubes, tetrahedra and octahedra at random orientations, their circumscribed spheres
    just apart (solid fraction of the spheres about 0.36), above a floor and inside walls."""
    n = case["n"]
    shapes = [W.shape_cube(1.0, 0.01), W.shape_tetrahedron(1.2, 0.01), W.shape_octahedron(1.0, 0.01)]
    rng = np.random.default_rng(seed)
    nx = max(3, round(math.sqrt(n / 43.0)))
    k = np.arange(n)
    pos = np.stack([k % nx, (k // nx) % nx, k // (nx * nx)], 1) * 1.78 + 0.92 + rng.uniform(-0.01, 0.01, (n, 3))
    arr = W.empty_particles(n)
    types = rng.integers(0, 3, n).astype(np.uint32)
    q = rng.standard_normal((n, 4))
    q /= np.linalg.norm(q, axis=1)[:, None]
    for c, f in enumerate(("rx", "ry", "rz")):
        arr[f] = np.ascontiguousarray(pos[:, c])
    for c, f in enumerate(("qw", "qx", "qy", "qz")):
        arr[f] = np.ascontiguousarray(q[:, c])
    arr["vz"] = rng.uniform(-1.0, 0.0, n)
    arr["type"], arr["id"] = types, np.arange(n, dtype=np.uint64)
    arr["radius"] = np.array([s["max_rcut"] for s in shapes])[types]
    arr["mass"] = 0.02 * np.array([s["volume"] for s in shapes])[types]
    for f in ("inertiax", "inertiay", "inertiaz"):
        arr[f] = arr["mass"] * np.array([s["i_over_m"] for s in shapes])[types]
    arr["homothety"] = np.ones(n)
    side = nx * 1.78 + 0.06
    cfg = dict(kn=1e5, kt=8e4, kr=0.0, mu=0.5, damp_rate=0.9)
    p = W.make_params((0, 0, 0), (side, side, float(pos[:, 2].max()) + 2.0), (0, 0, 0), rcut_inc=0.05, dt=1e-4,
                      gravity=(0, 0, -9.81), config=cfg, config_driver=cfg, **POLY)
    walls = [dict(offset=0.0, normal=(0.0, 0.0, 1.0)), dict(offset=0.0, normal=(1.0, 0.0, 0.0)),
             dict(offset=side, normal=(1.0, 0.0, 0.0)), dict(offset=0.0, normal=(0.0, 1.0, 0.0)),
             dict(offset=side, normal=(0.0, 1.0, 0.0))]
    w = W.Workload("falling_polyhedra", p, arr, surfaces=walls)
    w.shapes = shapes
    return w


def _workload(case, seed):
    k = case["kind"]
    if k == "box":
        return W.spheres_box(n=case["n"], box=30.0 * (case["n"] / 10000) ** (1 / 3), density=2.0, seed=seed, **SPHERES)
    if k == "bed":
        return _bed(case, seed)
    if k == "drums":
        return _drums(case, seed)
    if k == "fall":
        return _fall(case, seed)
    if k in ("pile", "forces"):
        return W.polyhedra_lattice(nx=case["nx"], ny=case["ny"], nz=case["nz"], seed=seed, **POLY)
    if k == "mixer":
        return W.spheres_mixer(n=case["n"], seed=seed, **SPHERES)
    bond = dict(kn=1e4, kt=8e3, damp_rate=0.87, g=1e9)  # holds: the run stays between two breaks
    return W.fragment_blocks(nblocks=case["blocks"], nx=5, ny=5, nz=5, seed=seed, bond=bond, **POLY)


# steps after which a run of the kind has settled; it goes on from the particles of that step
PREROLL = {"box": 2500, "drums": 2000, "pile": 300, "mixer": 1200}


def _settle(w, steps):
    s = w.build()
    s.first_iteration()
    s.step(steps)
    p = s.particles()
    s.close()
    first = 0
    for m in getattr(w, "members", [w]):
        m.particles = {k: np.ascontiguousarray(v[first: first + m.n]) for k, v in p.items()}
        first += m.n


def prepare(case, seed):
    w = _workload(case, seed)
    if case["kind"] in PREROLL:
        _settle(w, PREROLL[case["kind"]])
    st = {"case": dict(case), "w": w}
    s = st["s"] = w.build()
    n = st["n"] = s.n
    if case["kind"] == "fall":
        st["dev"] = _to_device(w.particles)
    else:
        s.first_iteration()
    st["stream"] = torch.cuda.ExternalStream(s.stream_handle())
    with torch.cuda.stream(st["stream"]):
        st["buf"] = torch.empty((len(FIELDS), n), dtype=torch.float64, device="cuda")
        st["id"] = torch.empty(n, dtype=torch.int64, device="cuda")
    out = A.Particles()
    out.n = n
    for k, f in enumerate(FIELDS):
        setattr(out, f, C.cast(C.c_void_p(st["buf"][k].data_ptr()), C.POINTER(C.c_double)))
    out.id = C.cast(C.c_void_p(st["id"].data_ptr()), C.POINTER(C.c_uint64))
    st["out"] = out
    return st


def _to_device(arrays):
    """The particles as device tensors, and the struct that hands them to dem_set_particles."""
    keep, p = [], A.Particles()
    p.n = len(arrays["rx"])
    ct = {"id": (C.c_uint64, np.int64), "type": (C.c_uint32, np.int32), "group": (C.c_uint32, np.int32)}
    for k, v in arrays.items():
        c, view = ct.get(k, (C.c_double, None))
        t = torch.from_numpy(np.ascontiguousarray(v).view(view) if view else np.ascontiguousarray(v, dtype=np.float64)).cuda()
        keep.append(t)
        setattr(p, k, C.cast(C.c_void_p(t.data_ptr()), C.POINTER(c)))
    torch.cuda.current_stream().synchronize()
    return p, keep


def _operators(s):
    s.combined_compute_prolog()
    if s.particle_displ_over():
        s.update_particle_neighbors()
    s.reset_force_moment()
    s.gravity_force()
    s.contact_sphere()
    s.force_to_accel()
    s.combined_compute_epilog()


def run(st):
    s, case = st["s"], st["case"]
    steps = case.get("steps", 0)
    if case["kind"] == "fall":
        s._check(s.b.set_particles(s.h, C.byref(st["dev"][0]), 1), "set_particles")
        s.first_iteration()
        s.step(steps)
    elif not steps:
        s.first_iteration()
    elif case.get("operators"):
        for _ in range(steps):
            _operators(s)
    else:
        s.step(steps)
    with torch.cuda.stream(st["stream"]):
        s._check(s.b.get_particles(s.h, C.byref(st["out"]), 1), "get_particles")
        ordered = st["buf"][:, torch.argsort(st["id"])]
        return _groups(ordered)


def _groups(rows):
    at, out = 0, {}
    for g, f in GROUPS.items():
        out[g] = rows[at: at + len(f)]
        at += len(f)
    return out


# ---------------------------------------------------- the same in torch, FP64
def exact(case, seed):
    if case["kind"] in ("mixer", "bonded"):
        return None  # mesh bins and bond interfaces: no plain form of a few seconds
    if case["kind"] in ("fall", "forces", "pile") and _count(case) * max(1, case.get("steps", 1)) > 30_000_000:
        return None
    st = prepare(case, seed)
    w, s = st["w"], st["s"]
    s.close()
    sim = (_Poly if case["kind"] in ("fall", "forces", "pile") else _Spheres)(w)
    sim.rebuild()
    sim.forces(True)
    if case["kind"] == "forces":
        sim.rebuild()
        sim.forces(True)
    for _ in range(case.get("steps", 0)):
        sim.step()
    return {g: t.cpu() for g, t in sim.state().items()}


def _cross(a, b):
    return torch.linalg.cross(a, b)


def _dot(a, b):
    return (a * b).sum(-1)


def _rot(q, v):
    u = q[:, 1:]
    t = _cross(u, v)
    return v + 2 * q[:, :1] * t + 2 * _cross(u, t)


class _Sim:
    """Velocity Verlet as the deck runs it: prolog, trigger and rebuild, forces, epilog."""

    def __init__(self, w):
        arrays = w.particles() if callable(w.particles) else w.particles
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        o = np.argsort(arrays["id"])
        t = lambda v: torch.from_numpy(np.ascontiguousarray(v[o])).to(self.dev)  # noqa: E731
        v3 = lambda f: torch.stack([t(arrays[x]) for x in GROUPS[f]], 1)  # noqa: E731
        self.r, self.v, self.a, self.w = v3("r"), v3("v"), v3("a"), v3("vrot")
        self.ar, self.mom, self.q = v3("arot"), v3("mom"), v3("quat")
        self.m, self.rad = t(arrays["mass"]), t(arrays["radius"])
        self.I = torch.stack([t(arrays[k]) for k in ("inertiax", "inertiay", "inertiaz")], 1)
        self.type = t(arrays["type"].astype(np.int64)) if "type" in arrays else None
        p = self.p = w.params
        self.n, self.dt, self.skin = len(self.m), p.dt, p.rcut_inc
        self.g = torch.tensor(list(p.gravity), dtype=torch.float64, device=self.dev)
        self.coh = p.law == A.LAW_HOOKE_COHESIVE
        self.keys = torch.zeros(0, dtype=torch.int64, device=self.dev)  # touching pairs and their history
        self.ft = torch.zeros((0, 3), dtype=torch.float64, device=self.dev)
        self.mo = torch.zeros((0, 3), dtype=torch.float64, device=self.dev)

    def state(self):
        rows = {"r": self.r, "v": self.v, "a": self.a, "vrot": self.w, "arot": self.ar, "mom": self.mom, "quat": self.q}
        return {k: x.T.contiguous() for k, x in rows.items()}

    def history(self, key):
        """Friction and moment of the pairs `key` from the last pass (zero for a new pair)."""
        ft = torch.zeros((len(key), 3), dtype=torch.float64, device=self.dev)
        mo = torch.zeros_like(ft)
        if len(self.keys) and len(key):
            at = torch.searchsorted(self.keys, key).clamp(max=len(self.keys) - 1)
            hit = self.keys[at] == key
            ft[hit], mo[hit] = self.ft[at[hit]], self.mo[at[hit]]
        return ft, mo

    def remember(self, key, ft, mo):
        self.keys, o = torch.sort(key)
        self.ft, self.mo = ft[o], mo[o]

    def law(self, cfg, dn, n, cp, ft, mo, meff, ri, vi, wi, rj, vj, wj):
        """Force on i, new friction and moment (contact_force.hpp:146-235, mur = 0)."""
        pre = self.coh & (dn >= 0) if self.coh else torch.zeros_like(dn, dtype=torch.bool)
        rel = (vj - _cross(cp - rj, wj)) - (vi - _cross(cp - ri, wi))
        vn = _dot(rel, n)
        nf = (cfg.damp_rate * 2 * torch.sqrt(cfg.kn * meff) * vn - cfg.kn * dn).clamp(min=0)
        if self.coh:
            nf = (nf - cfg.fc).clamp(min=-cfg.fc)
        fn = nf[:, None] * n
        ft = ft + cfg.kt * self.dt * (rel - vn[:, None] * n)
        thr = (cfg.mu * (nf + cfg.fc if self.coh else cfg.kn * dn)).abs()
        f2 = _dot(ft, ft)
        slip = (f2 > 0) & (f2 > thr * thr)
        ft = torch.where(slip[:, None], ft * (thr / torch.sqrt(torch.where(f2 > 0, f2, torch.ones_like(f2))))[:, None], ft)
        mo2 = mo + cfg.kr * (wj - wi) * self.dt
        mo2 = torch.where((wi == 0).all(1)[:, None], mo2, torch.zeros_like(mo2))
        f = fn + ft
        if self.coh:
            f = torch.where(pre[:, None], ((cfg.fc / cfg.dncut) * dn - cfg.fc)[:, None] * n, f)
            ft = torch.where(pre[:, None], torch.zeros_like(ft), ft)
            mo2 = torch.where(pre[:, None], mo, mo2)
        return f, ft, mo2

    def add(self, i, f, t):
        self.f.index_add_(0, i, f)
        self.t.index_add_(0, i, t)

    def forces(self, first):
        self.f = self.m[:, None] * self.g
        self.t = torch.zeros_like(self.f)
        self.contacts()
        self.mom = self.t
        if first:
            self.a = self.f  # the deck's first iteration leaves the force in f
            return
        dt2 = 0.5 * self.dt
        self.a = self.f / self.m[:, None]
        qi = self.q * torch.tensor([1.0, -1.0, -1.0, -1.0], dtype=torch.float64, device=self.dev)
        om, tb, I = _rot(qi, self.w), _rot(qi, self.t), self.I
        num = tb - torch.stack([(I[:, 2] - I[:, 1]) * om[:, 1] * om[:, 2], (I[:, 0] - I[:, 2]) * om[:, 2] * om[:, 0],
                                (I[:, 1] - I[:, 0]) * om[:, 0] * om[:, 1]], 1)
        self.ar = _rot(self.q, num / I)
        self.w = self.w + self.ar * dt2
        self.v = self.v + self.a * dt2

    def step(self):
        dt, dt2 = self.dt, 0.5 * self.dt
        self.r = self.r + (self.v * dt + self.a * (dt * dt * 0.5))
        self.v = self.v + self.a * dt2
        q, om = self.q, self.w
        d = torch.cat([-0.5 * _dot(om, q[:, 1:])[:, None], 0.5 * (_cross(om, q[:, 1:]) + om * q[:, :1])], 1)
        q = q + d * dt
        self.q = q / torch.sqrt(_dot(q, q))[:, None]
        self.w = om + self.ar * dt2
        self.trigger()
        self.forces(False)


def _near(pos, nreal, cut):
    """(i, j) with i < nreal and |pos_i - pos_j| < cut_i + cut_j, i != j; cut: one value a point."""
    size = 2 * float(cut.max())
    c = torch.floor((pos - pos.min(0).values) / size).long() + 1
    dims = c.max(0).values + 2
    key = (c[:, 0] * dims[1] + c[:, 1]) * dims[2] + c[:, 2]
    skey, order = torch.sort(key)
    out_i, out_j = [], []
    me = torch.arange(nreal, device=pos.device)
    for dx in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dz in (-1, 0, 1):
                k = key[:nreal] + (dx * dims[1] + dy) * dims[2] + dz
                at, end = torch.searchsorted(skey, k), torch.searchsorted(skey, k, right=True)
                i = me
                while True:
                    ok = at < end
                    if not bool(ok.any()):
                        break
                    i, at, end = i[ok], at[ok], end[ok]
                    j = order[at]
                    d = pos[i] - pos[j]
                    hit = (_dot(d, d) < (cut[i] + cut[j]) ** 2) & (i != j)
                    out_i.append(i[hit])
                    out_j.append(j[hit])
                    at = at + 1
    return torch.cat(out_i), torch.cat(out_j)


class _Spheres(_Sim):
    def __init__(self, w):
        super().__init__(w)
        members = getattr(w, "members", [w])
        sizes = torch.tensor([m.n for m in members])
        self.sys = torch.repeat_interleave(torch.arange(len(members)), sizes).to(self.dev)
        par = lambda k: torch.tensor([list(getattr(m.params, k)) for m in members], dtype=torch.float64,  # noqa: E731
                                     device=self.dev)
        self.lo, self.L = par("bounds_lo"), par("bounds_hi") - par("bounds_lo")
        self.per = par("periodic") > 0
        self.drv = []
        for k, m in enumerate(members):
            for c, d in enumerate(m.surfaces + m.cylinders):
                self.drv.append((k, c, d))

    def rebuild(self, which=None):
        which = torch.ones(len(self.L), dtype=torch.bool, device=self.dev) if which is None else which
        lo, L, per = self.lo[self.sys], self.L[self.sys], self.per[self.sys]
        wrap = torch.where(per & which[self.sys][:, None], -torch.floor((self.r - lo) / L), torch.zeros_like(self.r))
        self.r = self.r + wrap * L
        self.bak = torch.where(which[self.sys][:, None], self.r, getattr(self, "bak", self.r))
        self.find()

    def find(self):
        """Pairs within the skin, with the images across periodic faces as extra points."""
        cut = self.rad + 0.5 * self.skin + 0.03
        pos, src, shift = self.r, torch.arange(self.n, device=self.dev), torch.zeros_like(self.r)
        for d in range(3):
            if not bool(self.per[:, d].any()):
                continue
            L, lo, on = self.L[self.sys[src], d], self.lo[self.sys[src], d], self.per[self.sys[src], d]
            add = []
            for sign, edge in ((1.0, pos[:, d] < lo + 1.5), (-1.0, pos[:, d] > lo + L - 1.5)):
                g = edge & on
                s2 = shift[g].clone()
                s2[:, d] += sign
                p2 = pos[g].clone()
                p2[:, d] += sign * L[g]
                add.append((p2, src[g], s2))
            pos = torch.cat([pos] + [x[0] for x in add])
            src = torch.cat([src] + [x[1] for x in add])
            shift = torch.cat([shift] + [x[2] for x in add])
        apart = pos.clone()
        apart[:, 0] += self.sys[src] * (2 * float(self.L.max()) + 10)
        i, j = _near(apart, self.n, cut[src])
        keep = (src[j] > i) | (j >= self.n)
        self.i, j = i[keep], j[keep]
        self.j, self.img = src[j], j >= self.n
        self.shift = shift[j] * self.L[self.sys[self.i]]

    def trigger(self):
        d = self.r - self.bak
        over = _dot(d, d) >= (0.5 * self.skin) ** 2
        which = torch.zeros(len(self.L), dtype=torch.bool, device=self.dev)
        which[self.sys[over]] = True
        if bool(which.any()):
            self.rebuild(which)

    def contacts(self):
        i, j = self.i, self.j
        rj = self.r[j] + self.shift
        d = self.r[i] - rj
        dist = torch.sqrt(_dot(d, d))
        dn = dist - (self.rad[i] + self.rad[j])
        cfg = self.p.config
        hit = (dn < 0) | (dn <= cfg.dncut) if self.coh else dn < 0
        i, j, rj, dn, n, img = i[hit], j[hit], rj[hit], dn[hit], d[hit] / dist[hit][:, None], self.img[hit]
        cp = self.r[i] - n * (self.rad[i] + 0.5 * dn)[:, None]
        key = i * (1 << 31) + j
        ft, mo = self.history(key)
        meff = self.m[i] * self.m[j] / (self.m[i] + self.m[j])
        f, ft, mo = self.law(cfg, dn, n, cp, ft, mo, meff, self.r[i], self.v[i], self.w[i], rj, self.v[j], self.w[j])
        self.add(i, f, _cross(cp - self.r[i], f) + mo)
        o = ~img
        self.add(j[o], -f[o], (_cross(cp - rj, -f) - mo)[o])
        keys, fts, mos = [key], [ft], [mo]
        cfg = self.p.config_driver
        for k, index, dv in self.drv:
            i = torch.nonzero(self.sys == k)[:, 0]
            key, f, ft, mo, cp, i = self.driver(cfg, dv, index, i, self.r[i], self.rad[i])
            self.add(i, f, _cross(cp - self.r[i], f) + mo)
            keys.append(key)
            fts.append(ft)
            mos.append(mo)
        self.remember(torch.cat(keys), torch.cat(fts), torch.cat(mos))

    def driver(self, cfg, dv, index, i, pt, rad):
        vec = lambda k: torch.tensor(dv.get(k, (0.0, 0.0, 0.0)), dtype=torch.float64, device=self.dev)  # noqa: E731
        if "normal" in dv:
            nrm = vec("normal")
            d = _dot(pt, nrm)[:, None] * nrm - dv["offset"] * nrm
            dist = torch.sqrt(_dot(d, d))
            dn, centre = dist - rad, dv["offset"] * nrm
        else:
            centre = vec("axis") * vec("center")
            d = centre - pt * vec("axis")
            dist = torch.sqrt(_dot(d, d))
            dn = dv["radius"] - (rad + dist)
        hit = dn <= cfg.dncut if self.coh else dn <= 0
        i, pt, rad, dn, n = i[hit], pt[hit], rad[hit], dn[hit], d[hit] / dist[hit][:, None]
        n = torch.where((dn <= 0)[:, None], n, torch.zeros_like(n))  # the detector's normal before contact
        cp = pt - n * (rad + 0.5 * dn)[:, None]
        key = -(i * 1024 + index) - 1
        if self.sub is not None:
            key = -((i * 1024 + index) * 64 + self.sub[hit]) - 1
        ft, mo = self.history(key)
        z = torch.zeros_like(cp)
        f, ft, mo = self.law(cfg, dn, n, cp, ft, mo, self.m[i], self.r[i], self.v[i], self.w[i], z + centre, z,
                             z + vec("vrot"))
        return key, f, ft, mo, cp, i

    sub = None


class _Poly(_Spheres):
    """Polyhedra: the features listed at the last build (filters with the skin), each detected anew."""

    def __init__(self, w):
        _Sim.__init__(self, w)
        self.drv = [(0, c, d) for c, d in enumerate(w.surfaces + w.cylinders)]
        sh = w.shapes
        T = lambda x, dt: torch.tensor(x, dtype=dt, device=self.dev)  # noqa: E731
        mv, me, mf = (max(len(s[k]) for s in sh) for k in ("vertices", "edges", "faces"))
        ms = max(len(f) for s in sh for f in s["faces"])
        pad = lambda rows, m, fill: [list(r) for r in rows] + [list(fill)] * (m - len(rows))  # noqa: E731
        self.V = T([pad(np.asarray(s["vertices"]).tolist(), mv, (0, 0, 0)) for s in sh], torch.float64)
        self.E = T([pad(np.asarray(s["edges"]).tolist(), me, (0, 0)) for s in sh], torch.int64)
        self.F = T([pad([list(f) + [f[0]] * (ms - len(f)) for f in s["faces"]], mf, [0] * ms) for s in sh], torch.int64)
        self.nv, self.ne, self.nf = (T([len(s[k]) for s in sh], torch.int64) for k in ("vertices", "edges", "faces"))
        self.fs = T([[len(f) for f in s["faces"]] + [3] * (mf - len(s["faces"])) for s in sh], torch.int64)
        self.mr = sh[0]["radius"]
        self.vertices()

    def key(self, kind, i, si, j, sj):
        return (((kind * (1 << 20) + i) * 32 + si) * (1 << 20) + j) * 32 + sj

    def vertices(self):
        v = self.V[self.type]
        u, q0 = self.q[:, None, 1:].expand_as(v), self.q[:, None, :1]
        t = _cross(u, v)
        self.x = self.r[:, None] + (v + 2 * q0 * t + 2 * _cross(u, t))

    def trigger(self):
        self.vertices()
        d = self.x - self.bak
        real = torch.arange(self.V.shape[1], device=self.dev)[None] < self.nv[self.type][:, None]
        if bool(((_dot(d, d) >= (0.5 * self.skin) ** 2) & real).any()):
            self.rebuild()

    def rebuild(self):
        self.vertices()
        self.bak = self.x.clone()
        self.find()

    def find(self):
        pi, pj = _near(self.r, self.n, self.rad + 0.5 * self.skin)
        pairs = pi < pj
        pi, pj = pi[pairs], pj[pairs]
        got = [[], [], [], [], []]
        for a in range(0, len(pi), 20000):
            for kind, i, j in ((0, pi, pj), (1, pi, pj), (1, pj, pi), (2, pi, pj), (2, pj, pi), (3, pi, pj)):
                ii, jj = i[a: a + 20000], j[a: a + 20000]
                ni = (self.ne if kind == 3 else self.nv)[self.type[ii]]
                nj = (self.nv, self.ne, self.nf, self.ne)[kind][self.type[jj]]
                mi, mj = int(ni.max()), int(nj.max())
                si, sj = torch.meshgrid(torch.arange(mi, device=self.dev), torch.arange(mj, device=self.dev), indexing="ij")
                ok = (si[None] < ni[:, None, None]) & (sj[None] < nj[:, None, None])
                p, s, t = torch.nonzero(ok, as_tuple=True)
                c, _, _, _ = self.detect(kind, ii[p], s, jj[p], t, self.skin)
                for k, v in enumerate((torch.full_like(s[c], kind), ii[p[c]], s[c], jj[p[c]], t[c])):
                    got[k].append(v)
        self.feat = [torch.cat(g) if g else torch.zeros(0, dtype=torch.int64, device=self.dev) for g in got]

    def detect(self, kind, i, si, j, sj, skin):
        """(touches, dn, n, cp) of feature si of i against sj of j; with a skin, the list's filter."""
        R = 2 * self.mr + skin
        if kind == 3:
            ei, ej = self.E[self.type[i], si], self.E[self.type[j], sj]
            a0, b0 = self.x[i, ei[:, 0]], self.x[j, ej[:, 0]]
            Ei, Ej = self.x[i, ei[:, 1]] - a0, self.x[j, ej[:, 1]] - b0
            v = a0 - b0
            c, d, e = _dot(Ei, Ei), _dot(Ej, Ej), _dot(Ei, Ej)
            f = c * d - e * e
            ok = f.abs() > 1e-12
            f = torch.where(ok, f, torch.ones_like(f))
            a, b = _dot(Ei, v), _dot(Ej, v)
            s, t = (e * b - a * d) / f, (c * b - e * a) / f
            ok &= (s > 0) & (s < 1) & (t > 0) & (t < 1)
            at = a0 + Ei * s[:, None]
            n = at - (b0 + Ej * t[:, None])
        else:
            at = self.x[i, si]
            if kind == 0:
                n = at - self.x[j, sj]
                ok = torch.ones_like(si, dtype=torch.bool)
            elif kind == 1:
                e = self.E[self.type[j], sj]
                f0 = self.x[j, e[:, 0]]
                fs, fi = self.x[j, e[:, 1]] - f0, at - f0
                p = _dot(fs, fi) / _dot(fs, fs)
                ok = (p >= -skin) & (p <= 1 + skin) if skin else (p > 0) & (p < 1)
                n = fi - fs * p[:, None]
            else:
                f, m = self.F[self.type[j], sj], self.fs[self.type[j], sj]
                fx = self.x[j[:, None], f]
                last = fx[torch.arange(len(j), device=self.dev), m - 1]
                v1 = fx[:, 1] - fx[:, 0]
                v1 = v1 / torch.sqrt(_dot(v1, v1))[:, None]
                nn = _cross(v1, last - fx[:, 0])
                nn = nn / torch.sqrt(_dot(nn, nn))[:, None]
                h = _dot(nn, at - fx[:, 0])
                nn = torch.where((h < 0)[:, None], -nn, nn)
                n = nn * h.abs()[:, None]
                P, v2 = at - n, _cross(nn, v1)
                o1, o2 = _dot(P, v1), _dot(P, v2)
                odd = torch.zeros_like(o1, dtype=torch.bool)
                for k in range(f.shape[1]):
                    A0 = fx[:, k]
                    B0 = torch.where((k + 1 < m)[:, None], fx[:, (k + 1) % f.shape[1]], fx[:, 0])
                    pa2, pb2 = _dot(A0, v2), _dot(B0, v2)
                    cr = ((pa2 < o2) & (pb2 >= o2)) | ((pb2 < o2) & (pa2 >= o2))
                    den = torch.where(cr, pb2 - pa2, torch.ones_like(pa2))
                    odd ^= cr & (k < m) & (_dot(A0, v1) + (o2 - pa2) / den * (_dot(B0, v1) - _dot(A0, v1)) < o1)
                dn = h.abs() - R
                return odd & (dn <= 0), dn, nn, at - nn * (self.mr + 0.5 * dn)[:, None]
        dist = torch.sqrt(_dot(n, n))
        dn = dist - R
        n = n / dist[:, None]
        ok &= (dn < 0) if kind == 0 and not skin else (dn <= 0)
        return ok, dn, n, at - n * (self.mr + 0.5 * dn)[:, None]

    def contacts(self):
        self.vertices()
        keys, fts, mos = [], [], []
        for kind in range(4):
            sel = self.feat[0] == kind
            _, i, si, j, sj = (x[sel] for x in self.feat)
            c, dn, n, cp = self.detect(kind, i, si, j, sj, 0.0)
            i, si, j, sj, dn, n, cp = i[c], si[c], j[c], sj[c], dn[c], n[c], cp[c]
            key = self.key(torch.full_like(i, kind), i, si, j, sj)
            ft, mo = self.history(key)
            meff = self.m[i] * self.m[j] / (self.m[i] + self.m[j])
            f, ft, mo = self.law(self.p.config, dn, n, cp, ft, mo, meff, self.r[i], self.v[i], self.w[i], self.r[j],
                                 self.v[j], self.w[j])
            self.add(i, f, _cross(cp - self.r[i], f) + mo)
            self.add(j, -f, _cross(cp - self.r[j], -f) - mo)
            keys.append(key)
            fts.append(ft)
            mos.append(mo)
        real = torch.arange(self.V.shape[1], device=self.dev)[None] < self.nv[self.type][:, None]
        i, s = torch.nonzero(real, as_tuple=True)
        for _, index, dv in self.drv:
            self.sub = s
            key, f, ft, mo, cp, k = self.driver(self.p.config_driver, dv, index, i, self.x[i, s],
                                                torch.full_like(self.m[i], self.mr))
            self.add(k, f, _cross(cp - self.r[k], f) + mo)
            keys.append(key)
            fts.append(ft)
            mos.append(mo)
        self.remember(torch.cat(keys), torch.cat(fts), torch.cat(mos))
