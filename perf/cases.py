"""Workloads for timing the DEM step through its public entry points.

Each case is one call pattern of a user's program over a seeded scene:

  steps   a run in memory: `GlobalData.simulate(k)`, then the particle state
          into page-locked arrays (`GlobalData.particles(out=...)`)
  loop    a host loop that owns the state (a coupled solver, a controller):
          one `StateBuffers.step(1)` per pass, state in and out every step
  save    a save interval of the driver: `simulate(k)`, then what a snapshot
          writes, the particle state and the contact records
  init    a body is bonded and takes its first step: `initialize()`,
          `simulate(1)`, particle state
  arena   many independent scenes in one `Arena`: `step(k)`, then every
          scene's state
  sort    `dem_bucket_sort_noalloc` on a caller's own device arrays

The scenes are the ones the repository's benchmark and tests use, made here
from a seed: lattice cubes of bonded spheres (whole, or cracked: a share of
the bonds missing, so that bonds and Hertz-Mindlin contacts lie side by side),
beds of touching columns of polydisperse spheres, and pours of spheres that
do not touch yet.  `exact` steps the same scene with plain torch operations in
float64.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from taichi_dem_julia_port_gb300 import (Arena, DEMConfig, GlobalData, Material, ParticleInput,
                                         Surface, Tables, Wall, _abi)

FIELDS = {"pos": 3, "vel": 3, "omega": 3, "quat": 4, "force": 3, "moment": 3, "wall_shear": 3}
ARENA_FIELDS = ("pos", "vel", "omega", "force")


# ---- the cases ----------------------------------------------------------------

def listed():
    return [
        # the smallest scene in use, one call per step with the state in and
        # out: launches and latency
        dict(name="loop_cube_1000", kind="loop", scene="cube", n=1_000, precision="fp64"),
        # the benchmark's cube in the same host loop
        dict(name="loop_cracked_17576", kind="loop", scene="cracked", n=17_576, precision="fp64"),
        # the smallest scene stepped on the device
        dict(name="steps_cube_1000", kind="steps", scene="cube", n=1_000, precision="fp64",
             steps=50),
        # the benchmark's cube with bonds and Hertz contacts mixed, as after an impact
        dict(name="steps_cracked_17576", kind="steps", scene="cracked", n=17_576,
             precision="fp64", steps=50),
        # a larger body in the reference's precision
        dict(name="steps_cracked_103823", kind="steps", scene="cracked", n=103_823,
             precision="fp64", steps=20),
        # a save interval of an unbonded scene of odd size in FP64
        dict(name="save_bed_30011", kind="save", scene="bed", n=30_011, precision="fp64",
             steps=50),
        # the largest scenes, FP32 forces: a bed with a contact per sphere ...
        dict(name="steps_bed_2000000", kind="steps", scene="bed", n=2_000_000,
             precision="fp32", steps=50),
        # ... and a pour before its spheres meet
        dict(name="steps_pour_2000000", kind="steps", scene="pour", n=2_000_000,
             precision="fp32", steps=100),
        # two materials, two walls and damping (a scene's own tables)
        dict(name="tables_cracked_20011", kind="steps", scene="cracked", n=20_011,
             precision="fp64", steps=50, tables=True),
        # a parameter study: cubes and pours of 500-20,000 spheres stepped together
        dict(name="arena_256", kind="arena", scenes=256, nmin=500, nmax=20_000,
             precision="fp32", steps=50),
        # bonding a large body: the full pair search
        dict(name="init_cube_110592", kind="init", scene="cube", n=110_592, precision="fp64"),
        # the bucket sort on a caller's arrays
        dict(name="sort_1000000", kind="sort", n=1_000_000, buckets=1 << 20),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["loop", "steps", "steps", "steps", "save", "tables", "arena", "init",
                       "sort"])
    if kind == "loop":
        return dict(kind="loop", scene=rng.choice(["cube", "cracked"]), n=_log(rng, 700, 60_000),
                    precision=rng.choice(["fp64", "fp64", "fp32"]))
    if kind == "steps":
        scene = rng.choice(["cube", "cracked", "bed", "pour"])
        precision = rng.choice(["fp64", "fp32"])
        top = 120_000 if scene in ("cube", "cracked") else 1_500_000
        if precision == "fp64" and scene == "bed":
            top = 400_000
        n = _log(rng, 700, top)
        return dict(kind="steps", scene=scene, n=n, precision=precision,
                    steps=20 if n > 60_000 else 50)
    if kind == "save":
        return dict(kind="save", scene=rng.choice(["bed", "cube"]), n=_log(rng, 2_000, 80_000),
                    precision=rng.choice(["fp64", "fp32"]), steps=50)
    if kind == "tables":
        return dict(kind="steps", scene=rng.choice(["cracked", "bed"]), n=_log(rng, 2_000, 60_000),
                    precision="fp64", steps=30, tables=True)
    if kind == "arena":
        return dict(kind="arena", scenes=rng.randint(8, 200), nmin=500,
                    nmax=_log(rng, 2_000, 20_000), precision=rng.choice(["fp64", "fp32"]),
                    steps=rng.randint(20, 40))
    if kind == "init":
        return dict(kind="init", scene=rng.choice(["cube", "bed"]), n=_log(rng, 2_000, 110_000),
                    precision=rng.choice(["fp64", "fp32"]))
    return dict(kind="sort", n=_log(rng, 5_000, 1_000_000),
                buckets=rng.choice([1_024, 50_021, 1 << 20]))


# ---- seeded scenes --------------------------------------------------------------

def _config(**kw):
    c = dict(particle_contact_radius_multiplier=1.1, neighboring_search_safety_factor=1.01,
             particle_elastic_modulus=1e8, particle_poisson_ratio=0.3,
             wall_normal=[0.0, 0.0, -1.0], wall_distance=0.0, wall_density=7800.0,
             wall_elastic_modulus=2e11, wall_poisson_ratio=0.25, bond_radius_ratio=0.5,
             bond_elastic_modulus=1e8, bond_poisson_ratio=0.2, bond_compressive_strength=3e8,
             bond_tensile_strength=1e6, bond_shear_strength=1e6, pp_coefficient_friction=0.5,
             pp_coefficient_restitution=0.9, pw_coefficient_friction=0.35,
             pw_coefficient_restitution=0.7, max_coordinate_number=16, tolerance=1e-12,
             gravity=[0.0, 0.0, -9.81], global_damping=0.0, dt=1e-6, target_time=1.0,
             saving_interval_time=1e-3)
    c.update(kw)
    return c


def _cube(rng, n, cracked, speed=0.5, friction=0.5, E=1e8):
    """A simple-cubic lattice of n spheres of about 10 mm (the last layer of a
    ragged n is not full) that has just met the plane below it, with small
    random velocities and spins.  `bonds`: the face neighbours' bonds, of
    which a cracked body has lost one in five."""
    side = max(1, math.ceil(n ** (1.0 / 3.0) - 1e-9))
    k = np.arange(n)
    ijk = np.stack([k % side, (k // side) % side, k // (side * side)], axis=1)
    spacing = 0.02
    r = 0.01 * (1.0 + rng.uniform(-0.01, 0.01, n))
    pos = ijk * spacing + rng.uniform(-1e-6, 1e-6, (n, 3))
    vel = rng.normal(0.0, 0.02, (n, 3))
    vel[:, 2] -= speed
    omega = rng.normal(0.0, 2.0, (n, 3))
    wall_z = float(np.min(pos[:, 2] - r)) + 2e-5
    lo, hi = pos.min(axis=0) - 0.1, pos.max(axis=0) + 0.1
    bonds = []
    for axis, stride in ((0, 1), (1, side), (2, side * side)):
        a = k[(ijk[:, axis] < side - 1) & (k + stride < n)]
        bonds.append(np.stack([a, a + stride], axis=1))
    bonds = np.concatenate(bonds)
    if cracked:
        bonds = bonds[rng.random(len(bonds)) < 0.8]
    bonds = bonds[np.lexsort((bonds[:, 1], bonds[:, 0]))]
    cfg = _config(domain_min=lo.tolist(), domain_max=hi.tolist(), wall_distance=-wall_z,
                  pp_coefficient_friction=friction, particle_elastic_modulus=E)
    return dict(cfg=cfg, r=r, pos=pos, vel=vel, omega=omega, bonds=bonds)


def _radii(rng, n):
    return np.clip(1e-3 * np.exp(0.25 * rng.standard_normal(n)), 0.5e-3, 2e-3)


def _grains_config(pos, **kw):
    return _config(domain_min=[-0.05] * 3, domain_max=(pos.max(axis=0) + 0.05).tolist(),
                   pp_coefficient_friction=kw.pop("friction", 0.4), dt=2e-7, **kw)


def _bed(rng, n):
    """Columns of touching spheres (log-normal radii of 0.5-2 mm) on a square
    grid, each sphere resting on the one below and the first on the plane,
    about 1.8 cube roots of n high, in slow random motion."""
    r = _radii(rng, n)
    levels = max(1, round(1.8 * n ** (1.0 / 3.0)))
    nx = max(1, math.ceil(math.sqrt(n / levels)))
    ncol = nx * nx
    off_max, pitch = 0.125e-3, 4.004e-3 + 0.25e-3
    col = np.arange(n) % ncol
    pos = np.empty((n, 3))
    pos[:, :2] = (np.stack([col % nx, col // nx], axis=1) + 0.5) * pitch
    pos[:, :2] += rng.uniform(-1.0, 1.0, (n, 2)) * off_max
    z = r * (1.0 - 1e-3)
    for s in range(ncol, n, ncol):
        cur = slice(s, min(s + ncol, n))
        low = slice(s - ncol, s - ncol + (cur.stop - cur.start))
        d = (r[cur] + r[low]) * (1.0 - 1e-3)
        z[cur] = z[low] + np.sqrt(d * d - np.sum((pos[cur, :2] - pos[low, :2]) ** 2, axis=1))
    pos[:, 2] = z
    return dict(cfg=_grains_config(pos), r=r, pos=pos, vel=rng.normal(0.0, 0.01, (n, 3)),
                omega=rng.normal(0.0, 5.0, (n, 3)), bonds=None)


def _pour(rng, n, friction=0.4, E=1e8):
    """Spheres at rest above the plane: n sites, two in three, of a lattice of
    spacing 4 mm, each sphere somewhere inside its own site."""
    r = _radii(rng, n)
    h = 4.004e-3
    s = max(1, math.ceil((n / (0.68 * 3)) ** (1.0 / 3.0)))
    site = np.sort(rng.permutation(3 * s ** 3)[:n])
    ijk = np.stack([site % s, (site // s) % s, site // (s * s)], axis=1)
    pos = (ijk + 0.5) * h + rng.uniform(-1.0, 1.0, (n, 3)) * (0.5 * h - r)[:, None]
    return dict(cfg=_grains_config(pos, friction=friction, particle_elastic_modulus=E), r=r,
                pos=pos, vel=np.zeros((n, 3)), omega=np.zeros((n, 3)), bonds=None)


def _scene(case, seed):
    rng = np.random.default_rng(seed)
    n = case["n"]
    if case["scene"] == "bed":
        sc = _bed(rng, n)
    elif case["scene"] == "pour":
        sc = _pour(rng, n)
    else:
        sc = _cube(rng, n, case["scene"] == "cracked")
    if case.get("tables"):
        sc["cfg"]["global_damping"] = 0.05
        sc["material"] = (rng.random(n) < 0.4).astype(np.int32)
        x0 = float(np.min(sc["pos"][:, 0] - sc["r"])) + 1e-5
        sc["tables"] = _tables(sc["cfg"], x0)
    return sc


def _tables(cfg, x0):
    """Two particle materials and a wall material; the scene's plane and a
    side wall at x = x0."""
    mats = [(2500.0, cfg["particle_elastic_modulus"], 0.3), (2500.0, 6e7, 0.25),
            (7800.0, 2e11, 0.25)]

    def surface(mu, e, ratio, strength):
        return dict(mu=mu, e=e, ratio=ratio, E=cfg["bond_elastic_modulus"], nu=0.2,
                    sc=3e8, st=strength, ss=strength)
    s00, s11, s01 = (surface(0.5, 0.9, 0.5, 1e6), surface(0.3, 0.8, 0.45, 2e6),
                     surface(0.4, 0.85, 0.4, 1.5e6))
    w0, w1 = surface(0.35, 0.7, 0.5, 1e6), surface(0.2, 0.6, 0.5, 1e6)
    return dict(materials=mats, surfaces=[[s00, s01, w0], [s01, s11, w1], [w0, w1, w0]],
                walls=[([0.0, 0.0, -1.0], cfg["wall_distance"], 2), ([1.0, 0.0, 0.0], x0, 2)])


def _arena_scenes(case, seed):
    """Cubes about to hit their plane at 10 m/s and pours in turn, sizes
    log-uniform (the case's own), each with its own stiffness and friction."""
    m = case["scenes"]
    sizes = np.exp(np.random.default_rng(m).uniform(math.log(case["nmin"]),
                                                    math.log(case["nmax"]), m))
    rng = np.random.default_rng(seed)
    E, mu = rng.uniform(1e7, 1e9, m), rng.uniform(0.2, 0.8, m)
    out = []
    for k in range(m):
        n = int(round(sizes[k]))
        if k % 2 == 0:
            sc = _cube(rng, n, False, speed=10.0, friction=float(mu[k]), E=float(E[k]))
            sc["cfg"]["wall_distance"] += 1.2e-4  # the plane 0.1 mm below the cube
        else:
            sc = _pour(rng, n, friction=float(mu[k]), E=float(E[k]))
        sc["omega"] = np.zeros_like(sc["omega"])
        out.append(sc)
    return out


def _mass(sc):
    return 2500.0 * (4.0 / 3.0 * math.pi * sc["r"] ** 3)


# ---- a user's program -----------------------------------------------------------

def _pinned(n, fields):
    return {f: torch.empty((n, FIELDS[f]), dtype=torch.float64, pin_memory=True).numpy()
            for f in fields}


def _handle(case, sc):
    cfg = DEMConfig.from_dict(sc["cfg"])
    p = ParticleInput.from_arrays(sc["r"], sc["pos"], sc["vel"], 2500.0)
    tables = None
    if "tables" in sc:
        t = sc["tables"]
        tables = Tables(
            materials=[Material(*m) for m in t["materials"]],
            surfaces=[[Surface(s["mu"], s["e"], 0.0, s["ratio"], s["E"], s["nu"], s["sc"],
                               s["st"], s["ss"]) for s in row] for row in t["surfaces"]],
            walls=[Wall(*w) for w in t["walls"]], grain_material=sc["material"])
    g = GlobalData(cfg, p, precision=case["precision"], tables=tables)
    g.set_particles(omega=sc["omega"])
    if sc["bonds"] is not None and case["kind"] != "init":
        g.set_contacts(dict(i=sc["bonds"][:, 0], j=sc["bonds"][:, 1],
                            bonded=np.ones(len(sc["bonds"]))))
    return g


class _View(np.ndarray):
    """An array that keeps the owner of its memory alive."""


def _kept(a, owner):
    v = a.view(_View)
    v.owner = owner
    return v


def prepare(case, seed):
    kind = case["kind"]
    if kind == "sort":
        pos, cell, lo = _sort_inputs(case, seed)
        n = case["n"]
        return dict(case=case, lib=_abi.load_library(), pos=[torch.tensor(p, device="cuda")
                                                              for p in pos],
                    lo=(C.c_double * 3)(*lo), cell=cell,
                    bucket=torch.zeros(n, dtype=torch.int32, device="cuda"),
                    order=torch.zeros(n, dtype=torch.int32, device="cuda"))
    if kind == "arena":
        scenes = _arena_scenes(case, seed)
        total = sum(len(s["r"]) for s in scenes)
        arena = Arena(total, max_scenes=len(scenes), precision=case["precision"])
        flat, views, at = _pinned(total, ARENA_FIELDS), [], 0
        for sc in scenes:
            n = len(sc["r"])
            k = arena.add(DEMConfig.from_dict(sc["cfg"]),
                          ParticleInput.from_arrays(sc["r"], sc["pos"], sc["vel"], 2500.0),
                          init_bonds=sc["bonds"] is not None)
            views.append((k, {f: a[at:at + n] for f, a in flat.items()}))
            at += n
        return dict(case=case, arena=arena, out=flat, views=views)
    g = _handle(case, _scene(case, seed))
    if kind == "loop":
        buf = g.state_buffers(forces=True)
        return dict(case=case, buf=buf, out={f: _kept(a, buf) for f, a in buf.arrays.items()})
    if kind == "save":
        return dict(case=case, g=g)
    return dict(case=case, g=g, out=_pinned(case["n"], FIELDS))


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "loop":
        state["buf"].step(1)
        return state["out"]
    if kind == "steps":
        state["g"].simulate(case["steps"])
        return state["g"].particles(out=state["out"])
    if kind == "save":
        state["g"].simulate(case["steps"])
        p = state["g"].particles(forces=False)
        c = state["g"].io_contacts()
        return dict(particles=p, i=c["i"], j=c["j"], bonded=c["bonded"], point=c["point"],
                    force=c["force"])
    if kind == "init":
        state["g"].initialize()
        state["g"].simulate(1)
        return state["g"].particles(out=state["out"])
    if kind == "arena":
        state["arena"].step(case["steps"])
        for k, views in state["views"]:
            state["arena"].particles(k, out=views)
        return state["out"]
    x, y, z = state["pos"]
    _abi.check(state["lib"], state["lib"].dem_bucket_sort_noalloc(
        x.data_ptr(), y.data_ptr(), z.data_ptr(), case["n"], state["lo"], state["cell"],
        case["buckets"], state["bucket"].data_ptr(), state["order"].data_ptr(),
        torch.cuda.current_stream().cuda_stream), "dem_bucket_sort_noalloc")
    return state["bucket"], state["order"]


def _sort_inputs(case, seed):
    """A mixed bed of n spheres of about 1 mm: positions in no spatial order."""
    rng = np.random.default_rng(seed)
    n = case["n"]
    side = (n * 1.2e-8) ** (1.0 / 3.0)
    return rng.uniform(0.0, side, (3, n)), 4 * 2e-3 * 1.1 * 1.01, [-0.05, -0.05, -0.05]


# ---- what a pass cannot do without ------------------------------------------------

def _contacts(kind, n):
    """About how many bonds and Hertz contacts a scene holds."""
    if kind == "pour":
        return 0, 0
    if kind == "bed":
        return 0, n
    faces = 3 * (n - n ** (2.0 / 3.0))
    return (faces, 0) if kind == "cube" else (0.8 * faces, 0.1 * faces)


def work(case):
    if case["kind"] == "sort":
        return {"bytes": case["n"] * (24 + 8), "flops": case["n"] * 20}
    steps = case.get("steps", 1)
    if case["kind"] == "arena":
        a, b = case["nmin"], case["nmax"]
        mean = (b - a) / math.log(b / a)
        parts = [("cube", mean, case["scenes"] / 2), ("pour", mean, case["scenes"] / 2)]
    else:
        parts = [(case["scene"], case["n"], 1)]
    out = {"bytes": 0.0, "flops": 0.0}
    for scene, n, times in parts:
        bonds, hertz = _contacts(scene, n)
        if case["kind"] == "init":
            bonds, hertz = bonds + hertz, 0
        # per step: position, velocity, spin and orientation read and
        # written, mass, radius and inertia read, the force and moment
        # written; per bond its ids, force and torques read and written and
        # its point written; per Hertz contact its ids, shear read and
        # written, its point and force written
        step = n * (2 * 13 * 8 + 3 * 8 + 6 * 8) + bonds * (8 + 144 + 24) + hertz * (8 + 48 + 48)
        out["bytes"] += times * (steps * step + n * 22 * 8)
        out["flops"] += times * steps * (n * 90 + bonds * 220 + hertz * 260)
    return out


# ---- the same in 64 bits with plain torch -----------------------------------------

def exact(case, seed):
    if case["kind"] == "sort":
        return _exact_sort(case, seed)
    steps = case.get("steps", 1)
    if case["kind"] == "arena":
        p = _Exact(_arena_scenes(case, seed), bond_now=True).step(steps).particles()
        return {f: p[f] for f in ARENA_FIELDS}
    e = _Exact([_scene(case, seed)], bond_now=case["kind"] == "init").step(steps)
    p = e.particles()
    if case["kind"] == "save":
        c = e.contacts()
        return dict(particles={f: p[f] for f in FIELDS if f not in ("force", "moment")}, **c)
    return p


def _exact_sort(case, seed):
    pos, cell, lo = _sort_inputs(case, seed)
    morton = np.zeros(case["n"], np.int64)
    for c in range(3):
        k = np.ceil((pos[c] - lo[c]) / cell).astype(np.int64) - 1
        for bit in range(10):
            morton |= ((k >> bit) & 1) << (3 * bit + c)
    bucket = (morton + 1) % case["buckets"]
    return (bucket + 1).astype(np.int32), np.argsort(bucket, kind="stable").astype(np.int32)


def _hertz_constants(m1, m2, e):
    (_, E1, n1), (_, E2, n2) = m1, m2
    Y = 1.0 / ((1 - n1 * n1) / E1 + (1 - n2 * n2) / E2)
    G = 1.0 / (2 * (2 - n1) * (1 + n1) / E1 + 2 * (2 - n2) * (1 + n2) / E2)
    beta = math.log(e) / math.hypot(math.log(e), math.pi)
    return Y, G, beta


def _material_tables(sc):
    """(materials, surfaces, walls, each sphere's material) of a scene."""
    c = sc["cfg"]
    if "tables" in sc:
        tb = sc["tables"]
        return tb["materials"], tb["surfaces"], tb["walls"], sc["material"]
    mats = [(2500.0, c["particle_elastic_modulus"], c["particle_poisson_ratio"]),
            (c["wall_density"], c["wall_elastic_modulus"], c["wall_poisson_ratio"])]
    pp = dict(mu=c["pp_coefficient_friction"], e=c["pp_coefficient_restitution"],
              ratio=c["bond_radius_ratio"], E=c["bond_elastic_modulus"],
              nu=c["bond_poisson_ratio"], sc=c["bond_compressive_strength"],
              st=c["bond_tensile_strength"], ss=c["bond_shear_strength"])
    pw = dict(pp, mu=c["pw_coefficient_friction"], e=c["pw_coefficient_restitution"])
    return (mats, [[pp, pw], [pw, pw]], [(c["wall_normal"], c["wall_distance"], 1)],
            np.zeros(len(sc["r"]), np.int32))


class _Exact:
    """Scenes of the same shape of tables, side by side, stepped with torch
    operations in float64."""

    def __init__(self, scenes, bond_now):
        dev = "cuda" if torch.cuda.is_available() else "cpu"

        def t(a):
            return torch.as_tensor(np.asarray(a), dtype=torch.float64, device=dev)

        def ints(a):
            return torch.as_tensor(np.asarray(a, np.int64), device=dev)

        def cat(f):
            return t(np.concatenate([f(sc) for sc in scenes]))
        sizes = [len(sc["r"]) for sc in scenes]
        n = sum(sizes)
        self.scene = ints(np.repeat(np.arange(len(scenes)), sizes))
        c = scenes[0]["cfg"]
        self.tol, self.damping, self.grav = c["tolerance"], c["global_damping"], t(c["gravity"])
        self.dt = cat(lambda sc: np.full(len(sc["r"]), sc["cfg"]["dt"]))[:, None]
        self.x, self.v = cat(lambda sc: sc["pos"]), cat(lambda sc: sc["vel"])
        self.w, self.m = cat(lambda sc: sc["omega"]), cat(_mass)
        self.r = cat(lambda sc: np.cbrt(_mass(sc) / 2500.0 / (4.0 / 3.0 * math.pi)))
        self.q = torch.zeros((n, 4), dtype=torch.float64, device=dev)
        self.q[:, 0] = 1.0
        self.I = 0.4 * self.m * self.r ** 2
        tabs = [_material_tables(sc) for sc in scenes]
        np_ = len(tabs[0][0]) - 1  # the last material is the walls'
        mid = ints(np.concatenate([tb[3] for tb in tabs]))
        hz = [[[_hertz_constants(mats[a], mats[b], surf[a][b]["e"]) for b in range(np_ + 1)]
               for a in range(np_ + 1)] for mats, surf, _, _ in tabs]
        consts = ("Y", "G", "beta")
        self.walls = []
        for k in range(len(tabs[0][2])):
            normal, wm = tabs[0][2][k][0], tabs[0][2][k][2]
            per = {q: t([[z[a][wm][u] for a in range(np_)] for z in hz])[self.scene, mid]
                   for u, q in enumerate(consts)}
            per["mu"] = t([[tb[1][a][wm]["mu"] for a in range(np_)] for tb in tabs])[self.scene, mid]
            self.walls.append((t(normal), t([tb[2][k][1] for tb in tabs])[self.scene], per))
        self.ws = [torch.zeros((n, 3), dtype=torch.float64, device=dev) for _ in self.walls]
        self._pairs()
        i, j = self.i, self.j
        at = (self.scene[i], mid[i], mid[j])
        self.pc = {q: t([[[z[a][b][u] for b in range(np_)] for a in range(np_)] for z in hz])[at]
                   for u, q in enumerate(consts)}
        for q in ("mu", "ratio", "E", "nu", "sc", "st", "ss"):
            self.pc[q] = t([[[tb[1][a][b][q] for b in range(np_)] for a in range(np_)]
                            for tb in tabs])[at]
        M = len(i)
        self.bond = torch.zeros(M, dtype=torch.bool, device=dev)
        has = torch.as_tensor([sc["bonds"] is not None or len(scenes) == 1 for sc in scenes],
                              device=dev)
        if bond_now:
            r0 = self.r * c["particle_contact_radius_multiplier"]
            self.bond = ((self.x[i] - self.x[j]).norm(dim=1) < r0[i] + r0[j]) & has[self.scene[i]]
        elif scenes[0]["bonds"] is not None:
            b = ints(scenes[0]["bonds"])
            key = b[:, 0] * n + b[:, 1]
            at = torch.searchsorted(i * n + j, key)
            assert bool((i[at] * n + j[at] == key).all())
            self.bond[at] = True
        self.active = self.bond.clone()
        self.F, self.ti, self.tj, self.s, self.k = (
            torch.zeros((M, 3), dtype=torch.float64, device=dev) for _ in range(5))
        self.force = self.moment = None

    def _pairs(self):
        """Pairs i < j near enough to touch or bond at any time of the run, in order."""
        x, r = self.x, self.r
        n = len(r)
        big = torch.zeros(int(self.scene.max()) + 1, dtype=r.dtype, device=r.device)
        big.scatter_reduce_(0, self.scene, r, "amax")
        reach = 1.15 * big[self.scene]  # bonds join within 1.1 (ri + rj)
        cell = torch.floor((x - x.min(dim=0).values) / (2 * reach)[:, None]).long() + 1
        dims = (cell.max(dim=0).values + 2).tolist()
        key = ((self.scene * dims[2] + cell[:, 2]) * dims[1] + cell[:, 1]) * dims[0] + cell[:, 0]
        key, order = torch.sort(key)
        I, J = [], []
        for dz in (-1, 0, 1):
            for dy in (-1, 0, 1):
                for dx in (-1, 0, 1):
                    want = key + (dz * dims[1] + dy) * dims[0] + dx
                    a = torch.searchsorted(key, want)
                    b = torch.searchsorted(key, want, right=True)
                    for u in range(int((b - a).max())):
                        ok = a + u < b
                        i, j = order[ok], order[(a + u)[ok]]
                        near = (j > i)
                        i, j = i[near], j[near]
                        near = (x[i] - x[j]).norm(dim=1) < 1.15 * (r[i] + r[j])
                        I.append(i[near])
                        J.append(j[near])
        i, j = torch.cat(I), torch.cat(J)
        order = torch.argsort(i * n + j)
        self.i, self.j = i[order], j[order]

    @staticmethod
    def _frame(a, tol):
        """Rows of the rotation that takes a onto the x axis."""
        s2 = a[:, 1] ** 2 + a[:, 2] ** 2
        flat = s2 < tol * tol
        f = torch.where(flat, torch.zeros_like(s2),
                        (1.0 - a[:, 0]) / torch.where(flat, torch.ones_like(s2), s2))
        sg = torch.where(a[:, 0] > 0, 1.0, -1.0).to(a)
        z, one = torch.zeros_like(s2), torch.ones_like(s2)
        a1, a2, a3 = (torch.where(flat, sg, a[:, 0]), torch.where(flat, z, a[:, 1]),
                      torch.where(flat, z, a[:, 2]))
        return torch.stack([
            torch.stack([a1, a2, a3], 1),
            torch.stack([-a2, one - a2 * a2 * f, -a2 * a3 * f], 1),
            torch.stack([-a3, -a2 * a3 * f, torch.where(flat, sg, one - a3 * a3 * f)], 1)], 1)

    @staticmethod
    def _mv(R, v):
        return (R * v[:, None, :]).sum(dim=2)

    @staticmethod
    def _friction(Ft, s, kt, gt, vc, mu, F1):
        """The tangential force and the shear history of a sliding or sticking contact."""
        nFt = Ft.norm(dim=1)
        slide = nFt >= mu * F1
        ratio = torch.where(slide, mu * F1 / torch.where(slide, nFt, torch.ones_like(nFt)),
                            torch.zeros_like(nFt))
        out = torch.where(slide[:, None], ratio[:, None] * Ft, Ft - gt[:, None] * vc)
        new = torch.where(slide[:, None], out / kt[:, None], s)
        return out, torch.cat([s[:, :1], new[:, 1:]], dim=1)

    def step(self, steps):
        for _ in range(steps):
            self._step()
        return self

    def _step(self):
        dt, tol = self.dt, self.tol
        x, v, w, r, i, j = self.x, self.v, self.w, self.r, self.i, self.j
        force, moment = torch.zeros_like(x), torch.zeros_like(x)
        d = x[j] - x[i]
        touch = d.norm(dim=1) < r[i] + r[j]
        new = touch & ~self.active
        self.s[new] = 0.0
        self.active = self.bond | touch

        def add(i, j, fi, mi, mj):
            force.index_add_(0, i, fi)
            force.index_add_(0, j, -fi)
            moment.index_add_(0, i, mi)
            moment.index_add_(0, j, mj)

        b = torch.nonzero(self.bond)[:, 0]
        if len(b):
            I, J = i[b], j[b]
            L = d[b].norm(dim=1)
            R = self._frame(d[b] / L[:, None], tol)
            D = self._mv(R, v[I] - v[J]) * dt[I]
            ta, tb = self._mv(R, w[I]) * dt[I], self._mv(R, w[J]) * dt[I]
            k = {q: a[b] for q, a in self.pc.items()}
            rb = k["ratio"] * torch.minimum(r[I], r[J])
            A, S = math.pi * rb ** 2, math.pi / 4 * rb ** 4
            phi = 20.0 / 3.0 * rb ** 2 / L ** 2 * (1 + k["nu"])
            EI = k["E"] * S
            k1 = k["E"] * A / L
            k2 = 12 * EI / L ** 3 / (1 + phi)
            k3 = 6 * EI / L ** 2 / (1 + phi)
            k4 = EI / L / (1 + k["nu"])
            k5 = EI * (4 + phi) / L / (1 + phi)
            k6 = EI * (2 - phi) / L / (1 + phi)
            F = self.F[b] + torch.stack([
                k1 * D[:, 0], k2 * D[:, 1] + k3 * (ta + tb)[:, 2],
                k2 * D[:, 2] - k3 * (ta + tb)[:, 1]], 1)
            ti = self.ti[b] + torch.stack([
                k4 * (ta - tb)[:, 0], -k3 * D[:, 2] + k5 * ta[:, 1] + k6 * tb[:, 1],
                k3 * D[:, 1] + k5 * ta[:, 2] + k6 * tb[:, 2]], 1)
            tj = self.tj[b] + torch.stack([
                k4 * (tb - ta)[:, 0], -k3 * D[:, 2] + k6 * ta[:, 1] + k5 * tb[:, 1],
                k3 * D[:, 1] + k6 * ta[:, 2] + k5 * tb[:, 2]], 1)
            bi = rb / S * torch.hypot(ti[:, 1], ti[:, 2])
            bj = rb / S * torch.hypot(tj[:, 1], tj[:, 2])
            fa = -F[:, 0] / A
            breaks = ((-torch.minimum(fa - bi, fa - bj) >= k["sc"])
                      | (torch.maximum(fa - bi, fa - bj) >= k["st"])
                      | (ti[:, 0].abs() * rb / 2 / S
                         + 4.0 / 3.0 / A * torch.hypot(F[:, 1], F[:, 2]) >= k["ss"]))
            self.F[b], self.ti[b], self.tj[b] = F, ti, tj
            self.k[b] = 0.5 * (x[I] + x[J])
            ok = ~breaks
            Rt = R[ok].transpose(1, 2)
            add(I[ok], J[ok], self._mv(Rt, -F[ok]), self._mv(Rt, -ti[ok]), self._mv(Rt, -tj[ok]))
            gone = b[breaks]

        h = torch.nonzero(self.active & ~self.bond)[:, 0]
        if len(h):
            I, J = i[h], j[h]
            L = d[h].norm(dim=1)
            a = d[h] / L[:, None]
            R = self._frame(a, tol)
            gap = L - r[I] - r[J]
            ki = a * (r[I] - gap.abs())[:, None]
            kj = ki - d[h]
            vc = self._mv(R, v[J] - v[I] + torch.linalg.cross(w[J], kj)
                          - torch.linalg.cross(w[I], ki))
            k = {q: t[h] for q, t in self.pc.items()}
            Rs = r[I] * r[J] / (r[I] + r[J])
            ms = self.m[I] * self.m[J] / (self.m[I] + self.m[J])
            F, self.s[h] = self._hertz(k, Rs, ms, gap, vc, self.s[h], dt[I])
            self.F[h] = F
            self.k[h] = x[I] + ki
            fi = self._mv(R.transpose(1, 2), -F)
            add(I, J, fi, torch.linalg.cross(ki, fi), torch.linalg.cross(kj, -fi))
        if len(b):  # bonds that broke: no contact until the next step looks
            self.bond[gone] = False
            self.active[gone] = False

        for wall, (normal, dist, k) in enumerate(self.walls):
            L = (x * normal).sum(dim=1) - dist
            on = torch.nonzero(L.abs() < r)[:, 0]
            s = torch.zeros_like(self.ws[wall])
            if len(on):
                Lo = L[on]
                gap = Lo.abs() - r[on]
                ki = -torch.sign(Lo)[:, None] * (Lo.abs() + gap.abs() / 2)[:, None] * normal
                R = self._frame(normal.expand(len(on), 3), tol)
                vc = -self._mv(R, torch.linalg.cross(w[on], ki) + v[on])
                F, s[on] = self._hertz({q: t[on] for q, t in k.items()}, r[on], self.m[on], gap,
                                       vc, self.ws[wall][on], dt[on])
                f = self._mv(R.transpose(1, 2), -F)
                force[on] += f
                moment[on] += torch.linalg.cross(ki, f)
            self.ws[wall] = s

        force = force + self.m[:, None] * self.grav
        if self.damping:
            force = force - self.damping * force.abs() * torch.sign(v)
            moment = moment - self.damping * moment.abs() * torch.sign(w)
        acc = force / self.m[:, None]
        self.x = x + v * dt + 0.5 * acc * dt * dt
        self.v = v + acc * dt
        q, (q0, q1, q2, q3) = self.q, self.q.unbind(dim=1)
        h0, h1, h2 = (0.5 * w).unbind(dim=1)
        q = q + torch.stack([-q1 * h0 - q2 * h1 - q3 * h2, q0 * h0 + q2 * h2 - q3 * h1,
                             q0 * h1 + q1 * h2 + q3 * h0, q0 * h2 + q1 * h1 - q2 * h0], 1)
        self.q = q / q.norm(dim=1, keepdim=True)
        self.w = w + moment / self.I[:, None] * dt
        self.force, self.moment = force, moment

    def _hertz(self, k, Rs, ms, gap, vc, s, dt):
        """Hertz-Mindlin force in the contact frame and the new shear history."""
        sq = torch.sqrt(Rs * gap.abs())
        kn, kt = 4.0 / 3.0 * k["Y"] * sq, 8.0 * k["G"] * sq
        gn = -2 * k["beta"] * torch.sqrt(5.0 / 6.0 * 2 * k["Y"] * sq * ms)
        gt = -2 * k["beta"] * torch.sqrt(5.0 / 6.0 * kt * ms)
        z = torch.zeros_like(gap)
        s = s + torch.stack([z, vc[:, 1], vc[:, 2]], 1) * dt
        F1 = -kn * gap - gn * vc[:, 0]
        Ft, s = self._friction(-kt[:, None] * s, s, kt, gt, vc, k["mu"], F1)
        return torch.cat([F1[:, None], Ft[:, 1:]], 1), s

    def particles(self):
        got = dict(pos=self.x, vel=self.v, omega=self.w, quat=self.q, force=self.force,
                   moment=self.moment, wall_shear=self.ws[0])
        return {f: a.cpu().numpy() for f, a in got.items()}

    def contacts(self):
        a = torch.nonzero(self.active)[:, 0]
        got = dict(i=self.i[a].int(), j=self.j[a].int(), bonded=self.bond[a].int(),
                   point=self.k[a], force=self.F[a])
        return {f: t.cpu().numpy() for f, t in got.items()}
