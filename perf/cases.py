"""What users of this framework have it do, as cases that can be timed: whole FDTD runs, stepped
sessions, batches of grids, flux gradients, far fields and mesh rasterisation, each through its
public entry point, from the smallest calls to the largest.

`listed()` names the cases, `draw(rng)` makes more of the same ranges, `prepare(case, seed)` makes a
case's inputs and the handles a program keeps, `run(state)` is one pass, `work(case)` the bytes and
operations a pass cannot do without, and `exact(case, seed)` what a pass returns in 64 bits, from
plain torch on the same inputs.
"""
import math

import numpy as np
import torch

from fieldgrid_b200 import fdtd, raster
from fieldgrid_b200.gpu import Gpu
from fieldgrid_b200.grid import Grid

C0 = 299_792_458.0
EPS0 = 8.854_187_812_8e-12
MU0 = 1.256_637_062_12e-6
ETA0 = 376.730_313_668
DX = 1e-3

#: Steps a session or a batch of grids is made for; stepping on beyond them is allowed.
SESSION_STEPS = 2000


def listed():
    return [
        # An empty closed box on a graded axis, stepped by the separate H and E kernels (the default
        # of Extras): the known-answer resonator run, a few thousand nodes, all launches and latency.
        dict(name="run cavity 29x19x14", kind="run", nx=28, ny=18, nz=13, pml=0, steps=2000, fused=False, model="cavity",
             ports=1, freqs=0, keep=True),
        # The plain FDTD run of the parity tests: a dielectric box, a point source, four probes, 1000
        # steps, the final fields read back. One design iteration of a small model.
        dict(name="run box 64", kind="run", nx=64, ny=64, nz=64, pml=8, steps=1000, fused=True, model="box", ports=5,
             freqs=0, keep=True),
        # An uneven, odd-sized lossy and dispersive scene with a plane DFT, by the separate kernels:
        # what a caller of run() with default options gets on a middling model.
        dict(name="run separate 97x131x203", kind="run", nx=97, ny=131, nz=203, pml=10, steps=300, fused=False,
             model="spheres", ports=2, freqs=3, keep=True),
        # One grid of the batched workload's range run on its own with the fused step.
        dict(name="run spheres 160x120x88", kind="run", nx=160, ny=120, nz=88, pml=8, steps=600, fused=True,
             model="spheres", ports=1, freqs=0, keep=True),
        # The antenna run: a PEC patch on a substrate, the near-to-far-field box at three frequencies.
        dict(name="run patch 256x256x192", kind="run", nx=256, ny=256, nz=192, pml=12, steps=600, fused=True,
             model="patch", ports=1, freqs=3, keep=False),
        # The throughput configuration: random spheres in 512^3 cells, a session stepped by its program.
        dict(name="session spheres 512", kind="session", nx=512, ny=512, nz=512, pml=10, steps=20),
        # Two dozen independent grids of uneven sizes stepped together (a parameter study).
        dict(name="batch 24 grids", kind="batch", count=24, lo=48, hi=160, pml=8, steps=50),
        # One gradient of the flux objective, 16,384 design voxels, with checkpoints 64 steps apart.
        dict(name="flux 160x160x96", kind="flux", nx=160, ny=160, nz=96, pml=8, dx=32, dy=32, dz=8, steps=640,
             checkpoints=10, debye=False),
        # Gradients of several small designs at once, a Debye slab beside each design.
        dict(name="flux batch 8 grids", kind="fluxbatch", count=8, lo=48, hi=96, pml=8, design=16, steps=300,
             checkpoints=6),
        # The far-field pattern of the antenna run's box on the 5-degree grid of directions.
        dict(name="far pattern 5 deg", kind="far", nx=226, ny=226, nz=162, dirs=2664),
        # One cut through the pattern of a small antenna.
        dict(name="far cut 73", kind="far", nx=36, ny=30, nz=24, dirs=73),
        # A closed mesh onto the grid of a solve: the cells it fills, the edges inside it and the
        # edges its surface passes through (dielectric and metal parts of an antenna model).
        dict(name="raster torus 12k", kind="raster", nx=160, ny=128, nz=96, rings=96, sides=64),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "session", "batch", "flux", "fluxbatch", "far", "raster"])
    if kind == "run":
        model = rng.choice(["box", "spheres", "spheres", "patch"])
        pml = rng.choice([4, 6, 8, 10, 12])
        lo = max(28, 2 * pml + 20)
        nx, ny, nz = (_log_int(rng, lo, 200) for _ in range(3))
        cells = nx * ny * nz
        steps = max(60, min(1200, int(2.4e9 / cells)))
        steps = max(60, steps - rng.randrange(0, 50))
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, pml=pml, steps=steps, fused=rng.random() < 0.7, model=model,
                    ports=1 if model == "patch" else rng.randint(1, 4), freqs=3 if model == "patch" else rng.choice([0, 0, 1, 2]),
                    keep=cells < 3_000_000)
    if kind == "session":
        n = [_log_int(rng, 100, 400) for _ in range(3)]
        return dict(kind=kind, nx=n[0], ny=n[1], nz=n[2], pml=rng.choice([0, 6, 8, 10, 12]), steps=rng.randint(5, 40))
    if kind == "batch":
        lo = rng.choice([40, 48, 56])
        return dict(kind=kind, count=rng.randint(4, 24), lo=lo, hi=lo + 8 * rng.randint(3, 12), pml=rng.choice([6, 8]),
                    steps=rng.randint(20, 60))
    if kind == "flux":
        nx, ny = _log_int(rng, 64, 168), _log_int(rng, 64, 168)
        return dict(kind=kind, nx=nx, ny=ny, nz=_log_int(rng, 64, 100), pml=rng.choice([6, 8, 10]),
                    dx=rng.randint(8, 32), dy=rng.randint(8, 32), dz=rng.randint(4, 10), steps=rng.randint(150, 640),
                    checkpoints=rng.choice([0, 4, 8, 12]), debye=rng.random() < 0.4)
    if kind == "fluxbatch":
        return dict(kind=kind, count=rng.randint(3, 8), lo=48, hi=48 + 8 * rng.randint(1, 6), pml=8,
                    design=rng.randint(8, 16), steps=rng.randint(100, 300), checkpoints=rng.randint(2, 8))
    if kind == "far":
        nx, ny, nz = (_log_int(rng, 20, 226) for _ in range(3))
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, dirs=_log_int(rng, 1, 2664))
    return dict(kind="raster", nx=_log_int(rng, 40, 200), ny=_log_int(rng, 40, 200), nz=_log_int(rng, 40, 200),
                rings=_log_int(rng, 16, 128), sides=_log_int(rng, 12, 96))


# ---- inputs ------------------------------------------------------------------------------------

_gpu_handle = None


def _gpu():
    """The program's one device handle."""
    global _gpu_handle
    if _gpu_handle is None:
        _gpu_handle = Gpu.open()
    return _gpu_handle


def _lines(nx, ny, nz, dx=DX):
    return [np.arange(n + 1) * dx for n in (nx, ny, nz)]


class Scene:
    """One solve's inputs as plain arrays: node lines, cell materials, PEC edges, ports, pulse."""

    def __init__(self, lines, pml, f0=10e9, fc=5e9):
        self.lines, self.pml = lines, pml
        self.n = tuple(len(v) for v in lines)
        self.cells = tuple(v - 1 for v in self.n)
        self.eps = np.ones(self.cells, np.float32)
        self.sigma = np.zeros(self.cells, np.float32)
        self.inf = np.ones(self.cells, np.float32)
        self.debye = np.zeros(self.cells, np.float32)
        self.poles = []
        self.pec = None
        self.ports = []            # (edges of one column along z, resistance)
        self.f0, self.fc = f0, fc
        self.freqs = []
        self.plane_k = None
        self.ntff_inset = None

    def sim(self):
        grid = Grid(*self.lines, self.pml)
        mats = fdtd.Materials(self.eps, self.sigma, self.inf, self.debye)
        ports = [fdtd.PortDef("p%d" % q, [[fdtd.Edge(2, at) for at in col]], r) for q, (col, r) in enumerate(self.ports)]
        return fdtd.Sim.try_new(grid, mats, self.pec, [], ports, [], fdtd.Media(fdtd.Sheets(), fdtd.Debye(self.poles), []))

    def pulse(self):
        return fdtd.Pulse(self.f0, self.fc)


def _point(rng, sc):
    return tuple(int(rng.randint(sc.pml + 2, v - sc.pml - 3)) for v in sc.cells)


def _add_spheres(sc, rng, count, rmin, rmax):
    """Random spheres of eps 1..10, sigma up to 0.05 S/m, a fifth of them one-pole Debye (later ones
    overwrite earlier ones)."""
    sc.poles = [(1.0 / rng.uniform(5e-12, 50e-12), 1.0)]
    for _ in range(count):
        c = [rng.uniform(sc.pml, v - sc.pml) for v in sc.cells]
        r = rng.randint(rmin, rmax + 1)
        er, s = rng.uniform(1.0, 10.0), rng.uniform(0.0, 0.05)
        de = rng.uniform(1.0, 5.0) if rng.uniform() < 0.2 else 0.0
        lo = [max(int(math.floor(v - r)), 0) for v in c]
        hi = [min(int(math.ceil(v + r)) + 1, n) for v, n in zip(c, sc.cells)]
        x, y, z = (np.arange(a, b) + 0.5 - v for a, b, v in zip(lo, hi, c))
        m = x[:, None, None] ** 2 + y[None, :, None] ** 2 + z[None, None, :] ** 2 <= r * r
        box = tuple(slice(a, b) for a, b in zip(lo, hi))
        for arr, v in ((sc.eps, er + de), (sc.inf, er if de else 1.0), (sc.debye, de), (sc.sigma, s)):
            arr[box][m] = v


def _scene_run(case, rng):
    if case["model"] == "cavity":
        # node lines of a 100 x 70 x 50 mm box, the x axis graded from fine to coarse
        w = 1.0 + 0.6 * np.minimum(np.arange(case["nx"]) / 10.0, 1.0)
        x = np.concatenate([[0.0], np.cumsum(w)])
        sc = Scene([0.10 * x / x[-1], 0.07 * np.arange(case["ny"] + 1) / case["ny"],
                    0.05 * np.arange(case["nz"] + 1) / case["nz"]], 0, 3.0e9, 2.5e9)
        sc.ports = [([tuple(int(rng.randint(n // 4, n // 2)) for n in sc.cells)], 1e7)]
        return sc
    dx = 0.25e-3 if case["model"] == "patch" else DX
    sc = Scene(_lines(case["nx"], case["ny"], case["nz"], dx), case["pml"])
    nx, ny, nz = sc.cells
    if case["model"] == "box":
        lo, hi = [3 * n // 8 for n in sc.cells], [5 * n // 8 for n in sc.cells]
        sc.eps[lo[0]:hi[0], lo[1]:hi[1], lo[2]:hi[2]] = rng.uniform(2.0, 6.0)
        sc.ports = [([(nx // 2, ny // 2, nz // 2)], 1e7)]
    elif case["model"] == "spheres":
        small = min(sc.cells)
        _add_spheres(sc, rng, max(4, int(200 * (small / 512.0) ** 2 * 4)), max(2, small // 40), max(4, small // 6))
        sc.ports = [([_point(rng, sc)], 50.0)]
    else:
        kg = sc.pml + max(3, nz // 12)
        g = [int(n * 0.625) for n in (nx, ny)]
        p = [max(4, n // 6) + int(rng.randint(0, 3)) for n in (nx, ny)]
        g0, p0 = [(n - w) // 2 for n, w in zip((nx, ny), g)], [(n - w) // 2 for n, w in zip((nx, ny), p)]
        box = (slice(g0[0], g0[0] + g[0]), slice(g0[1], g0[1] + g[1]))
        sc.eps[box + (slice(kg, kg + 2),)] = rng.uniform(3.0, 5.0)
        sc.sigma[box + (slice(kg, kg + 2),)] = 0.002
        sc.pec = np.zeros((3,) + sc.n, bool)
        sc.pec[:2][(slice(None),) + box + (kg,)] = True
        sc.pec[:2, p0[0]:p0[0] + p[0], p0[1]:p0[1] + p[1], kg + 2] = True
        at = (p0[0] + p[0] // 4, p0[1] + p[1] // 2)
        sc.ports = [([at + (kg,), at + (kg + 1,)], 50.0)]
        sc.ntff_inset = 3
    while len(sc.ports) < case["ports"]:
        sc.ports.append(([_point(rng, sc)], 1e7))
    sc.freqs = [8e9, 10e9, 12e9][:case["freqs"]]
    if sc.freqs and sc.ntff_inset is None:
        sc.plane_k = nz // 2
    return sc


def _scene_session(case, rng):
    sc = Scene(_lines(case["nx"], case["ny"], case["nz"]), case["pml"])
    small = min(sc.cells)
    _add_spheres(sc, rng, max(8, int(200 * small / 512)), 5, max(8, small // 13))
    # the port low in x, so that every index a run stores in f32 stays below 2^24
    at = (min(48, max(sc.pml + 2, sc.cells[0] // 10)), sc.cells[1] // 2, sc.cells[2] // 2)
    # inside a dielectric block, which the first steps' records show
    sc.eps[tuple(slice(v - 6, v + 6) for v in at)] = rng.uniform(2.0, 6.0)
    sc.ports = [([at], 50.0)]
    return sc


def _scenes_batch(case, rng):
    """Grids of lo..hi cells along each axis in steps of 8, spheres and a point source in each. The
    sizes are the case's own (the seed moves the materials and sources)."""
    dims = np.random.RandomState(case["count"] * 1000 + case["lo"])
    out = []
    for _ in range(case["count"]):
        sc = Scene(_lines(*(8 * int(dims.randint(case["lo"] // 8, case["hi"] // 8 + 1)) for _ in range(3))), case["pml"])
        small = min(sc.cells)
        _add_spheres(sc, rng, max(4, int(200 * (small / 512.0) ** 2 * 4)), max(2, small // 40), max(4, small // 6))
        sc.ports = [([_point(rng, sc)], 1e7)]
        out.append(sc)
    return out


def _design(sc, rng, lo, hi):
    box = tuple(slice(a, b) for a, b in zip(lo, hi))
    shape = tuple(b - a for a, b in zip(lo, hi))
    sc.eps[box] = rng.uniform(1.0, 12.0, shape)
    sc.sigma[box] = rng.uniform(0.0, 0.01, shape)


def _debye_slab(sc, x, y, z):
    sc.poles = [(1.0 / 20e-12, 1.0)]
    sc.inf[x, y, z], sc.debye[x, y, z], sc.eps[x, y, z] = 2.0, 3.0, 5.0


def _scene_flux(case, rng):
    """A source below a design block of random voxels, the flux plane above it; with `debye` a slab
    beside the block. Returns the scene, the block and the plane."""
    sc = Scene(_lines(case["nx"], case["ny"], case["nz"]), case["pml"], 10e9, 5e9)
    nx, ny, nz = sc.cells
    dw = (case["dx"], case["dy"], case["dz"])
    ks = sc.pml + max(2, nz // 8)
    kd = ks + max(2, nz // 8)
    kp = min(kd + dw[2] + max(2, nz // 8), nz - sc.pml - 2)
    lo = (nx // 2 - dw[0] // 2, ny // 2 - dw[1] // 2, kd)
    hi = tuple(a + b for a, b in zip(lo, dw))
    _design(sc, rng, lo, hi)
    if case["debye"]:
        _debye_slab(sc, slice(max(sc.pml + 1, lo[0] - 6), lo[0] - 1), slice(lo[1], hi[1]), slice(lo[2] - 1, hi[2] + 1))
    sc.ports = [([(nx // 2, ny // 2, ks)], 50.0)]
    return sc, lo, hi, kp


def _scenes_fluxbatch(case, rng):
    dims = np.random.RandomState(case["count"] * 1000 + case["hi"])
    out = []
    for _ in range(case["count"]):
        sc = Scene(_lines(*(8 * int(dims.randint(case["lo"] // 8, case["hi"] // 8 + 1)) for _ in range(3))), case["pml"],
                   10e9, 5e9)
        d = min(case["design"], min(sc.cells) - 2 * sc.pml - 12)
        lo = tuple(n // 2 - d // 2 for n in sc.cells)
        hi = tuple(a + d for a in lo)
        _design(sc, rng, lo, hi)
        _debye_slab(sc, slice(lo[0] - 5, lo[0] - 2), slice(lo[1], hi[1]), slice(lo[2], hi[2]))
        sc.ports = [([(lo[0] + d // 2, lo[1] + d // 2, max(sc.pml + 2, lo[2] - 4))], 1e7)]
        out.append((sc, lo, hi, hi[2] + 2))
    return out


def _far_inputs(case, seed):
    """The patches of a closed box of cells (centres, areas) and accumulated currents on them, with
    the magnitudes a run leaves (f32); directions over the sphere, or a cut when there are few."""
    rng = np.random.RandomState(seed)
    d, n = 0.25e-3, (case["nx"], case["ny"], case["nz"])
    pos = []
    for axis in range(3):
        u, v = (axis + 1) % 3, (axis + 2) % 3
        for plane in (0.0, n[axis] * d):
            p = np.zeros((n[u], n[v], 3))
            p[..., axis] = plane
            p[..., u] = ((np.arange(n[u]) + 0.5) * d)[:, None]
            p[..., v] = ((np.arange(n[v]) + 0.5) * d)[None, :]
            pos.append(p.reshape(-1, 3))
    pos = np.concatenate(pos) - 0.5 * d * np.asarray(n)
    area = np.full(len(pos), d * d)
    acc = (rng.standard_normal((len(pos), 12)) * 1e-12).astype(np.float32)
    acc[:, 6:] *= ETA0
    m = case["dirs"]
    if m < 200:
        th = np.linspace(0.0, math.pi, m) if m > 1 else np.array([0.3])
        ph = np.full(m, 0.4)
    else:
        cols = max(1, int(round(math.sqrt(2 * m))))
        q = np.arange(m)
        th = math.pi * (q // cols + 0.5) / math.ceil(m / cols)
        ph = 2 * math.pi * (q % cols) / cols
    dirs = np.stack([np.sin(th) * np.cos(ph), np.sin(th) * np.sin(ph), np.cos(th)], axis=1)
    return pos, area, acc, dirs


def _torus(case, seed):
    """A closed torus mesh, 2 rings x sides triangles, its minor radius rippled by the seed."""
    rng = np.random.RandomState(seed)
    d, n = DX, (case["nx"], case["ny"], case["nz"])
    big, small = 0.3 * d * min(n[0], n[1]), 0.3 * d * min(n[2], 0.5 * min(n[0], n[1]))
    u = 2 * math.pi * np.arange(case["rings"]) / case["rings"]
    v = 2 * math.pi * np.arange(case["sides"]) / case["sides"]
    r = small * (1.0 + 0.1 * rng.uniform(-1, 1) * np.cos(3 * u[:, None]) + 0.1 * rng.uniform(-1, 1) * np.sin(2 * v[None, :]))
    c = [0.5 * k * d + 0.31 * d * rng.uniform(-1, 1) for k in n]
    p = np.stack([c[0] + (big + r * np.cos(v)[None, :]) * np.cos(u)[:, None],
                  c[1] + (big + r * np.cos(v)[None, :]) * np.sin(u)[:, None], c[2] + r * np.sin(v)[None, :]], axis=-1)
    a, b = p, np.roll(p, -1, axis=0)
    a1, b1 = np.roll(a, -1, axis=1), np.roll(b, -1, axis=1)
    return np.concatenate([np.stack([a, b, b1], axis=2).reshape(-1, 3, 3), np.stack([a, b1, a1], axis=2).reshape(-1, 3, 3)])


# ---- the cases ---------------------------------------------------------------------------------

def prepare(case, seed):
    rng = np.random.RandomState(seed)
    kind, g = case["kind"], _gpu()
    st = dict(kind=kind, case=case, gpu=g)
    if kind == "run":
        sc = _scene_run(case, rng)
        st["sim"], st["pulse"] = sc.sim(), sc.pulse()
        ntff = fdtd.patches(st["sim"], sc.ntff_inset).gpu if sc.ntff_inset is not None else None
        st["extras"] = fdtd.Extras(max_steps=case["steps"], decay_db=math.inf, freqs=sc.freqs, plane_k=sc.plane_k,
                                   ntff=ntff, fused_e=case["fused"])
    elif kind == "session":
        sc = _scene_session(case, rng)
        sim = sc.sim()
        st["session"] = fdtd.Session(g, sim, 0, sc.pulse(), fdtd.Extras(max_steps=SESSION_STEPS, decay_db=math.inf,
                                                                        fused_e=True))
    elif kind == "batch":
        scs = _scenes_batch(case, rng)
        st["batch"] = fdtd.Batch(g, [sc.sim() for sc in scs], [sc.pulse() for sc in scs], SESSION_STEPS)
    elif kind == "flux":
        sc, lo, hi, kp = _scene_flux(case, rng)
        st["sim"], st["pulse"] = sc.sim(), sc.pulse()
        st["spec"] = fdtd.FluxSpec(lo, hi, kp, sc.f0, case["steps"], checkpoints=case["checkpoints"])
    elif kind == "fluxbatch":
        scs = _scenes_fluxbatch(case, rng)
        st["sims"], st["pulses"] = [s[0].sim() for s in scs], [s[0].pulse() for s in scs]
        st["specs"] = [fdtd.FluxSpec(lo, hi, kp, sc.f0, case["steps"], checkpoints=case["checkpoints"])
                       for sc, lo, hi, kp in scs]
    elif kind == "far":
        pos, area, acc, dirs = _far_inputs(case, seed)
        p = fdtd.Patches(pos, area, np.zeros(0, np.uint32))
        st["far"], st["dirs"] = fdtd.Far.load(p, acc, 1, 0, 10e9, gpu=g), dirs
    else:
        st["mesh"], st["grid"] = _torus(case, seed), Grid(*_lines(case["nx"], case["ny"], case["nz"]), 8)
    return st


def run(st):
    kind, case = st["kind"], st["case"]
    if kind == "run":
        r = fdtd.run(st["gpu"], st["sim"], 0, st["pulse"], st["extras"], keep_fields=case["keep"])
        out = {"series": r.series, "decay_db": r.decay_db, "plane": r.plane, "ntff": r.ntff}
        if case["keep"]:
            out["e"], out["h"] = r.e, r.h
        return out
    if kind == "session":
        s = st["session"]
        s.step(case["steps"])
        return {"energy": s.energy(), "series": s.read("series", 2 * SESSION_STEPS)}
    if kind == "batch":
        b = st["batch"]
        b.step(case["steps"])
        b.sync()
        return [b.read(q, "series", 2 * SESSION_STEPS) for q in range(b.size)]
    if kind == "flux":
        r = fdtd.flux_gradient(st["gpu"], st["sim"], 0, st["pulse"], st["spec"])
        return {"objective": np.float64(r.objective), "eps": r.grad_eps, "sigma": r.grad_sigma}
    if kind == "fluxbatch":
        rs = fdtd.flux_gradient_batch(st["gpu"], st["sims"], st["pulses"], st["specs"])
        return [{"objective": np.float64(r.objective), "eps": r.grad_eps, "sigma": r.grad_sigma} for r in rs]
    if kind == "far":
        return st["far"].fields(st["dirs"])
    g, t, grid = st["gpu"], st["mesh"], st["grid"]
    return {"cells": raster.solid_cells(g, t, grid), "solid": raster.solid_edges(g, t, grid),
            "sheet": raster.sheet_edges(g, t, grid)}


def _patch_count(case):
    m = [case[k] + 1 - 2 * (case["pml"] + 3) - 1 for k in ("nx", "ny", "nz")]
    return 2 * (m[0] * m[1] + m[1] * m[2] + m[2] * m[0])


def work(case):
    """A step reads and writes the six field components of a node once (48 bytes, about 36
    operations). A gradient needs a forward and a backward pass of the same size; checkpoints and
    the passes that re-run from them are this code's choice and do not count."""
    kind = case["kind"]

    def nodes(c):
        return (c["nx"] + 1) * (c["ny"] + 1) * (c["nz"] + 1)

    if kind in ("run", "session"):
        steps = nodes(case) * case["steps"]
        b, f = 48.0 * steps, 36.0 * steps
        if kind == "run" and case["model"] == "patch":   # accumulators read and written, currents formed
            p = _patch_count(case) * case["steps"]
            b, f = b + 96.0 * case["freqs"] * p, f + (40.0 + 24.0 * case["freqs"]) * p
        elif kind == "run" and case["freqs"]:
            p = (case["nx"] + 1) * (case["ny"] + 1) * case["steps"]
            b, f = b + (20.0 + 80.0 * case["freqs"]) * p, f + 20.0 * case["freqs"] * p
        if kind == "run" and case["keep"]:
            b += 48.0 * nodes(case)
        return {"bytes": b, "flops": f}
    if kind == "batch" or kind == "fluxbatch":
        dims = np.random.RandomState(case["count"] * 1000 + (case["lo"] if kind == "batch" else case["hi"]))
        total = 0
        for _ in range(case["count"]):
            total += math.prod(8 * int(dims.randint(case["lo"] // 8, case["hi"] // 8 + 1)) + 1 for _ in range(3))
        steps = total * case["steps"] * (2 if kind == "fluxbatch" else 1)
        return {"bytes": 48.0 * steps, "flops": 36.0 * steps}
    if kind == "flux":
        steps = 2 * nodes(case) * case["steps"]
        edges = 3 * case["dx"] * case["dy"] * case["dz"] * case["steps"]
        return {"bytes": 48.0 * steps + 16.0 * edges, "flops": 36.0 * steps}
    if kind == "far":
        p = 2 * (case["nx"] * case["ny"] + case["ny"] * case["nz"] + case["nz"] * case["nx"])
        # per patch and direction six complex multiply-adds and a phase
        return {"bytes": 80.0 * p + 120.0 * case["dirs"], "flops": 60.0 * p * case["dirs"]}
    n = nodes(case)
    tri = 2 * case["rings"] * case["sides"]
    # the masks out, the mesh in; rays down each of the three axes for cells and for each component's edges
    cols = case["nx"] * case["ny"] + case["ny"] * case["nz"] + case["nz"] * case["nx"]
    return {"bytes": 7.0 * n + 72.0 * tri, "flops": 4 * cols * 100.0}


# ---- in 64 bits --------------------------------------------------------------------------------

class _Axis64:
    """One axis's spacings and absorbing-layer factors (convolutional PML, cubic grading)."""

    def __init__(self, line, pml, dt, dev):
        n = len(line)
        d = np.append(np.diff(line), line[-1] - line[-2])
        dd = np.concatenate([[d[0]], 0.5 * (line[2:] - line[:-2]), [d[n - 2]]])
        self.d, self.dd, self.n = d, dd, n
        self.pml = pml if pml > 0 and n > 2 * pml + 2 else 0
        left, right = line[pml], line[n - 1 - pml]

        def grade(x):
            b, c = np.zeros(len(x)), np.zeros(len(x))
            for q, v in enumerate(x):
                rho, depth, cell = (left - v, left - line[0], d[0]) if v < left else (v - right, line[-1] - right, d[n - 2])
                if self.pml == 0 or not rho > 0.0:
                    continue
                r = min(max(rho / depth, 0.0), 1.0)
                s = 3.2 / (ETA0 * cell) * r ** 3
                a = 0.05 * (1.0 - r) * 2.0 * math.pi * EPS0 * 1e9
                b[q] = math.exp(-(s + a) * dt / EPS0)
                c[q] = s * (b[q] - 1.0) / (s + a) if s > 0.0 else 0.0
            return b, c

        be, ce = grade(line)
        bh, ch = grade(0.5 * (line[:-1] + line[1:]))
        t = lambda v: torch.as_tensor(v, dtype=torch.float64, device=dev)  # noqa: E731
        self.inv_d, self.inv_dd = t(1.0 / d), t(1.0 / dd)
        self.be, self.ce, self.bh, self.ch = t(be), t(ce), t(bh), t(ch)


def _along(v, axis):
    return v.reshape([-1 if a == axis else 1 for a in range(3)])


class _Solve64:
    """The Yee update in f64 with torch arrays: H half, E half, Debye poles, the driven port's
    source, port records, running DFTs."""

    def __init__(self, sc, dev, eps=None, sigma=None):
        self.sc, self.dev = sc, dev
        self.n = sc.n
        s = sum(1.0 / np.min(np.diff(v)) ** 2 for v in sc.lines)
        self.dt = 0.99 / (C0 * math.sqrt(s))
        self.ax = [_Axis64(np.asarray(v, np.float64), sc.pml, self.dt, dev) for v in sc.lines]
        self.tau = math.sqrt(math.log(10.0)) / (math.pi * sc.fc)
        self.t0 = 4.0 * self.tau
        self._coefficients(eps, sigma)

    def t(self, v):
        return torch.as_tensor(v, dtype=torch.float64, device=self.dev)

    def _mean(self, cells, c):
        """The area-weighted mean of the four cells around the edges of component c off the faces."""
        u, v = (c + 1) % 3, (c + 2) % 3
        num = den = 0.0
        for ou in (0, 1):
            for ov in (0, 1):
                sl = [slice(None)] * 3
                sl[u], sl[v] = slice(ou, self.n[u] - 2 + ou), slice(ov, self.n[v] - 2 + ov)
                w = _along(self.t(self.ax[u].d[sl[u]]), u) * _along(self.t(self.ax[v].d[sl[v]]), v)
                num = num + cells[tuple(sl)] * w
                den = den + w
        return num / den

    def inner(self, c):
        """The edges of component c off the faces, in the node grid."""
        return tuple(slice(0, self.n[a] - 1) if a == c else slice(1, self.n[a] - 1) for a in range(3))

    def _coefficients(self, eps, sigma):
        sc, dt = self.sc, self.dt
        self.eps_t = self.t(sc.eps) if eps is None else eps
        self.sig_t = self.t(sc.sigma) if sigma is None else sigma
        inf, deb = self.t(sc.inf), self.t(sc.debye)
        half = 0.5 * sum(a * x * dt / (1.0 + 0.5 * x * dt) for x, a in sc.poles)
        self.b = [(1.0 - 0.5 * x * dt) / (1.0 + 0.5 * x * dt) for x, _ in sc.poles]
        self.c = [EPS0 * a * x / (1.0 + 0.5 * x * dt) for x, a in sc.poles]
        self.ca, self.cb, self.dd, self.src = [], [], [], []
        for c in range(3):
            e = EPS0 * self._mean(self.eps_t, c)
            s = self._mean(self.sig_t, c)
            x = s * dt / (2.0 * e)
            ca, cb = (1.0 - x) / (1.0 + x), dt / e / (1.0 + x)
            if sc.pec is not None:
                keep = (~torch.as_tensor(sc.pec[c], device=self.dev)[self.inner(c)]).to(torch.float64)
                ca, cb = ca * keep, cb * keep
            dd = self._mean(deb, c)
            live = (dd > 0.0) & (cb != 0.0)
            if c == 2:
                for q, (col, r) in enumerate(sc.ports):
                    r_edge = r / len(col)
                    for i, j, k in col:
                        p = (i - 1, j - 1, k)
                        area, length = self.ax[0].dd[i] * self.ax[1].dd[j], self.ax[2].d[k]
                        beta = dt * length / (2.0 * r_edge * float(e[p]) * area) + float(x[p])
                        ca[p], cb[p] = (1.0 - beta) / (1.0 + beta), dt / (float(e[p]) * (1.0 + beta))
                        live[p] = False
                        if q == 0:
                            self.src.append(((i, j, k), dt / (float(e[p]) * (1.0 + beta) * r_edge * area) / len(col)))
            if sc.poles:
                eps_d = EPS0 * (self._mean(inf, c) + dd * half)
                ca, cb = torch.where(live, torch.ones_like(ca), ca), torch.where(live, dt / eps_d, cb)
            self.ca.append(ca)
            self.cb.append(cb)
            self.dd.append(torch.where(live, dd, torch.zeros_like(dd)) if bool(live.any()) else None)
        self.debye_on = bool(sc.poles) and any(d is not None for d in self.dd)

    def start(self):
        z = lambda *s: torch.zeros(s, dtype=torch.float64, device=self.dev)  # noqa: E731
        st = {"e": [z(*self.n) for _ in range(3)], "h": [z(*self.n) for _ in range(3)], "psi": {}, "s": {}}
        return st

    def _term(self, st, key, diff, axis, inv, b, c, lo, hi):
        """diff / spacing along `axis`, with the layer's convolution in the slots [0, lo) and [hi, ...)."""
        t = diff * _along(inv, axis)
        if self.ax[axis].pml == 0:
            return t
        out = t.clone()
        for side, sl in ((0, slice(0, lo)), (1, slice(hi, diff.shape[axis]))):
            ix = tuple(sl if a == axis else slice(None) for a in range(3))
            old = st["psi"].get(key + (side,))
            r = _along(c[sl], axis) * t[ix]
            if old is not None:
                r = r + _along(b[sl], axis) * old
            st["psi"][key + (side,)] = r
            out[ix] = out[ix] + r
        return out

    def step(self, st, m):
        """Step m; returns a new state (the old one is left as it was)."""
        n, ax, sc = self.n, self.ax, self.sc
        st = {"e": list(st["e"]), "h": list(st["h"]), "psi": dict(st["psi"]), "s": dict(st["s"])}
        e, kmu = st["e"], self.dt / MU0
        new = []
        for c in range(3):
            u, v = (c + 1) % 3, (c + 2) % 3
            at = lambda du, dv: tuple(slice(du, n[a] - 1 + du) if a == u else slice(dv, n[a] - 1 + dv) if a == v  # noqa: E731
                                      else slice(None) for a in range(3))
            p = [ax[w].pml for w in range(3)]
            t1 = self._term(st, ("h", c, u), e[v][at(1, 0)] - e[v][at(0, 0)], u, ax[u].inv_d[:-1], ax[u].bh, ax[u].ch,
                            p[u], n[u] - 1 - p[u])
            t2 = self._term(st, ("h", c, v), e[u][at(0, 1)] - e[u][at(0, 0)], v, ax[v].inv_d[:-1], ax[v].bh, ax[v].ch,
                            p[v], n[v] - 1 - p[v])
            h = st["h"][c].clone()
            h[at(0, 0)] -= kmu * (t1 - t2)
            new.append(h)
        st["h"] = h = new
        new = []
        for c in range(3):
            u, v = (c + 1) % 3, (c + 2) % 3
            at = lambda du, dv: tuple(slice(0, n[a] - 1) if a == c else slice(1 - du, n[a] - 1 - du) if a == u  # noqa: E731
                                      else slice(1 - dv, n[a] - 1 - dv) for a in range(3))
            p = [ax[w].pml for w in range(3)]
            here = at(0, 0)
            t1 = self._term(st, ("e", c, u), h[v][here] - h[v][at(1, 0)], u, ax[u].inv_dd[1:-1], ax[u].be[1:-1],
                            ax[u].ce[1:-1], max(p[u] - 1, 0), n[u] - 1 - p[u])
            t2 = self._term(st, ("e", c, v), h[u][here] - h[u][at(0, 1)], v, ax[v].inv_dd[1:-1], ax[v].be[1:-1],
                            ax[v].ce[1:-1], max(p[v] - 1, 0), n[v] - 1 - p[v])
            old = e[c][here]
            x = self.ca[c] * old + self.cb[c] * (t1 - t2)
            if self.debye_on and self.dd[c] is not None:
                s = [st["s"].get((c, q)) for q in range(len(self.b))]
                for q, b in enumerate(self.b):
                    if s[q] is not None:
                        x = x - self.cb[c] * (0.5 * (1.0 + b)) * s[q]
                for q, (b, k) in enumerate(zip(self.b, self.c)):
                    r = self.dd[c] * k * (x - old)
                    st["s"][(c, q)] = r if s[q] is None else r + b * s[q]
            ec = e[c].clone()
            ec[here] = x
            new.append(ec)
        st["e"] = new
        t = (m + 0.5) * self.dt
        y = (t - self.t0) / self.tau
        p = math.exp(-y * y) * math.cos(2.0 * math.pi * sc.f0 * (t - self.t0))
        for at, w in self.src:
            new[2][at] -= w * p
        return st

    def probe(self, st):
        """Each port's voltage along its column and current around it."""
        out = []
        dx, dy, dz = self.ax[0].dd, self.ax[1].dd, self.ax[2].d
        for col, _ in self.sc.ports:
            height = sum(dz[k] for _, _, k in col)
            v = cur = 0.0
            for i, j, k in col:
                v = v - st["e"][2][i, j, k] * dz[k]
                hx, hy = st["h"][0], st["h"][1]
                cur = cur + dz[k] / height * ((hy[i, j, k] - hy[i - 1, j, k]) * dy[j] - (hx[i, j, k] - hx[i, j - 1, k]) * dx[i])
            out += [v, cur]
        return torch.stack(out)

    def phases(self, m, f, sign):
        """(cos, sin) dt of e^{-jwt} at the times of E and of H after step m."""
        w = 2.0 * math.pi * f
        return [(math.cos(w * t) * self.dt, sign * math.sin(w * t) * self.dt) for t in ((m + 1.0) * self.dt, (m + 0.5) * self.dt)]

    def add_plane(self, st, m, k, freqs, acc):
        """The running DFT of Ex, Ey, Ez, Hx, Hy on the plane k: acc (frequency, value, i, j)."""
        f = torch.stack([st["e"][0][:, :, k], st["e"][1][:, :, k], st["e"][2][:, :, k], st["h"][0][:, :, k], st["h"][1][:, :, k]])
        rows = []
        for fr in freqs:
            (ec, es), (hc, hs) = self.phases(m, fr, -1.0)
            w = self.t([[ec, es]] * 3 + [[hc, hs]] * 2)
            rows.append((f[:, None] * w[:, :, None, None]).reshape(10, *f.shape[1:]))
        return acc + torch.stack(rows)

    def currents(self, st, inset):
        """J = n x H and M = E x n on the patches of the box `inset` cells inside the layer, (3, patches) each."""
        p = self.sc.pml + inset
        lo, hi = [p] * 3, [v - 1 - p for v in self.n]
        js, ms = [], []
        for axis in range(3):
            u, v = (axis + 1) % 3, (axis + 2) % 3
            for side, plane in ((-1.0, lo[axis]), (1.0, hi[axis])):
                def at(f, da, du, dv):
                    ix = [0, 0, 0]
                    ix[axis], ix[u], ix[v] = plane + da, slice(lo[u] + du, hi[u] + du), slice(lo[v] + dv, hi[v] + dv)
                    r = f[tuple(ix)]
                    return r if u < v else r.transpose(0, 1)
                e, h = st["e"], st["h"]
                eu = 0.5 * (at(e[u], 0, 0, 0) + at(e[u], 0, 0, 1))
                ev = 0.5 * (at(e[v], 0, 0, 0) + at(e[v], 0, 1, 0))
                hu = 0.25 * (at(h[u], 0, 0, 0) + at(h[u], -1, 0, 0) + at(h[u], 0, 1, 0) + at(h[u], -1, 1, 0))
                hv = 0.25 * (at(h[v], 0, 0, 0) + at(h[v], -1, 0, 0) + at(h[v], 0, 0, 1) + at(h[v], -1, 0, 1))
                j, m = [None] * 3, [None] * 3
                zero = torch.zeros_like(eu)
                j[axis], j[u], j[v] = zero, -side * hv, side * hu
                m[axis], m[u], m[v] = zero, side * ev, -side * eu
                js.append(torch.stack([x.reshape(-1) for x in j]))
                ms.append(torch.stack([x.reshape(-1) for x in m]))
        return torch.cat(js, 1), torch.cat(ms, 1)

    def energy(self, st):
        return float(sum((x * x).sum() for x in st["e"]) + 376.73 ** 2 * sum((x * x).sum() for x in st["h"]))


def _exact_run(case, sc, dev):
    s = _Solve64(sc, dev)
    st = s.start()
    steps, series = case["steps"], []
    nf = len(sc.freqs)
    plane = torch.zeros((nf, 10) + s.n[:2], dtype=torch.float64, device=dev) if sc.plane_k is not None else None
    ntff = None
    peak = decay = 0.0
    for m in range(steps):
        st = s.step(st, m)
        series.append(s.probe(st))
        if plane is not None:
            plane = s.add_plane(st, m, sc.plane_k, sc.freqs, plane)
        if sc.ntff_inset is not None:
            j, mm = s.currents(st, sc.ntff_inset)
            if ntff is None:
                ntff = torch.zeros(nf, 2, 3, 2, j.shape[1], dtype=torch.float64, device=dev)
            for q, f in enumerate(sc.freqs):
                (ec, es), (hc, hs) = s.phases(m, f, -1.0)
                ntff[q, 0, :, 0] += hc * j
                ntff[q, 0, :, 1] += hs * j
                ntff[q, 1, :, 0] += ec * mm
                ntff[q, 1, :, 1] += es * mm
        if (m + 1) % 1000 == 0 or m + 1 == steps:   # run()'s energy checks
            en = s.energy(st)
            peak = max(peak, en)
            decay = 10.0 * math.log10(peak / en) if en > 0.0 else 0.0
    none = np.zeros(0)
    out = {"series": torch.stack(series).reshape(-1), "decay_db": decay,
           "plane": plane.reshape(nf * 10, -1).t().reshape(-1) if plane is not None else none,
           "ntff": ntff.reshape(nf * 12, -1).t().reshape(-1) if ntff is not None else none}
    if case["keep"]:
        out["e"], out["h"] = torch.stack(st["e"]).reshape(-1), torch.stack(st["h"]).reshape(-1)
    return {k: v.cpu().numpy() if isinstance(v, torch.Tensor) else v for k, v in out.items()}


def _exact_steps(sc, steps, dev):
    s = _Solve64(sc, dev)
    st = s.start()
    series = np.zeros((SESSION_STEPS, 2))
    for m in range(steps):
        st = s.step(st, m)
        series[m] = s.probe(st).cpu().numpy()
    return s.energy(st), series.reshape(-1)


def _exact_flux(sc, lo, hi, kp, steps, dev):
    from torch.utils.checkpoint import checkpoint
    box = tuple(slice(a, b) for a, b in zip(lo, hi))
    eps, sig = (torch.as_tensor(a[box].astype(np.float64), device=dev).requires_grad_() for a in (sc.eps, sc.sigma))
    full = []
    for a, part in ((sc.eps, eps), (sc.sigma, sig)):
        t = torch.as_tensor(a, dtype=torch.float64, device=dev).clone()
        t[box] = part
        full.append(t)
    s = _Solve64(sc, dev, *full)
    st = s.start()
    acc = torch.zeros((1, 10) + s.n[:2], dtype=torch.float64, device=dev)

    def piece(st, acc, a, b):
        for m in range(a, b):
            st = s.step(st, m)
            acc = s.add_plane(st, m, kp, [sc.f0], acc)
        return st, acc

    for a in range(0, steps, 20):
        st, acc = checkpoint(piece, st, acc, a, min(a + 20, steps), use_reentrant=False)
    f = torch.view_as_complex(acc[0].reshape(5, 2, *s.n[:2]).permute(0, 2, 3, 1).contiguous())
    w = slice(sc.pml, s.n[0] - sc.pml), slice(sc.pml, s.n[1] - sc.pml)
    da = s.t(s.ax[0].dd)[w[0], None] * s.t(s.ax[1].dd)[None, w[1]]
    f = [x[w] for x in f]
    flux = (da * (f[0] * f[4].conj() - f[1] * f[3].conj())).sum()
    obj = flux.real ** 2 + flux.imag ** 2
    ge, gs = torch.autograd.grad(obj, (eps, sig))
    return {"objective": np.float64(float(obj.detach())), "eps": ge.cpu().numpy(), "sigma": gs.cpu().numpy()}


def _exact_far(case, seed, dev):
    pos, area, acc, dirs = (torch.as_tensor(v, dtype=torch.float64, device=dev) for v in _far_inputs(case, seed))
    k = 2.0 * math.pi * 10e9 / C0
    cur = torch.view_as_complex(acc.reshape(-1, 6, 2).contiguous())
    out = []
    for d in dirs.split(max(1, 40_000_000 // len(pos))):
        arg = k * (d @ pos.t())
        s = torch.polar(area.expand_as(arg), arg) @ cur
        nn, ll = s[:, :3], s[:, 3:]
        dc = d.to(nn.dtype)
        perp = nn - (nn * dc).sum(1, keepdim=True) * dc
        out.append((torch.linalg.cross(dc, ll) - ETA0 * perp) * (k / (4.0 * math.pi)))
    return torch.cat(out).cpu().numpy()


def exact(case, seed):
    dev = torch.device("cuda")
    rng = np.random.RandomState(seed)
    kind = case["kind"]
    if kind == "flux":
        return _exact_flux(*_scene_flux(case, rng), case["steps"], dev)
    if kind == "fluxbatch":
        return [_exact_flux(*s, case["steps"], dev) for s in _scenes_fluxbatch(case, rng)]
    with torch.no_grad():
        if kind == "run":
            return _exact_run(case, _scene_run(case, rng), dev)
        if kind == "session":
            en, series = _exact_steps(_scene_session(case, rng), case["steps"], dev)
            return {"energy": en, "series": series}
        if kind == "batch":
            return [_exact_steps(sc, case["steps"], dev)[1] for sc in _scenes_batch(case, rng)]
        if kind == "far":
            return _exact_far(case, seed, dev)
    return None   # raster: truth values
