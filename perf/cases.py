"""Performance cases of the batch evaluator and its adjoint, through the package's public calls.

A case is one call that a design search makes: a population of edited terrains run through a
storm (run_batch, run_primitives, run_ladder), or the gradient of the assets' objective
(vjp, vjp_primitives). Terrain, storm, assets and guard of a case are fixed, as in a search;
the designs come from the seed. One GpuSolver serves the whole process, as a search keeps
one. `exact` is a plain torch restatement of the scheme in 64 bits.
"""
from __future__ import annotations

import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "inverse-terrain-engine_b200"))

from itr_gpu import (Asset, FineTerrain, GeoTransform, GpuSolver, Hyetograph, MonitorSet, Objective, ObjectiveDef,  # noqa: E402
                     PreparedTerrain, Primitive, Segment, SolverParams, TerrainBase, TerrainEdit)

MAX_DZ = 1.0          # largest edit of a cell [m]
FLOPS_STEP = 220      # additions, multiplications, divisions and roots of one cell and step (2 faces, 1 update)
FLOPS_ADJOINT = 700   # the same of one backward step


def _case(name, call, nx, ny, cell, designs, seconds, **kw):
    c = {"name": name, "call": call, "nx": nx, "ny": ny, "cell": cell, "designs": designs, "seconds": seconds, "level": 1,
         "edges": "outlet", "rain": 100.0, "depth": 0.0, "prims": 4, "abort": False, "interval": 128}
    c.update(kw)
    return c


def listed():
    return [
        # one candidate on the coarsest valley grid, the first five minutes: the shortest call of a search
        _case("valley 45x35 x1", "batch", 45, 35, 10.0, 1, 300.0, prims=2),
        # a generation on a coarse fidelity level (crest faces, two jumps each)
        _case("crest 45x35 x32", "batch", 90, 70, 5.0, 32, 1200.0, level=2, rain=80.0, prims=3),
        # a generation of the valley scene, whole storm, designs stopped when they breach the guard
        _case("valley 90x70 x16 guarded", "batch", 90, 70, 5.0, 16, 2400.0, rain=80.0, prims=2, abort=True),
        # the population workload of the benchmark, whole storm
        _case("hills 120x96 x64", "batch", 120, 96, 5.0, 64, 3600.0),
        # grid sizes that divide by nothing, more designs than one round of clusters
        _case("odd 157x101 x40", "batch", 157, 101, 3.7, 40, 900.0),
        # three fidelity levels of one scene in one call, aborts live
        _case("ladder 45/90/180 x112", "ladder", 180, 140, 2.5, 16, 900.0, rain=80.0, prims=3, abort=True),
        # rain-free valley fed through its edges: stage and inflow ghosts, dry rows
        _case("river valley 90x70 x48", "batch", 90, 70, 5.0, 48, 900.0, edges="river", rain=0.0, prims=2),
        # the fine hills grid, designs as primitives
        _case("hills 240x192 x32", "primitives", 240, 192, 2.5, 32, 900.0),
        # the largest grid: one candidate, and a generation
        _case("fractal 1024x1024 x1", "batch", 1024, 1024, 2.0, 1, 600.0, rain=60.0),
        _case("fractal 1024x1024 x16", "primitives", 1024, 1024, 2.0, 16, 600.0, rain=60.0, prims=6),
        # gradients: a population of face jumps on the fine hills grid (below 2^18 cells), ponded start
        _case("adjoint 240x192 x8", "vjp", 240, 192, 2.5, 8, 60.0, depth=0.2),
        # the polishing step of one incumbent and its neighbours on a large grid, gradient per primitive
        _case("adjoint 600x512 x4", "vjp_primitives", 600, 512, 2.0, 4, 40.0, rain=60.0, depth=0.2, prims=6),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    most = max(work(c)["flops"] for c in listed())
    while True:
        kind = rng.choice(["batch", "batch", "batch", "primitives", "crest", "river", "ladder", "vjp", "vjp_primitives"])
        big = kind in ("batch", "primitives") and rng.random() < 0.25
        nx = _log_int(rng, 300, 1024) if big else _log_int(rng, 24, 300)
        ny = max(20, int(round(nx * rng.uniform(0.6, 1.3))))
        seconds = round(math.exp(rng.uniform(math.log(120.0), math.log(2400.0))), 0)
        kw = {"rain": round(rng.uniform(40.0, 120.0), 1), "prims": rng.randint(1, 6)}
        designs = _log_int(rng, 1, 16 if big else 96)
        call = kind
        if kind == "batch":
            kw["abort"] = rng.random() < 0.3
            kw["depth"] = rng.choice([0.0, 0.0, 0.1])
        elif kind == "crest":
            call, kw["level"] = "batch", 2
            nx, ny, designs = min(nx, 180), min(ny, 180), min(designs, 48)
        elif kind == "river":
            call, kw["edges"], kw["rain"] = "batch", "river", rng.choice([0.0, 20.0])
        elif kind == "ladder":
            nx, ny, designs = 4 * min(max(nx // 4, 12), 40), 4 * min(max(ny // 4, 12), 40), min(designs, 24)
            kw["abort"] = rng.random() < 0.7
        elif kind != "primitives":
            designs, seconds, kw["depth"] = min(designs, 8), float(rng.randint(20, 60)), rng.choice([0.1, 0.2, 0.3])
            kw["interval"] = rng.choice([32, 64, 128])
        c = _case("drawn", call, nx, ny, round(math.exp(rng.uniform(math.log(2.0), math.log(10.0))), 1), designs, seconds, **kw)
        del c["name"]
        if work(c)["flops"] <= 0.6 * most:
            return c


# ---------------------------------------------------------------- the scene of a case ----
@functools.lru_cache(maxsize=4)
def _dem(nx, ny, cell):
    """A sloping field with hills, one winding channel and noise, the same for every cell size of one domain."""
    rng = np.random.default_rng(20261203)
    Lx, Ly = nx * cell, ny * cell
    x = (np.arange(nx) + 0.5)[None, :] * cell / Lx
    y = 1.0 - (np.arange(ny) + 0.5)[:, None] * cell / Ly
    size = min(Lx, Ly)
    z = 40.0 + 0.02 * size * y + 0.004 * size * x
    for _ in range(4):
        hx, hy, a, s = rng.uniform(0.1, 0.9), rng.uniform(0.2, 0.9), rng.uniform(0.004, 0.012), rng.uniform(0.06, 0.12)
        z = z + a * size * np.exp(-((x - hx) ** 2 + (y - hy) ** 2) / (2 * s * s))
    mid = 0.5 + 0.15 * np.sin(5.0 * y + 1.0)
    z = z - 1.8 * np.exp(-((x - mid) * Lx / max(12.0, 0.03 * Lx)) ** 2)
    for _ in range(24):
        k, ph = rng.normal(0.0, 22.0, size=2), rng.uniform(0.0, 2 * math.pi)
        z = z + 0.08 * np.cos(k[0] * x + k[1] * y + ph)
    return z


def _rect(nx, ny, fx, fy, w):
    c0, r0 = int(fx * nx), int((1.0 - fy) * ny)
    return [r * nx + c for r in range(r0, min(r0 + w, ny)) for c in range(c0, min(c0 + w, nx))]


@functools.lru_cache(maxsize=4)
def _scene(nx, ny, cell, level, edges):
    geo = GeoTransform(0.0, ny * cell, cell, cell)
    walls = np.zeros((ny, nx), bool)
    walls[int(0.55 * ny):int(0.55 * ny) + 2, int(0.3 * nx):int(0.3 * nx) + 3] = True   # a building
    dem = _dem(nx, ny, cell)
    fine = FineTerrain(dem, walls, np.full((ny, nx), 0.04), geo)
    segs = [Segment("transmissive", "south")]
    if edges == "river":
        L = nx * cell
        top, low = float(dem[0].min()), float(dem[-1].min())
        segs = [Segment("inflow", "north", (0.35 * L, 0.75 * L), hydrograph=[(0.0, 0.5), (300.0, 6.0), (900.0, 3.0), (2400.0, 0.5)]),
                Segment("stage", "west", (0.6 * ny * cell, 0.8 * ny * cell), stage_m=top - 1.0),
                Segment("transmissive", "east"), Segment("stage", "south", stage_m=low + 0.2)]
    base = TerrainBase(fine, level, segs)
    bx, by = base.nx, base.ny
    w = max(2, bx // 40)
    assets = [Asset(f"house{i}", _rect(bx, by, fx, fy, w), 0.05)
              for i, (fx, fy) in enumerate(((0.44, 0.35), (0.56, 0.3), (0.4, 0.2), (0.62, 0.55)))]
    obj = Objective(ObjectiveDef(assets, sorted(set(_rect(bx, by, 0.45, 0.12, 2 * w))), guard_tolerance_m=0.02))
    editable = ~walls
    return base, obj, editable


def _storm(case):
    p = case["rain"]
    pts = [(0, 0), (2400, 0)] if p == 0.0 else [(0, 0.1 * p), (900, p), (3600, 0.2 * p)]
    return SolverParams(duration_s=case["seconds"], sync_interval_s=60.0, rain=Hyetograph.from_mm_h(pts),
                        infil_capacity=6.0 / 1000.0 / 3600.0, initial_depth=case["depth"])


def _primitives(case, seed):
    """Seeded berms, swales, cuts and mounds around the middle of the domain, quantised as a search gives them."""
    rng = np.random.default_rng(seed)
    Lx, Ly = case["nx"] * case["cell"], case["ny"] * case["cell"]
    size = min(Lx, Ly)
    out = []
    for _ in range(case["designs"]):
        one = []
        for _ in range(case["prims"]):
            ht = round(float(rng.uniform(-0.5, 0.5)), 2)
            kind = int(rng.integers(0, 4)) if ht > 0 else 1
            one.append(Primitive(kind, round(2 * float(rng.uniform(0.25, 0.75)) * Lx) / 2, round(2 * float(rng.uniform(0.25, 0.75)) * Ly) / 2,
                                 round(2 * float(rng.uniform(0.05, 0.2)) * size) / 2, max(2.0 * case["cell"], round(2 * float(rng.uniform(3.0, 9.0))) / 2),
                                 float(rng.integers(0, 180)), ht if kind != 2 else -abs(ht)))
        out.append(one)
    return out


def _dz(prims, case, editable):
    """Edit of every cell: heights times profiles, a mean of 4x4 samples a cell, clamped."""
    nx, ny, cell = case["nx"], case["ny"], case["cell"]
    dz = np.zeros((ny, nx))
    for p in prims:
        a = p.angle_deg * math.pi / 180.0
        ex, ey = (0.0, 0.0) if p.kind == 3 else (0.5 * p.length * math.cos(a), 0.5 * p.length * math.sin(a))
        r = 0.5 * p.width
        c0 = min(max(int((p.cx - abs(ex) - r) / cell) - 1, 0), nx - 1)
        c1 = min(int((p.cx + abs(ex) + r) / cell) + 2, nx)
        r0 = min(max(int(ny - (p.cy + abs(ey) + r) / cell) - 1, 0), ny - 1)
        r1 = min(int(ny - (p.cy - abs(ey) - r) / cell) + 2, ny)
        if c0 >= c1 or r0 >= r1 or p.height == 0.0:
            continue
        X = (c0 + (np.arange(4 * (c1 - c0)) + 0.5) / 4) * cell
        Y = ny * cell - (r0 + (np.arange(4 * (r1 - r0)) + 0.5) / 4) * cell
        X, Y = np.meshgrid(X, Y)
        vx, vy = 2 * ex, 2 * ey
        l2 = vx * vx + vy * vy
        t = np.clip(((X - p.cx + ex) * vx + (Y - p.cy + ey) * vy) / l2, 0.0, 1.0) if l2 > 0 else 0.0
        s = np.hypot(p.cx - ex + t * vx - X, p.cy - ey + t * vy - Y) / r
        u = np.where(s <= 0.5, 0.0, 2 * s - 1) if p.kind == 2 else s
        f = np.where(s < 1.0, (1 - u * u) ** 2, 0.0)
        dz[r0:r1, c0:c1] += p.height * f.reshape(r1 - r0, 4, c1 - c0, 4).mean(axis=(1, 3))
    return np.where(editable, np.clip(dz, -MAX_DZ, MAX_DZ), 0.0)


def _prepared(base, dz):
    """The edited terrain as run_batch takes it."""
    cell = base.fine.geo.dx
    cut, fill = float(-dz[dz < 0].sum()) * cell * cell, float(dz[dz > 0].sum()) * cell * cell
    t = PreparedTerrain(base)
    if base.level > 1:
        rows, cols = np.nonzero(dz)
        if len(rows):
            r0, r1, c0, c1 = rows.min(), rows.max() + 1, cols.min(), cols.max() + 1
            t.apply_edit(TerrainEdit(int(c0), int(r0), int(c1 - c0), int(r1 - r0), dz[r0:r1, c0:c1].ravel().copy(), cut, fill))
        return t
    t.z = np.where(base.wall, base.z, base.fine.z + dz)
    t.dzx[:, 1:-1] = (t.z[:, 1:] - t.z[:, :-1]).astype(np.float32)
    t.dzy[1:-1, :] = (t.z[1:, :] - t.z[:-1, :]).astype(np.float32)
    t.cut_m3, t.fill_m3 = cut, fill
    return t


@functools.lru_cache(maxsize=1)
def _solver():
    return GpuSolver()


@functools.lru_cache(maxsize=8)
def _baseline(key):
    """Monitor maxima of the unedited terrain, which guard tests compare with."""
    case = dict(key)
    base, obj, _ = _scene(case["nx"], case["ny"], case["cell"], case["level"], case["edges"])
    return _solver().run_batch(_storm(case), [PreparedTerrain(base)], obj.monitors, want_depth=False)[0].monitor_max


def _levels(case):
    """The ladder's groups: the coarse, middle and fine grids of one domain, more designs on the coarser ones."""
    return [dict(case, nx=case["nx"] // k, ny=case["ny"] // k, cell=case["cell"] * k, designs=case["designs"] * m)
            for k, m in ((4, 4), (2, 2), (1, 1))]


def _group(case, seed):
    base, obj, editable = _scene(case["nx"], case["ny"], case["cell"], case["level"], case["edges"])
    g = {"terrains": [_prepared(base, _dz(p, case, editable)) for p in _primitives(case, seed)], "monitors": obj.monitors,
         "objective": obj}
    if case["abort"]:
        g["baseline_max"] = _baseline(tuple(sorted((k, v) for k, v in case.items() if k != "name")))
        g["guard_abort"] = True
    return g


def prepare(case, seed):
    s = {"case": case, "solver": _solver(), "params": _storm(case)}
    if case["call"] == "ladder":
        s["groups"] = [_group(c, seed + k) for k, c in enumerate(_levels(case))]
    elif case["call"] in ("primitives", "vjp_primitives"):
        s["base"], s["objective"], s["editable"] = _scene(case["nx"], case["ny"], case["cell"], case["level"], case["edges"])
        s["prims"] = _primitives(case, seed)
    else:
        s.update(_group(case, seed))
    return s


def _answer(runs):
    out = {"monitor_max": np.stack([r.monitor_max for r in runs]), "j": np.array([r.j for r in runs]),
           "steps": np.array([r.steps for r in runs]), "status": np.array([r.status for r in runs]),
           "feasible": np.array([r.feasible for r in runs]), "t_end": np.array([r.t_end for r in runs])}
    for k in ("depth", "peak", "dj_ddzx", "dj_ddzy"):
        if getattr(runs[0], k) is not None:
            out[k] = np.stack([getattr(r, k) for r in runs])
    return out


def run(s):
    g, p, c = s["solver"], s["params"], s["case"]
    if c["call"] == "batch":
        return _answer(g.run_batch(p, s["terrains"], s["monitors"], objective=s["objective"], baseline_max=s.get("baseline_max"),
                                   guard_abort=s.get("guard_abort", False), want_peak=True))
    if c["call"] == "ladder":
        return [_answer(r) for r in g.run_ladder(p, s["groups"])]
    if c["call"] == "primitives":
        runs, cut, fill = g.run_primitives(p, s["base"], s["prims"], s["objective"].monitors, s["editable"], MAX_DZ,
                                           objective=s["objective"], want_depth=False)
        return dict(_answer(runs), cut=cut, fill=fill)
    if c["call"] == "vjp":
        return _answer(g.vjp(p, s["terrains"], s["monitors"], s["objective"], checkpoint_interval=c["interval"]))
    runs, gp = g.vjp_primitives(p, s["base"], s["prims"], s["objective"].monitors, s["objective"], s["editable"], MAX_DZ,
                                checkpoint_interval=c["interval"])
    return dict(_answer(runs), dj_dprim=np.stack(gp))


def _steps(case):
    """About how many steps the storm takes: the wave speed grows as water gathers."""
    speed = 0.5 + 1.6 * math.sqrt(case["depth"] * 9.81) + 2.5 * min(1.0, case["seconds"] / 2400.0) ** 0.7
    return case["seconds"] * max(0.2, 2.0 * speed / (0.35 * case["cell"] * case["level"]))


def work(case):
    if case["call"] == "ladder":
        parts = [work(dict(c, call="batch")) for c in _levels(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    nx, ny = -(-case["nx"] // case["level"]), -(-case["ny"] // case["level"])
    cells, n = nx * ny, case["designs"]
    jumps = (2 if case["level"] > 1 else 1) * 2 * 4 * cells
    outs = {"batch": 8, "primitives": 0, "vjp": 20, "vjp_primitives": 20}[case["call"]] * cells
    ins = 8 * cells + (0 if "primitives" in case["call"] else n * jumps)
    per = FLOPS_STEP if "vjp" not in case["call"] else FLOPS_STEP + FLOPS_ADJOINT
    return {"bytes": float(ins + n * outs), "flops": float(per) * cells * n * _steps(case)}


# ------------------------------------------------- the scheme in 64 bits, plain torch ----
def _jumps(t, mode):
    a = [torch.from_numpy(np.asarray(v, dtype=np.float64)) for v in ((t.dzx, t.dzx2, t.dzy, t.dzy2) if mode else (t.dzx, t.dzy))]
    return a if mode else [a[0].clamp(min=0), (-a[0]).clamp(min=0), a[1].clamp(min=0), (-a[1]).clamp(min=0)]


def _root(x):
    """sqrt with derivative 0 at 0."""
    ok = x > 0
    return torch.where(ok, torch.sqrt(torch.where(ok, x, torch.ones_like(x))), torch.zeros_like(x))


class _Exact:
    """One batch on one grid: state [3][n, ny, nx], per-design time, the step as a function of state and jumps."""

    def __init__(self, base, p, terrains):
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        f = lambda a: torch.from_numpy(np.asarray(a, dtype=np.float64)).to(self.dev)  # noqa: E731
        self.base, self.p, self.n = base, p, len(terrains)
        self.wet, self.gn2 = f(base.wet)[None], f(base.gn2)[None]
        js = [_jumps(t, base.mode) for t in terrains]
        self.cuts = [torch.stack([j[k] for j in js]).to(self.dev) for k in range(4)]   # left, right of x-faces, upper, lower of y-faces
        b = base
        self.code = torch.from_numpy(b.bc.astype(np.int64)).to(self.dev)
        st = np.where(b.bc == 2, b.bc_stage, 0.0)
        self.stage = torch.stack([f(np.maximum(st - t.z_edge(), 0.0)) for t in terrains])
        self.inv_len, self.hydro = f(b.bc_inv_len), b.bc_inflow
        self.pts = torch.tensor(p.rain.pts, dtype=torch.float64, device=self.dev)
        n, ny, nx = self.n, b.ny, b.nx
        h0 = f(np.where(base.wall, 0.0, np.float32(p.initial_depth)))
        self.state = torch.stack([h0.expand(n, ny, nx), torch.zeros(n, ny, nx, dtype=torch.float64, device=self.dev),
                                  torch.zeros(n, ny, nx, dtype=torch.float64, device=self.dev)])
        self.t = torch.zeros(n, dtype=torch.float64, device=self.dev)

    def rate_sum(self, x):
        """The storm's integral from 0 to x."""
        t, r = self.pts[:, 0], self.pts[:, 1]
        seg = torch.diff(t) * (r[1:] + r[:-1]) / 2
        cum = torch.cat([torch.zeros(1, dtype=torch.float64, device=self.dev), torch.cumsum(seg, 0)])
        k = torch.clamp(torch.searchsorted(t, x, right=True) - 1, 0, len(t) - 1)
        k1 = torch.clamp(k + 1, max=len(t) - 1)
        span = torch.where(k1 > k, t[k1] - t[k], torch.ones_like(x))
        rx = r[k] + (r[k1] - r[k]) * torch.where(k1 > k, (x - t[k]) / span, torch.zeros_like(x))
        return cum[k] + (x - t[k]) * (r[k] + rx) / 2

    def inflow(self):
        """Discharge per metre of every boundary cell [n, 2 nx + 2 ny]."""
        q = torch.zeros(self.n, len(self.code), dtype=torch.float64, device=self.dev)
        for k, pts in enumerate(self.base.hydrographs):
            v = torch.from_numpy(np.interp(self.t.cpu().numpy(), [a for a, _ in pts], [b for _, b in pts])).to(self.dev)
            at = torch.from_numpy(self.hydro == k).to(self.dev)
            q[:, at] = v[:, None] * self.inv_len[at][None] * self.p.inflow_scale
        return q

    def ghost(self, h, qx, qy, lo, hi, normal_x, sign, q):
        code = self.code[lo:hi][None]
        flip = torch.where(code == 0, -1.0, 1.0)
        gh, a, b = h, qx * (flip if normal_x else 1.0), qy * (1.0 if normal_x else flip)
        if self.base.has_stage or self.base.has_inflow:
            gh = torch.where(code == 2, self.stage[:, lo:hi], gh)
            qi = q[:, lo:hi]
            crit = (qi * qi / 9.81) ** (1.0 / 3.0)
            gh = torch.where(code == 3, torch.maximum(h, crit), gh)
            nrm, tan = torch.where(code == 3, sign * qi, a if normal_x else b), torch.where(code == 3, torch.zeros_like(a), b if normal_x else a)
            a, b = (nrm, tan) if normal_x else (tan, nrm)
        return gh, a, b

    def vel(self, h, qx, qy):
        h2 = h * h
        t = 2 * h / (h2 + torch.clamp(h2, min=self.p.h_eps ** 2))
        return h, qx * t, qy * t, _root(9.81 * h)

    def face(self, L, R, dl, dr, normal_x):
        hl, hr = torch.clamp(L[0] - dl, min=0), torch.clamp(R[0] - dr, min=0)
        cl, cr = torch.where(dl > 0, _root(9.81 * hl), L[3]), torch.where(dr > 0, _root(9.81 * hr), R[3])
        ul, tl, ur, tr = (L[1], L[2], R[1], R[2]) if normal_x else (L[2], L[1], R[2], R[1])
        dry_l, dry_r = ~(hl > 0), ~(hr > 0)
        us, cs = 0.5 * (ul + ur) + cl - cr, 0.5 * (cl + cr) + 0.25 * (ul - ur)
        sl = torch.where(dry_l, ur - 2 * cr, torch.where(dry_r, ul - cl, torch.minimum(ul - cl, us - cs)))
        sr = torch.where(dry_l, ur + cr, torch.where(dry_r, ul + 2 * cl, torch.maximum(ur + cr, us + cs)))
        ml, mr, pl0, pr0 = hl * ul, hr * ur, 4.905 * hl * hl, 4.905 * hr * hr
        pl, pr = ml * ul + pl0, mr * ur + pr0
        none, left, right = dry_l & dry_r, sl >= 0, sr <= 0
        den = torch.where(none | left | right, torch.ones_like(sl), sr - sl)
        fm = torch.where(left, ml, torch.where(right, mr, (sr * ml - sl * mr + sl * sr * (hr - hl)) / den))
        fn = torch.where(left, pl, torch.where(right, pr, (sr * pl - sl * pr + sl * sr * (mr - ml)) / den))
        fm, fn = torch.where(none, 0.0, fm), torch.where(none, 0.0, fn)
        return fm, fn - pl0, fn - pr0, fm * torch.where(fm > 0, tl, tr)

    def step(self, state, cuts, dt, rain, q):
        """The state after one step, and its largest wave rate per design."""
        p, b = self.p, self.base
        nx, ny = b.nx, b.ny
        h, qx, qy = state
        W = self.ghost(h[:, :, 0], qx[:, :, 0], qy[:, :, 0], 2 * nx, 2 * nx + ny, True, 1.0, q)
        E = self.ghost(h[:, :, -1], qx[:, :, -1], qy[:, :, -1], 2 * nx + ny, 2 * nx + 2 * ny, True, -1.0, q)
        N = self.ghost(h[:, 0], qx[:, 0], qy[:, 0], 0, nx, False, 1.0, q)
        S = self.ghost(h[:, -1], qx[:, -1], qy[:, -1], nx, 2 * nx, False, -1.0, q)
        X = self.vel(*(torch.cat([w[..., None], a, e[..., None]], 2) for w, a, e in zip(W, (h, qx, qy), E)))
        Y = self.vel(*(torch.cat([u[:, None], a, d[:, None]], 1) for u, a, d in zip(N, (h, qx, qy), S)))
        fx = self.face([v[:, :, :-1] for v in X], [v[:, :, 1:] for v in X], cuts[0], cuts[1], True)
        fy = self.face([v[:, :-1] for v in Y], [v[:, 1:] for v in Y], cuts[2], cuts[3], False)
        dx, dy = (dt / b.dx)[:, None, None], (dt / b.dy)[:, None, None]
        w, e, u, d = [f[:, :, :-1] for f in fx], [f[:, :, 1:] for f in fx], [f[:, :-1] for f in fy], [f[:, 1:] for f in fy]
        h1 = torch.clamp(h - dx * (e[0] - w[0]) - dy * (d[0] - u[0]), min=0)
        x1 = qx - dx * (e[1] - w[2]) - dy * (d[3] - u[3])
        y1 = qy - dx * (e[3] - w[3]) - dy * (d[1] - u[2])
        h2 = h1 + rain[:, None, None] * self.wet
        h3 = h2 - torch.minimum(p.infil_capacity * dt[:, None, None] * self.wet, h2)
        dry = h3 < p.h_dry
        hs = torch.where(dry, torch.ones_like(h3), h3)
        keep = torch.where(dry, 0.0, 1.0) / (1 + dt[:, None, None] * self.gn2 * _root(x1 * x1 + y1 * y1) * hs ** (-7.0 / 3.0))
        x2, y2 = x1 * keep, y1 * keep
        c = _root(9.81 * h3)
        rate = ((x2.abs() / hs + c) / b.dx + (y2.abs() / hs + c) / b.dy).amax((1, 2))
        return torch.stack([h3, x2, y2]), rate

    def plan(self, dt_cfl, sync):
        p = self.p
        t_sync = torch.clamp((sync + 1) * p.sync_interval_s, max=p.duration_s)
        dt = torch.clamp(dt_cfl, max=p.dt_max_s)
        hits = self.t + dt >= t_sync - 1e-9 * p.sync_interval_s
        t_new = torch.where(hits, t_sync, self.t + dt)
        return t_new - self.t, t_new, hits

    def run(self, obj, baseline=None, tape=None, limit=12000):
        """Every design to its end, or to the sync point at which it breaches the guard. None beyond `limit` steps."""
        p, b = self.p, self.base
        s0 = torch.where(self.state[0] > p.h_dry, torch.sqrt(9.81 * self.state[0]) * (1 / b.dx + 1 / b.dy), 0.0).amax((1, 2))
        dt_cfl = torch.where(s0 > 0, p.cfl / torch.where(s0 > 0, s0, 1.0), p.dt_max_s)
        sync = torch.zeros(self.n, dtype=torch.float64, device=self.dev)
        peak = torch.zeros_like(self.state[0])
        alive = torch.full((self.n,), p.duration_s > 0, device=self.dev)
        mon = torch.from_numpy(obj.monitors.cells.astype(np.int64)).to(self.dev)
        guard = torch.tensor(obj.guard_pos, device=self.dev)
        arg = torch.zeros_like(peak, dtype=torch.int64) if tape is not None else None
        for k in range(limit):
            if k % 16 == 0 and not bool(alive.any()):
                break
            dt, t_new, hits = self.plan(dt_cfl, sync)
            dt = torch.where(alive, dt, 0.0)
            rain = torch.where(alive, self.rate_sum(self.t + dt) - self.rate_sum(self.t), 0.0)
            q = self.inflow() if b.has_inflow else None
            if tape is not None:
                tape.append((self.state, dt, rain, q))
            new, rate = self.step(self.state, self.cuts, dt, rain, q)
            live = alive[:, None, None]
            self.state = torch.where(live[None], new, self.state)
            if arg is not None:
                arg = torch.where(live & (self.state[0] > peak), k + 1, arg)
            peak = torch.where(live, torch.maximum(peak, self.state[0]), peak)
            self.t = torch.where(alive, t_new, self.t)
            dt_cfl = torch.where(rate > 0, p.cfl / torch.where(rate > 0, rate, 1.0), p.dt_max_s)
            sync = sync + (hits & alive)
            if baseline is not None:
                over = peak.flatten(1)[:, mon[guard]] - torch.from_numpy(np.asarray(baseline)).to(self.dev)[guard] - obj.d.guard_tolerance_m
                alive = alive & ~(hits & (over > 0).any(1))
            alive = alive & (self.t < p.duration_s)
        else:
            return None
        self.peak, self.arg = peak, arg
        mm = peak.flatten(1)[:, mon].cpu().numpy()
        return {"monitor_max": mm, "t_end": self.t.cpu().numpy(), "depth": self.state[0].cpu().numpy(), "peak": peak.cpu().numpy()}

    def gradient(self, obj, tape, mm, mode):
        """dJ/d(face jump), time steps held as they were taken: one step back at a time through torch's own derivative."""
        lam = torch.zeros_like(self.state)
        gx, gy = torch.zeros_like(self.cuts[0]), torch.zeros_like(self.cuts[2])
        seeds = []
        for a, pos in zip(obj.d.assets, obj.asset_pos):
            best = mm[:, pos].argmax(1)
            for d in range(self.n):
                cell, x = int(obj.monitors.cells[pos[best[d]]]), (mm[d, pos[best[d]]] - a.threshold_m) / obj.d.tau_m
                r, c = divmod(cell, self.base.nx)
                seeds.append((int(self.arg[d, r, c]), d, r, c, a.weight / (1 + math.exp(-x))))
        for k in range(len(tape) - 1, -1, -1):
            state, dt, rain, q = tape[k]
            for at, d, r, c, w in seeds:
                if at == k + 1:
                    lam[0, d, r, c] += w
            with torch.enable_grad():
                x = state.detach().requires_grad_(True)
                cuts = [c.detach().requires_grad_(True) for c in self.cuts]
                new, _ = self.step(x, cuts, dt, rain, q)
                lam, *g = torch.autograd.grad(new, [x] + cuts, lam)
            s = [(c > 0).double() for c in self.cuts]
            gx += g[0] * s[0] - g[1] * s[1]
            gy += g[2] * s[2] - g[3] * s[3]
        return gx.cpu().numpy(), gy.cpu().numpy()


def _exact_group(base, obj, params, terrains, baseline=None, gradient=False):
    e = _Exact(base, params, terrains)
    tape = [] if gradient else None
    with torch.no_grad():
        out = e.run(obj, baseline, tape)
    if out is None:
        return None
    d = obj.d
    j = []
    for k, t in enumerate(terrains):
        s = d.earth_weight * (d.cut_cost * t.cut_m3 + d.fill_cost * t.fill_m3)
        for a, pos in zip(d.assets, obj.asset_pos):
            x = (max(0.0, *out["monitor_max"][k, pos]) - a.threshold_m) / d.tau_m
            s += a.weight * d.tau_m * (max(x, 0.0) + math.log1p(math.exp(-abs(x))))
        j.append(s)
    out.update(j=np.array(j), steps=None, status=None, feasible=None)
    if gradient:
        out["dj_ddzx"], out["dj_ddzy"] = e.gradient(obj, tape, out["monitor_max"], base.mode)
    return out


def exact(case, seed):
    cost = work(case)["flops"] / (FLOPS_STEP + (FLOPS_ADJOINT if "vjp" in case["call"] else 0))   # cells times steps
    if cost > 4e9 or _steps(case) * (3.0 if "vjp" in case["call"] else 1.0) * (3.0 if case["call"] == "ladder" else 1.0) > 9000:
        return None
    s = prepare(case, seed)
    if case["call"] == "ladder":
        got = [_exact_group(g["terrains"][0].base, g["objective"], s["params"], g["terrains"], g.get("baseline_max")) for g in s["groups"]]
        for g in got:
            if g is None:
                return None
            g.update(depth=[], peak=[])
        return got
    if "prims" in s:
        s["terrains"] = [_prepared(s["base"], _dz(p, case, s["editable"])) for p in s["prims"]]
    base = s["terrains"][0].base
    out = _exact_group(base, s["objective"], s["params"], s["terrains"], s.get("baseline_max"), "vjp" in case["call"])
    if out is None:
        return None
    if case["call"] == "primitives":
        out.update(depth=[], peak=[], cut=np.array([t.cut_m3 for t in s["terrains"]]), fill=np.array([t.fill_m3 for t in s["terrains"]]))
    elif "vjp" in case["call"]:
        out["peak"] = []
    return out
