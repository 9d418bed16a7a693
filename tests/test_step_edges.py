"""The step kernels where their layouts and their branch-free arithmetic have edges, bit for bit
against the f32 oracle.

Sizes: the cluster kernel's windows hold 60 columns (30 pairs) and its strips split the rows over
CTAs; the row-band kernel's segments hold 64 columns and its bands at most 32 rows. Widths and
heights on both sides of those lines, odd and even (pairs aligned or not), down to one row or
column (one column runs on the tiled path, also where a cluster shape is asked for).

Arithmetic: parameters and states outside the bounds of the branch-free square roots and
reciprocals (tiny h_eps, a huge roughness, a long dt_max, crest jumps below 0, a thin stage
ghost, water so deep that the bound on the wave rate is passed and left again) take the scalar
operations: the same bits with and without option exact_special, which forces those.
"""
from __future__ import annotations

import math

import numpy as np
import pytest

import oracle_ref as orc
from helpers import base_arrays, design_dict
from itr_gpu import GpuSolver, Hyetograph, MonitorSet, PreparedTerrain, Segment, SolverParams, UnsupportedError, synthetic_terrain
from test_gpu_parity import compare_run

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    g = GpuSolver()
    yield g
    g.close()


def scene(nx, ny, bnd):
    dx = 2.0
    segs = [Segment("transmissive", "east")]
    if bnd:
        segs = [Segment("inflow", "west", hydrograph=[(0.0, 0.02), (30.0, 0.1)]), Segment("stage", "east", stage_m=3.15),
                Segment("inflow", "north", (0.0, 0.5 * nx * dx), hydrograph=[(0.0, 0.01), (30.0, 0.05)])]
    base = synthetic_terrain(nx, ny, dx, lambda x, y: 3.0 + 0.02 * math.sin(x / 5.0) * math.cos(y / 7.0),
                             lambda c, r: nx > 8 and ny > 8 and (c + 3 * r) % 41 == 17, n=0.035, segments=segs)
    p = SolverParams(24.0, 8.0, rain=Hyetograph.from_mm_h([(0, 0), (5, 300), (15, 0)]), infil_capacity=2e-6, initial_depth=0.12)
    return base, p


def check(gpu, base, p, terrs, what):
    mon = MonitorSet(np.arange(0, base.nx * base.ny, 5))
    runs = gpu.run_batch(p, terrs, mon, want_peak=True)
    for i, t in enumerate(terrs):
        o = orc.flat_run(base_arrays(base), design_dict(t, p), p, mon, want_peak=True, bnd=orc.bnd_dict(base, t))
        compare_run(runs[i], o, f"{what} design {i}")
    return runs


def with_options(gpu, opts, f):
    try:
        for k, v in opts.items():
            gpu.set_option(k, v)
        return f()
    finally:
        for k in opts:
            gpu.set_option(k, 0)


SIZES = [(2, 2), (3, 1), (1, 9), (4, 37), (59, 5), (60, 8), (61, 33), (62, 16), (119, 7), (120, 12), (121, 40), (181, 3)]


@pytest.mark.parametrize("bnd", [False, True])
@pytest.mark.parametrize("nx,ny", SIZES)
def test_cluster_kernel_edges(gpu, nx, ny, bnd):
    base, p = scene(nx, ny, bnd)
    terrs = [PreparedTerrain(base), PreparedTerrain(base)]
    check(gpu, base, p, terrs, f"{nx}x{ny} chosen shape")
    for cluster, threads in [(1, 64), (2, 128), (8, 256), (1, 384), (1, 576)]:
        if ny >= cluster and threads >= 32 * ((nx + 64) // 64):   # (else refused, below)
            with_options(gpu, {"cluster": cluster, "threads": threads},
                         lambda: check(gpu, base, p, terrs[:1], f"{nx}x{ny} {cluster} x {threads}"))


@pytest.mark.parametrize("nx,ny,n", [(250, 230, 1), (250, 230, 3), (249, 221, 2), (240, 192, 2)])
def test_either_side_of_the_path_rule(gpu, nx, ny, n):
    """Grids whose strips are too tall for the cluster kernel take the tiled path, shorter ones do not: the same bits."""
    base, p = scene(nx, ny, n == 3)
    p.duration_s, p.sync_interval_s = 4.0, 2.0
    check(gpu, base, p, [PreparedTerrain(base)] * n, f"{nx}x{ny} x{n}")


def test_refused_shapes(gpu):
    """Cluster shapes are taken and refused by the same lines, whatever layout the kernel has: fewer rows
    than CTAs, fewer threads than one strip, more cells than the shared memory."""
    for nx, ny, cluster, threads in [(20, 3, 4, 64), (64, 9, 1, 32), (300, 200, 1, 512), (1100, 8, 1, 512)]:
        base, p = scene(nx, ny, False)
        with pytest.raises(UnsupportedError):
            with_options(gpu, {"cluster": cluster, "threads": threads}, lambda: gpu.run_batch(p, [PreparedTerrain(base)], MonitorSet()))


@pytest.mark.parametrize("bnd", [False, True])
@pytest.mark.parametrize("nx,ny", [(1, 9), (2, 2), (3, 1), (63, 31), (64, 32), (65, 33), (127, 6), (128, 64), (129, 34), (257, 65)])
def test_row_band_kernel_edges(gpu, nx, ny, bnd):
    base, p = scene(nx, ny, bnd)
    with_options(gpu, {"impl": 2}, lambda: check(gpu, base, p, [PreparedTerrain(base), PreparedTerrain(base)], f"{nx}x{ny} tiled"))


def form(name):
    base, p = scene(26, 22, False)
    p.duration_s, p.sync_interval_s = 16.0, 4.0
    p.infil_capacity = 0.0
    t = None
    if name == "tiny h_eps":
        p.h_eps = 1e-15
    elif name == "long dt_max":
        p.dt_max_s = 1e5
    elif name == "rough":
        base = synthetic_terrain(26, 22, 2.0, lambda x, y: 3.0 - 0.004 * x, n=20.0, segments=[Segment("transmissive", "east")])
    elif name == "thin stage":
        base = synthetic_terrain(26, 22, 2.0, lambda x, y: 3.0, n=0.03, segments=[Segment("stage", "east", stage_m=3.000002)])
    elif name == "deep":
        p.initial_depth = 50000.0   # celerity 700 m/s, past the bound; it drains below it through the east edge
        p.duration_s, p.sync_interval_s = 0.5, 0.1
    elif name == "crest below 0":
        from itr_gpu.scenes import valley_scene
        from itr_gpu.terrain import TerrainBase
        base = TerrainBase(valley_scene(5.0).base.fine, 2, [Segment("transmissive", "east")])
        t = PreparedTerrain(base)
        t.dzx2 = t.dzx2.copy()
        t.dzx2[t.dzx2 == 0.0] = -1e-3
    return base, p, t if t is not None else PreparedTerrain(base)


@pytest.mark.parametrize("impl", [0, 2])
@pytest.mark.parametrize("name", ["plain", "tiny h_eps", "long dt_max", "rough", "thin stage", "deep", "crest below 0"])
def test_scalar_operations_outside_the_bounds(gpu, name, impl):
    base, p, t = form(name)
    for exact in (0, 1):
        with_options(gpu, {"impl": impl, "exact_special": exact}, lambda: check(gpu, base, p, [t], f"{name} impl {impl} exact {exact}"))


def test_more_designs_than_a_grid_extent(gpu):
    """65535 is the extent of a launch's y and z: the cluster path takes more designs than that."""
    base, p = scene(3, 2, False)
    t, n = PreparedTerrain(base), 65535 + 3
    runs = gpu.run_batch(p, [t] * n, MonitorSet(np.arange(2)))
    o = orc.flat_run(base_arrays(base), design_dict(t, p), p, MonitorSet(np.arange(2)))
    for i in (0, 1, 65534, 65535, n - 1):
        compare_run(runs[i], o, f"design {i}")
