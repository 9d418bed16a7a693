"""Calls at the limits of the kernels' synchronisation, operand ranges and dispatch.

The forward is compared bit for bit with the f32 oracle; gradients are compared bit for bit
between kernels that evaluate the same arithmetic.
"""
from __future__ import annotations

import math

import numpy as np
import pytest

import oracle_ref as orc
from helpers import base_arrays, design_dict
from itr_gpu import GpuSolver, Hyetograph, MonitorSet, PreparedTerrain, Segment, SolverParams, synthetic_terrain
from test_gpu_parity import compare_run

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    g = GpuSolver()
    yield g
    g.close()


def with_options(gpu, opts, f, defaults=None):
    try:
        for k, v in opts.items():
            gpu.set_option(k, v)
        return f()
    finally:
        for k in opts:
            gpu.set_option(k, (defaults or {}).get(k, 0))


def check(gpu, base, p, terrs, what):
    mon = MonitorSet(np.arange(0, base.nx * base.ny, 5))
    runs = gpu.run_batch(p, terrs, mon, want_peak=True)
    for i, t in enumerate(terrs):
        o = orc.flat_run(base_arrays(base), design_dict(t, p), p, mon, want_peak=True, bnd=orc.bnd_dict(base, t))
        compare_run(runs[i], o, f"{what} design {i}")
    return runs


@pytest.mark.parametrize("nx,ny,cluster", [(959, 8, 0), (959, 8, 8), (480, 3, 0), (480, 3, 1), (479, 2, 2), (240, 1, 1)])
def test_low_wide_grids_with_flowing_edges(gpu, nx, ny, cluster):
    """Strips of one row beside north and south edges that flow: one warp sums the edges' fluxes after a
    step's barrier while the others are already through the next step's row. Few sync points, whose
    barriers would hold them together."""
    dx = 2.0
    segs = [Segment("transmissive", "south"), Segment("transmissive", "east"),
            Segment("inflow", "north", (0.0, 0.6 * nx * dx), hydrograph=[(0.0, 0.5), (30.0, 2.0)])]
    base = synthetic_terrain(nx, ny, dx, lambda x, y: 3.0 + 0.02 * math.sin(x / 5.0) - 0.01 * y, n=0.035, segments=segs)
    p = SolverParams(40.0, 20.0, rain=Hyetograph.from_mm_h([(0, 300), (20, 100)]), initial_depth=0.12)
    terrs = [PreparedTerrain(base)] * 2
    with_options(gpu, {"cluster": cluster, "threads": 512 if cluster else 0}, lambda: check(gpu, base, p, terrs, f"{nx}x{ny} cluster {cluster}"))


@pytest.mark.parametrize("name", ["smooth", "stage_inflow", "crest"])
def test_gradients_after_a_tiled_forward_on_16x16_tiles(gpu, name):
    """Option band = 0 (the forward on 16x16 tiles) with the replay and the backward step on row bands or tiles:
    the row-band replay needs its packed inputs whatever kernel ran the forward."""
    from test_adjoint_band import CASES
    p, terrains, obj, K = CASES[name](gpu)
    grad = lambda: gpu.vjp(p, terrains, obj.monitors, obj, checkpoint_interval=K)
    want = grad()
    for ab in (-1, 3, 1, 0):
        got = with_options(gpu, {"band": 0, "adj_band": ab}, grad, {"band": 1, "adj_band": -1})
        for i, (a, b) in enumerate(zip(got, want)):
            assert a.steps == b.steps and a.j == b.j, (name, ab, i)
            for f in ("dj_ddzx", "dj_ddzy", "dj_ddzx2", "dj_ddzy2"):
                ga, gb = getattr(a, f, None), getattr(b, f, None)
                assert (ga is None) == (gb is None)
                if ga is not None:
                    assert np.array_equal(np.asarray(ga).view(np.uint64), np.asarray(gb).view(np.uint64)), (name, ab, i, f)
