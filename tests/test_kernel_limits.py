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


def gradients_agree(a, b, what):
    """Bit for bit but for quotients below the normal range (2^-149 each, through the sweep's linear factors)."""
    nonzero = 0
    for i, (x, y) in enumerate(zip(a, b)):
        for f in ("dj_ddzx", "dj_ddzy", "dj_ddzx2", "dj_ddzy2"):
            gx, gy = getattr(x, f, None), getattr(y, f, None)
            assert (gx is None) == (gy is None)
            if gx is None:
                continue
            gx, gy = np.asarray(gx), np.asarray(gy)
            assert np.all(np.isfinite(gx)) and np.all(np.isfinite(gy)), (what, i, f, int(np.count_nonzero(~np.isfinite(gx))))
            assert np.all(np.abs(gx - gy) <= 1e-30), (what, i, f, float(np.max(np.abs(gx - gy))))
            nonzero += int(np.count_nonzero(gx))
    assert nonzero > 0, what


def half_dry(level):
    """A slope that a stage covers in part: beyond the shore lies a film far below h_eps (a drizzle of 1e-13 m/s; the
    adjoint of a cell without any water ends at the infiltration's minimum). Water runs in, so that the
    assets' peaks come late and the backward sweep covers most steps."""
    from itr_gpu import Asset, Objective, ObjectiveDef
    nx, ny = 70 * level, 45 * level
    base = synthetic_terrain(nx, ny, 5.0 / level, lambda x, y: 2.0 - 0.004 * x + 0.2 * math.sin(y / 15.0) + 0.1 * math.cos(x / 20.0), n=0.03,
                             segments=[Segment("inflow", "north", (200.0, 320.0), hydrograph=[(0.0, 0.1), (40.0, 0.5)])], level=level)
    p = SolverParams(40.0, 10.0, rain=Hyetograph([(0.0, 1e-13), (40.0, 1e-13)]), initial_depth=0.0, initial_stage=1.6)
    t = PreparedTerrain(base)
    h0 = t.initial_depth(0.0, 1.6).ravel()
    assert 0.2 < np.mean(h0 == 0.0) < 0.8
    wet = np.flatnonzero(h0 > 0.05)
    cells = [int(wet[len(wet) // 4]), int(wet[len(wet) // 2]), int(wet[3 * len(wet) // 4])]
    return p, [t], Objective(ObjectiveDef([Asset(f"a{i}", [c], float(h0[c]), 1.0 + i) for i, c in enumerate(cells)], []))


@pytest.mark.parametrize("h_eps", [1e-5, 1e-9, 1e-10, 1e-11, 1e-14])
@pytest.mark.parametrize("level", [1, 2])
def test_backward_step_over_small_h_eps(gpu, level, h_eps):
    """The velocity map's derivative divides by h_eps^4 and more in shallow and dry cells, below the range of the
    branch-free reciprocal from h_eps = 2^-31 down: the gradients are those of the scalar operations."""
    p, terrains, obj = half_dry(level)
    p.h_eps = h_eps
    grad = lambda: gpu.vjp(p, terrains, obj.monitors, obj, checkpoint_interval=24)
    for ab in (0, 1, 3):
        want = with_options(gpu, {"adj_band": ab, "exact_special": 1}, grad, {"adj_band": -1})
        got = with_options(gpu, {"adj_band": ab}, grad, {"adj_band": -1})
        gradients_agree(got, want, f"level {level} h_eps {h_eps} adj_band {ab}")


@pytest.mark.parametrize("nx", [24, 29, 30, 57])
@pytest.mark.parametrize("level", [1, 2])
def test_gradient_of_the_east_edge(gpu, level, nx):
    """The jumps of the domain's east face, whichever lane of the row-band backward step comes upon it (a warp owns
    29 columns): the same as the 16x16 tiles'."""
    from itr_gpu import Asset, Objective, ObjectiveDef
    ny = 16
    base = synthetic_terrain(nx * level, ny * level, 5.0 / level, lambda x, y: 2.0 - 0.004 * x + 0.1 * math.sin(y / 15.0), n=0.03,
                             segments=[Segment("transmissive", "east")], level=level)
    t = PreparedTerrain(base)
    t.dzx = t.dzx.copy()
    t.dzx.reshape(ny, nx + 1)[:, nx] = 0.02   # a step up at the outlet
    p = SolverParams(60.0, 20.0, rain=Hyetograph.from_mm_h([(0, 50), (60, 200)]), initial_depth=0.3)
    cells = [3 * nx + nx - 2, 9 * nx + nx // 2, 12 * nx + nx - 1]
    obj = Objective(ObjectiveDef([Asset(f"a{i}", [c], 0.3, 1.0 + i) for i, c in enumerate(cells)], []))
    grad = lambda: gpu.vjp(p, [t], obj.monitors, obj, checkpoint_interval=16)
    want = with_options(gpu, {"adj_band": 0}, grad, {"adj_band": -1})[0]
    assert np.count_nonzero(np.asarray(want.dj_ddzx).reshape(ny, nx + 1)[:, nx]) > 0
    got = with_options(gpu, {"adj_band": 3}, grad, {"adj_band": -1})[0]
    for f in ("dj_ddzx", "dj_ddzy", "dj_ddzx2", "dj_ddzy2"):
        ga, gb = getattr(got, f, None), getattr(want, f, None)
        assert (ga is None) == (gb is None)
        if ga is not None:
            assert np.array_equal(np.asarray(ga).view(np.uint64), np.asarray(gb).view(np.uint64)), (f, float(np.max(np.abs(ga - gb))))


RAIN = {"to infinity": [(0.0, 5e-5), (math.inf, 5e-5)], "steps": [(2.0, 0.0), (2.0, 4e-5), (9.0, 4e-5), (9.0, 1e-5)],
        "vanishing": [(0.0, 0.0), (8.0, 1e-310), (16.0, 1e-310)], "far off": [(-1e300, 3e-5), (0.0, 3e-5), (1e300, 3e-5)]}


@pytest.mark.parametrize("impl", [0, 1, 2])
@pytest.mark.parametrize("name", list(RAIN))
def test_storms_at_the_ends_of_the_number_range(gpu, name, impl):
    """Breakpoints at infinity or at one instant, vanishing rates: the storm by its general integral where the
    piecewise one leaves its range, bit for bit the oracle's."""
    base = synthetic_terrain(26, 22, 2.0, lambda x, y: 3.0 - 0.01 * x + 0.02 * math.sin(y / 5.0), n=0.03, segments=[Segment("transmissive", "east")])
    p = SolverParams(16.0, 4.0, rain=Hyetograph(RAIN[name]), initial_depth=0.05)
    with_options(gpu, {"impl": impl}, lambda: check(gpu, base, p, [PreparedTerrain(base)], f"{name} impl {impl}"))


def test_launch_shape_follows_option_band():
    """The kernel of a batch follows from its sizes and the options, not from the calls before it: a grid that takes the
    row bands, on solvers that had option band at 0 or 1 before."""
    base = synthetic_terrain(250, 230, 5.0, lambda x, y: 5.0 + 0.01 * x + 0.1 * math.sin(y / 9.0), n=0.03, segments=[Segment("transmissive", "west")])
    p = SolverParams(20.0, 10.0, rain=Hyetograph.from_mm_h([(0, 100)]), initial_depth=0.05)
    terrs, mon = [PreparedTerrain(base)] * 4, MonitorSet(np.arange(0, 250 * 230, 991))

    def run(bands):
        g = GpuSolver()
        try:
            for b in bands:
                g.set_option("band", b)
                r = g.run_batch(p, terrs, mon, ledger_rows=4)[0]
            return g.adapter_info().split("last batch:")[1], r
        finally:
            g.close()

    for bands in ((0,), (1,)):
        want, a = run(bands)
        got, b = run((1 - bands[0],) + bands)
        assert got == want and ("row bands" in want) == (bands == (1,))
        np.testing.assert_array_equal(a.ledger, b.ledger)


@pytest.mark.parametrize("nx,ny", [(161, 133), (40, 300), (1, 40)])
def test_dry_rows_beside_edges_that_come_alive(gpu, nx, ny):
    """The row bands' dry-row test on grids with more edge cells than a block has threads, an inflow that starts
    late and a stage on every side but one: the oracle's rows skipped, and its bits."""
    dx = 2.0
    segs = [Segment("inflow", "north", (0.3 * nx * dx, 0.8 * nx * dx), hydrograph=[(0.0, 0.0), (6.0, 0.0), (7.0, 1.5)]),
            Segment("stage", "south", (0.0, 0.5 * nx * dx), stage_m=0.6), Segment("stage", "east", (0.6 * ny * dx, 0.9 * ny * dx), stage_m=0.02 * ny + 0.2),
            Segment("inflow", "west", (0.1 * ny * dx, 0.3 * ny * dx), hydrograph=[(0.0, 0.0), (12.0, 0.0), (13.0, 0.5)])]
    base = synthetic_terrain(nx, ny, dx, lambda x, y: 0.02 * y + 0.1 * math.sin(x / 7.0) + 0.1, n=0.03, segments=segs)
    p = SolverParams(20.0, 5.0, dt_max_s=0.1, rain=Hyetograph([]), initial_depth=0.0)
    t, mon = PreparedTerrain(base), MonitorSet(np.arange(0, nx * ny, 5))
    o = orc.flat_run(base_arrays(base), design_dict(t, p), p, mon, want_peak=True, bnd=orc.bnd_dict(base, t))
    assert o["rows_skipped"] > 0
    r = with_options(gpu, {"impl": 2}, lambda: gpu.run_batch(p, [t, t], mon, want_peak=True))
    for i in range(2):
        compare_run(r[i], o, f"{nx}x{ny} design {i}")
        assert r[i].rows_skipped == o["rows_skipped"]


@pytest.mark.parametrize("nx,ny", [(16, 16), (512, 16), (528, 16), (256, 256), (4112, 16), (500, 400)])
def test_tile_partials_of_many_blocks(gpu, nx, ny):
    """The step's sums over the 16x16 tiles' partials, block counts around 32 and 256: the oracle's bits, and the
    ledgers of the row bands (f64 sums of the same terms in another order)."""
    base = synthetic_terrain(nx, ny, 2.0, lambda x, y: 3.0 + 0.02 * math.sin(x / 5.0) - 0.001 * y, n=0.035,
                             segments=[Segment("transmissive", "south"), Segment("inflow", "north", (0.0, nx), hydrograph=[(0.0, 0.5), (4.0, 1.0)])])
    p = SolverParams(4.0, 2.0, rain=Hyetograph.from_mm_h([(0, 300), (4, 100)]), initial_depth=0.12, infil_capacity=1e-5)
    t, mon = PreparedTerrain(base), MonitorSet(np.arange(0, nx * ny, 5))
    o = orc.flat_run(base_arrays(base), design_dict(t, p), p, mon, want_peak=True, bnd=orc.bnd_dict(base, t))
    go = lambda: gpu.run_batch(p, [t], mon, want_peak=True, ledger_rows=4)
    ref = with_options(gpu, {"impl": 2}, go)[0]
    for opts in ({"impl": 1}, {"impl": 2, "band": 0}):
        r = with_options(gpu, opts, go, {"band": 1})[0]
        compare_run(r, o, f"{nx}x{ny} {opts}")
        np.testing.assert_allclose(r.ledger, ref.ledger, rtol=1e-12, atol=1e-9)


@pytest.mark.parametrize("rain", [True, False])
@pytest.mark.parametrize("level", [1, 2])
@pytest.mark.parametrize("ny,cluster", [(1, 1), (9, 0), (9, 8), (40, 2), (300, 0), (301, 8)])
def test_single_column_on_the_cluster_kernel(gpu, ny, cluster, level, rain):
    """One column: its west and east faces, both flowing, belong to one lane. The oracle's bits, and the ledger's
    inflow and outflow as on the tiled path."""
    dx = 2.0
    segs = [Segment("inflow", "west", hydrograph=[(0.0, 0.02), (30.0, 0.1)]), Segment("transmissive", "east"), Segment("transmissive", "south")]
    base = synthetic_terrain(level, ny * level, dx / level, lambda x, y: 3.0 + 0.02 * math.cos(y / 7.0) - 0.01 * x, n=0.035, segments=segs, level=level)
    assert base.nx == 1
    p = SolverParams(24.0, 8.0, rain=Hyetograph.from_mm_h([(0, 0), (5, 300), (15, 0)] if rain else []), infil_capacity=2e-6, initial_depth=0.12 if rain else 0.0)
    terrs, mon = [PreparedTerrain(base)] * 3, MonitorSet(np.arange(0, ny, 2))
    ref = with_options(gpu, {"impl": 2}, lambda: gpu.run_batch(p, terrs, mon, ledger_rows=4))
    o = orc.flat_run(base_arrays(base), design_dict(terrs[0], p), p, mon, want_peak=True, bnd=orc.bnd_dict(base, terrs[0]))

    def run():
        r = gpu.run_batch(p, terrs, mon, want_peak=True, ledger_rows=4)
        assert "cluster kernel" in gpu.adapter_info()
        return r

    for r, a in zip(with_options(gpu, {"cluster": cluster, "threads": 128 if cluster else 0}, run), ref):
        compare_run(r, o, f"1x{ny} cluster {cluster}")
        assert r.rows_skipped == a.rows_skipped
        # (time, volume, rain, inflow, outflow: f64 sums; the infiltration of a step is summed in f32, in another order)
        np.testing.assert_allclose(r.ledger[:, :5], a.ledger[:, :5], rtol=1e-12, atol=1e-12)
        assert np.all(r.ledger[:, 3:5] > 0.0)


@pytest.mark.parametrize("level", [1, 2])
@pytest.mark.parametrize("nx,ny,n", [(16, 16, 1), (17, 15, 5), (16, 16, 444), (16, 16, 445), (300, 33, 2)])
def test_tiles_that_advance_the_integrator(gpu, nx, ny, n, level):
    """One launch a step on 16x16 tiles (up to 444 of them) and two (above): the oracle's bits, the row bands' ledgers."""
    dx = 2.0
    segs = [Segment("inflow", "west", (0.0, 0.6 * ny * dx), hydrograph=[(0.0, 0.02), (12.0, 0.1)]), Segment("stage", "east", stage_m=3.15),
            Segment("transmissive", "south")]
    base = synthetic_terrain(nx * level, ny * level, dx / level, lambda x, y: 3.0 + 0.02 * math.sin(x / 5.0) * math.cos(y / 7.0), n=0.035, segments=segs, level=level)
    p = SolverParams(12.0, 4.0, rain=Hyetograph.from_mm_h([(0, 100), (5, 300), (12, 50)]), infil_capacity=2e-6, initial_depth=0.12)
    mon = MonitorSet(np.arange(0, nx * ny, 5))
    terrs = []
    for i in range(n):
        t = PreparedTerrain(base)
        t.dzx = t.dzx.copy()
        t.dzx.flat[(7 * i + 3) % t.dzx.size] += np.float32(0.01 * (i + 1) / n)
        terrs.append(t)
    go = lambda: gpu.run_batch(p, terrs, mon, want_peak=True, ledger_rows=4)
    got = with_options(gpu, {"impl": 2, "band": 0}, go, {"band": 1})
    ref = with_options(gpu, {"impl": 2}, go)
    for i, (a, b) in enumerate(zip(got, ref)):
        assert a.steps == b.steps and np.array_equal(a.depth, b.depth) and np.array_equal(a.peak, b.peak)
        np.testing.assert_allclose(a.ledger[:, :5], b.ledger[:, :5], rtol=1e-12, atol=1e-12)
        if i % 89 == 0:
            o = orc.flat_run(base_arrays(base), design_dict(terrs[i], p), p, mon, want_peak=True, bnd=orc.bnd_dict(base, terrs[i]))
            compare_run(a, o, f"{nx}x{ny} design {i}")


def test_aborts_on_tiles_that_advance_the_integrator(gpu):
    from test_gpu_parity import small_valley
    sc = small_valley(1200.0)
    terrs = [t for _, _, t in sc.designs(6)]
    baseline = gpu.run_batch(sc.params, [PreparedTerrain(sc.base)], sc.monitors)[0].monitor_max
    sc.objective.d.guard_tolerance_m = 0.0005
    inc = sorted(r.j for r in gpu.run_batch(sc.params, terrs, sc.monitors, objective=sc.objective))[2]
    statuses = set()
    for kw in (dict(guard_abort=True), dict(incumbent=inc), dict(guard_abort=True, incumbent=inc)):
        go = lambda: gpu.run_batch(sc.params, terrs, sc.monitors, objective=sc.objective, baseline_max=baseline, **kw)
        want, got = go(), with_options(gpu, {"impl": 2, "band": 0}, go, {"band": 1})
        statuses |= {r.status for r in want}
        for a, b in zip(got, want):
            assert (a.status, a.steps, a.t_end, a.breach_cell, a.breach_sync, a.violation, a.lower_bound) == \
                   (b.status, b.steps, b.t_end, b.breach_cell, b.breach_sync, b.violation, b.lower_bound)
            assert np.array_equal(a.depth, b.depth)
    assert len(statuses) > 1


@pytest.mark.parametrize("nx,ny,n,rain,where", [(300, 180, 1, 60, "16x16 tiles"), (300, 180, 1, 0, "16x16 tiles"), (60, 900, 1, 60, "16x16 tiles"),
                                                (900, 40, 2, 60, "16x16 tiles"), (180, 140, 1, 60, "cluster"), (250, 230, 16, 60, "row bands"),
                                                (1000, 8, 4, 60, "16x16 tiles|cluster")])
def test_few_designs_of_large_grids(gpu, nx, ny, n, rain, where):
    """The kernel that the rule on sizes takes, and the oracle's bits there, with locked dt too."""
    base = synthetic_terrain(nx, ny, 5.0, lambda x, y: 5.0 + 0.01 * x + 0.1 * math.sin(y / 9.0), n=0.03, segments=[Segment("transmissive", "west")])
    p = SolverParams(20.0, 10.0, rain=Hyetograph.from_mm_h([(0, rain), (20, rain)]), initial_depth=0.05)
    terrs, mon = [PreparedTerrain(base)] * n, MonitorSet(np.arange(0, nx * ny, 97))
    r = gpu.run_batch(p, terrs, mon, want_peak=True)
    assert any(w in gpu.adapter_info() for w in where.split("|")), gpu.adapter_info()
    o = orc.flat_run(base_arrays(base), design_dict(terrs[0], p), p, mon, want_peak=True, bnd=orc.bnd_dict(base, terrs[0]))
    for i in range(n):
        compare_run(r[i], o, f"{nx}x{ny} design {i}")
        assert r[i].rows_skipped == o["rows_skipped"]
    p.locked_dt = np.full(1000, 0.3)   # kept, or refused where it breaks the limit: the same on every path
    lock = gpu.run_batch(p, terrs, mon)
    ref = with_options(gpu, {"impl": 2}, lambda: gpu.run_batch(p, terrs, mon))
    for a, b in zip(lock, ref):
        assert a.steps == b.steps and np.array_equal(a.depth, b.depth)


@pytest.mark.parametrize("nx,ny,level,cluster", [(961, 4, 1, 0), (1000, 8, 2, 0), (1020, 3, 1, 2), (1021, 5, 2, 2), (1100, 1, 1, 1), (1439, 9, 1, 8), (1440, 8, 1, 4), (1441, 4, 1, 0)])
@pytest.mark.parametrize("rain", [True, False])
def test_blocks_above_512_threads(gpu, nx, ny, level, cluster, rain):
    """Grids of 17 to 24 windows on the cluster kernel, widths on both sides of a window; 25 windows on the tiled path."""
    dx = 2.0
    segs = [Segment("inflow", "west", hydrograph=[(0.0, 0.02), (30.0, 0.1)]), Segment("stage", "east", stage_m=3.1),
            Segment("inflow", "north", (0.3 * nx * dx, 0.7 * nx * dx), hydrograph=[(0.0, 0.01), (3.0, 0.3)])]
    base = synthetic_terrain(nx * level, ny * level, dx / level, lambda x, y: 3.0 + 0.02 * math.sin(x / 5.0) - 0.01 * y, n=0.035, segments=segs, level=level)
    p = SolverParams(8.0, 4.0, dt_max_s=0.2, rain=Hyetograph.from_mm_h([(0, 100), (5, 300), (8, 50)] if rain else []), infil_capacity=2e-6,
                     initial_depth=0.12 if rain else 0.0)
    terrs, mon = [PreparedTerrain(base)] * 2, MonitorSet(np.arange(0, nx * ny, 5))
    o = orc.flat_run(base_arrays(base), design_dict(terrs[0], p), p, mon, want_peak=True, bnd=orc.bnd_dict(base, terrs[0]))

    def run():
        r = gpu.run_batch(p, terrs, mon, want_peak=True)
        assert ("cluster kernel" if nx <= 1440 else "tiled path") in gpu.adapter_info()
        return r

    opts = {"cluster": cluster, "threads": 768 if cluster else 0}
    for r in with_options(gpu, opts, run):
        compare_run(r, o, f"{nx}x{ny} cluster {cluster}")
    p.locked_dt = np.full(1000, 0.05)
    ref = with_options(gpu, {"impl": 2}, lambda: gpu.run_batch(p, terrs, mon))
    for a, b in zip(with_options(gpu, opts, run), ref):
        assert a.steps == b.steps and np.array_equal(a.depth, b.depth)


@pytest.mark.parametrize("impl", [0, 2])
def test_dry_rows_of_steps_taken_back(gpu, impl):
    """A locked run that returns to its last snapshot takes back the count of dry rows with the steps."""
    nx, ny, dx = 60, 50, 2.0
    segs = [Segment("inflow", "north", (0.3 * nx * dx, 0.8 * nx * dx), hydrograph=[(0.0, 0.0), (3.0, 0.0), (4.0, 1.5)]),
            Segment("stage", "south", (0.0, 0.5 * nx * dx), stage_m=0.6)]
    base = synthetic_terrain(nx, ny, dx, lambda x, y: 0.02 * y + 0.1 * math.sin(x / 7.0) + 0.1, n=0.03, segments=segs)
    p = SolverParams(10.0, 5.0, dt_max_s=0.1, rain=Hyetograph([]), initial_depth=0.0)
    t, mon = PreparedTerrain(base), MonitorSet(np.arange(0, nx * ny, 5))
    p.locked_dt = np.full(60, 0.1)
    o = orc.locked(lambda: orc.flat_run(base_arrays(base), design_dict(t, p), p, mon, want_peak=True, bnd=orc.bnd_dict(base, t)),
                   p.locked_dt, p.cfl_hard)
    back = o["dt_fallback_t"]
    assert back > 0.0 and o["rows_skipped"] > 0
    r = with_options(gpu, {"impl": impl}, lambda: gpu.run_batch(p, [t, t], mon, want_peak=True))
    for a in r:
        compare_run(a, o, f"impl {impl}")
        assert (a.dt_fallback_t, a.rows_skipped) == (back, o["rows_skipped"])


@pytest.mark.parametrize("nx,ny,n,level", [(300, 180, 1, 1), (300, 180, 2, 1), (61, 900, 1, 1), (250, 230, 2, 1), (80, 1200, 1, 2)])
def test_dry_rows_on_tiles(gpu, nx, ny, n, level):
    """Few designs of a large grid without rain on the 16x16 tiles, which count the dry rows that the other kernels skip:
    one launch a step (up to 444 tiles) and two, the oracle's count and bits; locked dt and a restored snapshot too."""
    dx = 2.0
    segs = [Segment("inflow", "north", (0.3 * nx * dx, 0.8 * nx * dx), hydrograph=[(0.0, 0.0), (3.0, 0.0), (4.0, 1.5)]),
            Segment("stage", "south", (0.0, 0.5 * nx * dx), stage_m=0.6)]
    base = synthetic_terrain(nx * level, ny * level, dx / level, lambda x, y: 0.02 * y + 0.1 * math.sin(x / 7.0) + 0.1, n=0.03, segments=segs, level=level)
    p = SolverParams(10.0, 5.0, dt_max_s=0.1, rain=Hyetograph([]), initial_depth=0.0)
    terrs, mon = [PreparedTerrain(base)] * n, MonitorSet(np.arange(0, nx * ny, 5))
    o = orc.flat_run(base_arrays(base), design_dict(terrs[0], p), p, mon, want_peak=True, bnd=orc.bnd_dict(base, terrs[0]))
    assert o["rows_skipped"] > 0

    def run():
        r = gpu.run_batch(p, terrs, mon, want_peak=True)
        return gpu.adapter_info(), r

    info, r = run()
    assert "16x16 tiles" in info, info
    for a in r:
        compare_run(a, o, f"{nx}x{ny}")
        assert a.rows_skipped == o["rows_skipped"]
    p.locked_dt = np.full(60, 0.1)   # runs out: back to the last snapshot, adaptive from there
    _, lock = run()
    _, ref = with_options(gpu, {"impl": 2}, run)
    for a, b in zip(lock, ref):
        assert a.steps == b.steps and a.rows_skipped == b.rows_skipped and np.array_equal(a.depth, b.depth)
