"""Materialised designs whose bounding boxes end at, before and after the chunks and warps of the
volume sums, and primitives at the edges of the test that leaves far cells out (thin, of no
height, overlapping, of both signs): volumes and jumps equal the host's materialisation bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import assert_bitwise
from itr_gpu import GpuSolver, Hyetograph, MonitorSet, PreparedTerrain, SolverParams, synthetic_terrain
from itr_gpu.design import CUT, MOUND, Primitive, materialize

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(64, 64), (65, 63), (33, 31), (129, 97)])
def test_boxes_around_the_chunks(nx, ny):
    base = synthetic_terrain(nx, ny, 2.0, lambda x, y: 3.0 - 0.01 * x, n=0.03)
    geo, ed = base.fine.geo, np.ones((ny, nx), dtype=bool)
    cx, cy, w, h = nx * 1.0, ny * 1.0, nx * 2.0, ny * 2.0
    sets = [
        [Primitive(MOUND, cx, cy, 0.0, 3.0 * (w + h), 0.0, 0.4)],                                   # the whole grid raised
        [Primitive(CUT, cx, cy, 3.0 * (w + h), 3.0 * (w + h), 0.0, -0.4)],                           # lowered to the last cell
        [Primitive(0, cx, cy, 0.8 * w, 5.0, 33.0, 0.3), Primitive(1, cx, cy, 0.7 * h, 7.0, 120.0, -0.2),
         Primitive(MOUND, 0.3 * w, 0.6 * h, 0.0, 0.5 * w, 0.0, -0.1)],                              # crossing, both signs
        [Primitive(0, cx, cy, w, 0.01, 45.0, 0.3)],                                                 # thinner than the samples
        [Primitive(MOUND, cx, cy, 0.0, 2.0, 0.0, 0.2)],                                             # one cell
        [Primitive(0, cx, cy, 0.5 * w, 6.0, 10.0, 0.0)],                                            # no height
        [],
    ]
    p = SolverParams(4.0, 2.0, rain=Hyetograph.from_mm_h([(0, 300), (4, 300)]), initial_depth=0.05)
    mon = MonitorSet(np.arange(0, nx * ny, 7))
    g = GpuSolver()
    try:
        edits = [materialize(s, geo, nx, ny, ed, 0.5) for s in sets]
        ref = g.run_batch(p, [PreparedTerrain(base).apply_edit(e) for e in edits], mon)
        got, cut, fill = g.run_primitives(p, base, sets, mon, ed, 0.5)
    finally:
        g.close()
    for i, e in enumerate(edits):
        assert cut[i] == e.cut_m3 and fill[i] == e.fill_m3, f"{nx}x{ny} design {i}: {cut[i]}, {fill[i]} vs {e.cut_m3}, {e.fill_m3}"
        assert_bitwise(got[i].depth, ref[i].depth, f"{nx}x{ny} design {i}")
