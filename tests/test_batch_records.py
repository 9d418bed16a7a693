"""The records that run_arrays hands to the library: one design per entry of dzx, whatever else the lists hold."""
from __future__ import annotations

import numpy as np
import pytest

from itr_gpu import GpuSolver, MonitorSet, PreparedTerrain, synthetic_terrain


def pack(n, **kw):
    base = synthetic_terrain(6, 5, 2.0, lambda x, y: 1.0 + 0.01 * x)
    t = [PreparedTerrain(base) for _ in range(n + 2)]
    a = dict(dzx=[x.dzx for x in t[:n]], dzy=[x.dzy for x in t[:n]], dzx2=None, dzy2=None, h0=None, vols=None, z_edge=None)
    a.update({k: v(t) for k, v in kw.items()})
    keep = []
    solver = GpuSolver.__new__(GpuSolver)   # (no device)
    b = solver._pack(base, a["dzx"], a["dzy"], a["dzx2"], a["dzy2"], a["h0"], a["vols"], MonitorSet([3]), None, None, False, None,
                     False, True, 0, keep, z_edge=a["z_edge"])
    return b, keep


def test_longer_lists_are_read_up_to_the_designs():
    depth = [np.full(30, 0.1 * i, dtype=np.float32) for i in range(4)]
    b, _ = pack(2, dzy=lambda t: [x.dzy for x in t], dzx2=lambda t: [None] * 4, h0=lambda t: depth, vols=lambda t: [(1.0 + i, 2.0 + i) for i in range(4)],
                z_edge=lambda t: [np.zeros(22) for _ in t])
    assert b["n"] == 2
    for i in range(2):
        assert [b["D"][i].h0[k] for k in range(30)] == depth[i].tolist()
        assert (b["D"][i].cut_m3, b["D"][i].fill_m3) == (1.0 + i, 2.0 + i)
        assert not b["D"][i].dzx2 and b["D"][i].z_edge


def test_empty_lists_mean_none():
    b, _ = pack(2, dzx2=lambda t: [], dzy2=lambda t: [], h0=lambda t: [], vols=lambda t: [], z_edge=lambda t: [])
    for i in range(2):
        assert b["D"][i].dzx and b["D"][i].dzy and not b["D"][i].h0 and not b["D"][i].z_edge and b["D"][i].cut_m3 == 0.0


@pytest.mark.parametrize("field", ["dzy", "dzx2", "h0", "vols", "z_edge"])
def test_shorter_lists_are_refused(field):
    one = {"dzy": lambda t: [t[0].dzy], "dzx2": lambda t: [t[0].dzx], "h0": lambda t: [np.zeros(30, np.float32)], "vols": lambda t: [(0.0, 0.0)],
           "z_edge": lambda t: [np.zeros(22)]}[field]
    with pytest.raises(IndexError):
        pack(2, **{field: one})
