"""Limited walks (light calls on skewed data) on the GPU: one that finishes
only because its passes hand work on, and one that gives up to the level
steps, whose attempt the statistics contain and whose like is then left to
them -- on that data graph alone."""
import numpy as np
import pytest

import gfsm_b200
from gfsm_b200 import synth

pytestmark = pytest.mark.gpu


def _path(ctx, k, vlabel):
    q = synth.UGraph(k, np.arange(k - 1, dtype=np.uint32), np.arange(1, k, dtype=np.uint32))
    s, d = q.directed()
    return ctx.pre_process_query(ctx.graph_from_edges(k, s, d, None, np.array(vlabel, np.uint32)))


def _data(ctx, n, m, seed, rare=()):
    g = synth.ba(n, m, seed=seed)
    s, d = g.directed()
    vl = np.zeros(n, np.uint32)
    vl[list(rare)] = 1
    data = ctx.graph_from_edges(n, s, d, None, vl).to_device()
    assert 64 < data.info()["max_degree"] <= 1024
    return data


def test_work_is_handed_on(monkeypatch):
    """One root: its warp ends a pass after 16 rounds of 32 candidates, so the
    rest of thousands was handed on."""
    ctx = gfsm_b200.GFSM(device=0, vertex_labels=1)
    data = _data(ctx, 3000, 4, 3, rare=[1500])
    plan = _path(ctx, 6, [0, 1, 0, 0, 0, 0])
    got, st = ctx.match_count(plan, data)
    assert st["driver"] == 2 and st["launches"] == 4
    assert st["candidates"] > 8 * 16 * 32
    monkeypatch.setenv("GFSM_DRIVER", "host")
    want, st = ctx.match_count(plan, data)
    assert got == want > 0 and st["driver"] == 0
    ctx.close()


def test_giving_up(monkeypatch):
    ctx = gfsm_b200.GFSM(device=0, vertex_labels=1)
    data = _data(ctx, 10000, 6, 3)
    plan = _path(ctx, 6, [0] * 6)
    got, tried = ctx.match_count(plan, data)
    again, left = ctx.match_count(plan, data)  # the class is left to the level steps for a while
    assert tried["driver"] != 2 and left["driver"] != 2
    assert got == again > 0
    # the attempt's four kernels, their time and copies are part of the call
    assert tried["launches"] == left["launches"] + 4
    assert tried["h2d_bytes"] > left["h2d_bytes"] and tried["d2h_bytes"] > left["d2h_bytes"]
    assert tried["wall_ms"] >= tried["kernel_ms"] > 0
    assert tried["candidates"] == left["candidates"]
    # another data graph of the same size and degree is tried
    other = _data(ctx, 10000, 6, 4, rare=[5000])
    light = _path(ctx, 6, [0, 1, 0, 0, 0, 0])
    assert ctx.match_count(light, other)[1]["driver"] == 2
    ctx.close()
