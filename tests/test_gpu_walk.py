"""The walk (one kernel per call) against the level steps (GFSM_DRIVER=host) on
the same device graph: every tuple length from 2 to 16 vertices, 1 to 300
queries a call (queues that fill and drain), more label groups than the row
pointers by group hold, edge labels, repeated entries, a self-loop, the
longest row of an unlimited walk and the next one, and limited walks on
skewed data, whose passes hand work on (one root with most of it, children in
groups, long slices in parts) or give up."""
import numpy as np
import pytest

import gfsm_b200
from gfsm_b200 import synth

pytestmark = pytest.mark.gpu


def _counts(ctx, plans, data, monkeypatch, walked):
    walk, st = ctx.batch_count(plans, data)
    if walked is not None:  # None: a limited walk, which may give up
        assert (st["driver"] == 2) == walked
    monkeypatch.setenv("GFSM_DRIVER", "host")
    level, st = ctx.batch_count(plans, data)
    monkeypatch.delenv("GFSM_DRIVER")
    assert st["driver"] == 0
    assert walk.tolist() == level.tolist() and level.sum() > 0
    # the parts of a partition as well
    parts = [ctx.batch_count_part(plans, data, p, 3)[0] for p in range(3)]
    assert sum(parts).tolist() == level.tolist()


@pytest.mark.parametrize("nq", [1, 2, 33, 300])
@pytest.mark.parametrize("form", ["labels", "many_labels", "edge_labels", "repeated", "loop", "nine_labels"])
def test_walk_equals_level_steps(monkeypatch, form, nq):
    ctx = gfsm_b200.GFSM(device=0, vertex_labels=1)
    g = synth.grid(40, 0.05, 0.05, seed=nq)
    g.vlabel = synth.vlabels(g.n, {"many_labels": 17, "nine_labels": 9}.get(form, 3), 0.0, seed=4)
    s, d = g.directed()
    lab = np.ones(len(s), np.uint32)
    if form == "edge_labels":
        lab = 1 + (s ^ d) % 2
    elif form == "repeated":
        s, d, lab = np.append(s, s[:50]), np.append(d, d[:50]), np.append(lab, lab[:50])
    elif form == "loop":
        s, d, lab = np.append(s, [3, 9]), np.append(d, [3, 9]), np.append(lab, [1, 1])
    data = ctx.graph_from_edges(g.n, s, d, lab, g.vlabel)
    qs = []
    for i in range(nq):
        q, seen = synth.rw_query(g, 2 + i % 11 if nq > 1 else 7, tree=i % 2 == 0, seed=70 + i)
        a, b = q.directed()
        ql = 1 + (seen[a] ^ seen[b]) % 2 if form == "edge_labels" else np.ones(len(a), np.uint32)
        qs.append((q.n, a, b, ql.astype(np.uint32), q.vlabel))
    _counts(ctx, ctx.prepare_queries(qs), data, monkeypatch, True)
    ctx.close()


@pytest.mark.parametrize("row,walked", [(64, True), (65, None)])
def test_longest_row(monkeypatch, row, walked):
    """A star of `row` leaves beside a path and a cycle: long queries, 15
    equal leaves (a falling factorial), leaves on several anchors."""
    ctx = gfsm_b200.GFSM(device=0)
    hub = [(0, i + 1) for i in range(row)]
    n = row + 1
    path = [(n + i, n + i + 1) for i in range(39)] + [(n + 39, n), (1, n), (2, n + 3)]
    e = np.array(hub + path, np.uint32)
    data = ctx.graph_from_edges(n + 40, np.concatenate([e[:, 0], e[:, 1]]), np.concatenate([e[:, 1], e[:, 0]]))
    shapes = [[(i, i + 1) for i in range(15)], [(0, i + 1) for i in range(6)], [(0, 1), (1, 2), (0, 3), (0, 4), (2, 5)],
              [(0, 1), (1, 2), (2, 3), (3, 0), (0, 4), (0, 5), (1, 6)], [(i, i + 1) for i in range(11)] + [(0, 12), (0, 13)]]
    qs = []
    for sh in shapes:
        q = np.array(sh, np.uint32)
        qs.append((int(q.max()) + 1, np.concatenate([q[:, 0], q[:, 1]]), np.concatenate([q[:, 1], q[:, 0]]), None, None))
    _counts(ctx, ctx.prepare_queries(qs), data, monkeypatch, walked)
    ctx.close()


@pytest.mark.parametrize("n,m,labels,nq", [(3000, 2, 1, 3), (3000, 4, 6, 1), (3000, 4, 6, 40), (60000, 4, 12, 9),
                                           (800, 12, 4, 25)])
def test_limited_walk(monkeypatch, n, m, labels, nq):
    ctx = gfsm_b200.GFSM(device=0, vertex_labels=1)
    g = synth.ba(n, m, seed=n)
    g.vlabel = synth.vlabels(g.n, labels, 1.0, seed=4)
    s, d = g.directed()
    data = ctx.graph_from_edges(g.n, s, d, None, g.vlabel)
    rng = np.random.default_rng(n)
    qs = []
    for i in range(nq):
        q, _ = synth.rw_query(g, 3 + i % 4, tree=i % 2 == 0, seed=90 + i)
        qs.append((q.n, *q.directed(), None, rng.integers(labels // 2, labels, q.n).astype(np.uint32)))
    _counts(ctx, ctx.prepare_queries(qs), data, monkeypatch, None)
    ctx.close()


def _path(k, vlabel):
    q = synth.UGraph(k, np.arange(k - 1, dtype=np.uint32), np.arange(1, k, dtype=np.uint32))
    q.vlabel = np.array(vlabel, np.uint32)
    return q


@pytest.mark.parametrize("form", ["labels", "edge_labels", "mappings", "clique"])
def test_few_roots_hand_work_on(monkeypatch, form):
    """A few warps hold all the work of a walk: ten roots of a rare label, or
    a clique whose vertices one warp takes at once.  They hand it on to the
    next pass (a launch each, and one between), with the same counts."""
    ctx = gfsm_b200.GFSM(device=0, vertex_labels=1)
    if form == "clique":  # 40 vertices of a 100 x 100 grid
        g = synth.grid(100, 0.0, 0.0, seed=1)
        a, b = np.triu_indices(40, 1)
        g = synth.UGraph(g.n, np.append(g.src, a.astype(np.uint32) * 7), np.append(g.dst, b.astype(np.uint32) * 7))
        g.vlabel = np.zeros(g.n, np.uint32)
        q = _path(5, [0] * 5)
    else:
        g = synth.er(20000, 16.0 if form == "mappings" else 24.0, seed=3)
        g.vlabel = np.zeros(g.n, np.uint32)
        g.vlabel[5::2003] = 1
        q = _path(5, [0, 1, 0, 0, 0])
    s, d = g.directed()
    a, b = q.directed()
    lab, ql = np.ones(len(s), np.uint32), np.ones(len(a), np.uint32)
    if form == "edge_labels":
        lab[:] = 1 + (s ^ d) % 2
    data = ctx.graph_from_edges(g.n, s, d, lab, g.vlabel).to_device()
    assert data.info()["max_degree"] <= 64
    plans = ctx.prepare_queries([(q.n, a, b, ql, q.vlabel)])
    got, st = ctx.match_count(plans[0], data)
    assert st["driver"] == 2 and st["launches"] >= 3
    rows = ctx.match_mappings(plans[0], data, max_rows=1 << 20)[0] if form == "mappings" else None
    monkeypatch.setenv("GFSM_DRIVER", "host")
    want, st = ctx.match_count(plans[0], data)
    assert st["driver"] == 0
    assert got == want > 0
    if form == "mappings":  # (every core vertex is enumerated there: far more rounds than the count took)
        level = ctx.match_mappings(plans[0], data, max_rows=1 << 20)[0]
        assert len(rows) == want and np.array_equal(rows[np.lexsort(rows.T)], level[np.lexsort(level.T)])
    plans.close()
    ctx.close()
