"""Stars (every later vertex a leaf of the first) counted by the walk on data
with long rows, against the level steps (a context with a candidate cap far
above the work keeps them): rows on both sides of what the walk takes, batches
of stars alone and mixed with other queries, with and without row pointers by
label group, parts of the root window, self-loops."""
import numpy as np
import pytest

import gfsm_b200
from gfsm_b200 import synth

pytestmark = pytest.mark.gpu

STARS = [(2, [(0, 1)]), (3, [(0, 1), (0, 2)]), (3, [(2, 0), (2, 1)]), (4, [(0, 1), (0, 2), (0, 3)])]


def _wide():
    """Two hubs, one above the longest row that a light call's walk tries."""
    a = np.arange(2, 1400, dtype=np.uint32)
    return synth.UGraph(1400, np.concatenate([np.zeros(len(a), np.uint32), np.ones(300, np.uint32), a[:-1]]),
                        np.concatenate([a, a[:300], a[1:]]))


GRAPHS = {"rmat": lambda: synth.rmat(12, 30000, seed=3), "wide": _wide}


@pytest.mark.parametrize("graph", sorted(GRAPHS))
@pytest.mark.parametrize("labels", [0, 1, 3, 20])
@pytest.mark.parametrize("mixed", [False, True])
def test_same_counts(graph, labels, mixed):
    g = GRAPHS[graph]()
    vl = int(labels > 0)
    if vl:
        g.vlabel = synth.vlabels(g.n, labels, 0.0, seed=5)
    s, d = g.directed()
    s, d = np.append(s, [0, 7]).astype(np.uint32), np.append(d, [0, 7]).astype(np.uint32)  # self-loops
    rng = np.random.default_rng(6)
    flat = []
    for i in range(24 if vl else 4):
        k, e = STARS[i % 4]
        e = np.array(e, np.uint32)
        flat.append((k, *synth.UGraph(k, e[:, 0], e[:, 1]).directed()))
    if mixed:
        for name in ("triangle", "4-cycle", "triangle"):
            q = synth.shape(name)
            flat.insert(1, (q.n, *q.directed()))
    flat = [(k, a, b, None, rng.integers(0, min(labels, 3), k).astype(np.uint32) if vl else None) for k, a, b in flat]
    got = []
    for kw in ({}, dict(max_candidates=1 << 60)):
        ctx = gfsm_b200.GFSM(device=0, vertex_labels=vl, **kw)
        data = ctx.graph_from_edges(g.n, s, d, None, g.vlabel).to_device()
        assert data.info()["max_degree"] > 64
        plans = ctx.prepare_queries(flat)
        batch, st = ctx.batch_count(plans, data)
        assert st["count"] == sum(batch.tolist())
        assert batch.tolist() == [ctx.match_count(p, data)[0] for p in plans]
        parts = [ctx.batch_count_part(plans, data, p, 3)[0] for p in range(3)]
        assert np.sum(parts, 0).tolist() == batch.tolist()
        got.append((batch.tolist(), st["driver"], st["candidates"]))
        plans.close()
        ctx.close()
    assert got[0][0] == got[1][0] and sum(got[0][0]) > 0
    if not mixed:
        assert got[0][1] == 2 and got[1][1] != 2
        assert got[0][2] < got[1][2]  # roots only
