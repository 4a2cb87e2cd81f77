"""The level steps' shortest-row candidates, last vertices counted at their
parents on long rows, and descending orbits against the same steps without
them (a context with a candidate cap far above the work keeps the earlier
form) and, for triangles, an independent counter: rows on both sides of the
register-held length, hubs (unlabelled, from rows of
512 entries, checked by bits), batches whose trie nodes mix children that are
counted with children that are not, both drivers."""
import numpy as np
import pytest

import gfsm_b200
from gfsm_b200 import synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu

GRAPHS = {
    "rmat": lambda: synth.rmat(11, 20000, seed=3),
    "hubs": lambda: synth.rmat(12, 30000, seed=3),
    "ba": lambda: synth.ba(3000, 3, seed=4),
    "hub": lambda: synth.UGraph(400, np.concatenate([np.zeros(399, np.uint32), np.arange(1, 399, dtype=np.uint32)]),
                                np.concatenate([np.arange(1, 400, dtype=np.uint32), np.arange(2, 400, dtype=np.uint32)])),
}


@pytest.mark.parametrize("graph", sorted(GRAPHS))
@pytest.mark.parametrize("labels", [0, 1, 3])
@pytest.mark.parametrize("driver", ["host", "graph"])
def test_same_counts(monkeypatch, graph, labels, driver):
    monkeypatch.setenv("GFSM_DRIVER", driver)
    monkeypatch.setenv("GFSM_TILE", "0")
    g = GRAPHS[graph]()
    vl = int(labels > 0)
    if vl:
        g.vlabel = synth.vlabels(g.n, labels, 0.0, seed=5)
    s, d = g.directed()
    qs = [synth.shape(x) for x in ("triangle", "4-clique", "path3", "4-cycle", "path3")]
    qs += [synth.rw_query(g, 3 + i % 2, tree=i % 3 == 0, seed=30 + i)[0] for i in range(40 if vl else 4)]
    rng = np.random.default_rng(6)
    flat = [(q.n, *q.directed(), None, rng.integers(0, labels, q.n).astype(np.uint32) if vl else None) for q in qs]
    got = []
    for kw in ({}, dict(max_candidates=1 << 60)):
        ctx = gfsm_b200.GFSM(device=0, vertex_labels=vl, **kw)
        data = ctx.graph_from_edges(g.n, s, d, None, g.vlabel).to_device()
        assert graph != "hubs" or data.info()["max_degree"] >= 512
        plans = ctx.prepare_queries(flat)
        batch, st = ctx.batch_count(plans, data)
        assert batch.tolist() == [ctx.match_count(p, data)[0] for p in plans]
        got.append((batch.tolist(), st["candidates"]))
        plans.close()
        ctx.close()
    assert got[0][0] == got[1][0] and sum(got[0][0]) > 0
    assert got[0][1] < got[1][1]  # fewer candidates, the same counts
    if not vl:
        assert got[0][0][0] == 6 * O.triangles(g.n, g.src, g.dst)
