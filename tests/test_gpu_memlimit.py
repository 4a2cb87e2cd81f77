"""MEMLIMIT covers the data graph, the tables derived from it and the arena:
under a tight limit the tables are left out, with the same counts."""
import numpy as np
import pytest
import torch

import gfsm_b200
from gfsm_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("labels,limit,tables", [(16, 120 << 20, False), (16, 700 << 20, True), (4, 420 << 20, True), (4, 380 << 20, False),
                                                 (0, 120 << 20, False), (0, 700 << 20, True)])
def test_device_bytes_stay_within_the_limit(labels, limit, tables):
    """labels 0: skewed data, whose table is the hubs' adjacency bits."""
    if labels:
        g = synth.er(600_000, 6.0, seed=3)
        g.vlabel = synth.vlabels(g.n, labels, 0.0, seed=4)
    else:
        g = synth.rmat(18, 1 << 20, seed=5)
    s, d = g.directed()
    q = synth.shape("triangle") if not labels else synth.rw_query(g, 4, tree=True, seed=1)[0]

    def call(limit):
        """Counts, what the data graph holds, and all that the call left allocated."""
        ctx = gfsm_b200.GFSM(device=0, vertex_labels=int(labels > 0), mem_limit=limit)
        free0 = torch.cuda.mem_get_info()[0]
        data = ctx.graph_from_edges(g.n, s, d, None, g.vlabel if labels else None).to_device()
        plan = ctx.pre_process_query(ctx.graph_from_edges(q.n, *q.directed(), None, q.vlabel if labels else None))
        count = ctx.match_count(plan, data)[0]
        held, info = free0 - torch.cuda.mem_get_info()[0], data.info()
        data.close()
        ctx.close()
        return count, info, held

    count, _, _ = call(limit)  # (and the build's workspace joins the pool, which keeps it)
    again, info, held = call(limit)
    want, roomy, _ = call(8 << 30)
    assert count == again == want
    ccsr = (2 * info["n"] + 1 + info["m"]) * 4
    assert (info["device_bytes"] > ccsr) == tables
    assert roomy["device_bytes"] > ccsr
    # allocations are whole pages of 2 MB: graph, table, fixed buffers, arena
    assert held <= limit + (8 << 20)
