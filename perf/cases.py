"""Workloads of the matcher through its public Python entry points.

A case names a data graph, the queries run against it and the call a program
makes:

  single    match_count: one query at a time, the plain form
  batch     batch_count over plans the program keeps
  ingest    prepare_queries_flat + batch_count + close: a batch of queries
            that arrive as edge lists, planned, counted and freed
  mappings  match_mappings: the embeddings themselves
  build     graph_from_edges + to_device + download: a data graph made resident
  serve     a running server: submit every request, drain, poll

Graphs and query shapes are those of the package's workload configurations
(gfsm_b200/synth.py); R-MAT edges are drawn on the GPU, which takes
milliseconds where the host generator takes seconds.
"""
import math

import numpy as np
import torch

import gfsm_b200
from gfsm_b200 import synth

EDGE_LABELS = 3
MAX_ROWS = 1 << 16
SHAPES = {
    "path3": (3, [(0, 1), (1, 2)]),
    "triangle": (3, [(0, 1), (1, 2), (0, 2)]),
    "4-clique": (4, [(0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3)]),
}


def listed():
    return [
        # the smallest call: one labelled five-vertex query on a graph of 2,000
        # vertices, where latency and launches are all there is
        dict(name="er_single", call="single", graph="er", n=2000, deg=8.0, labels=4, vl=1, k=5, nq=1),
        # the same graph with vertex labels ignored: millions of embeddings
        dict(name="er_unlabelled", call="single", graph="er", n=2000, deg=8.0, labels=4, vl=0, k=5, nq=1),
        # the embeddings of a query, not their number
        dict(name="er_mappings", call="mappings", graph="er", n=2000, deg=8.0, labels=4, vl=1, k=5, nq=1),
        # one query at a time against a resident road-like network
        dict(name="grid_single", call="single", graph="grid", side=1400, labels=4, vl=1, k=7, nq=1),
        # what a server slot sees under moderate load: a few dozen queries of uneven size
        dict(name="grid_batch_64", call="batch", graph="grid", side=1400, labels=4, vl=1, kmin=4, kmax=10, nq=64),
        # the headline batch, from edge lists to counts
        dict(name="grid_ingest_4096", call="ingest", graph="grid", side=1400, labels=4, vl=1, kmin=4, kmax=10,
             nq=4096),
        # requests to a running server
        dict(name="grid_serve_256", call="serve", graph="grid", side=1400, labels=4, vl=1, kmin=4, kmax=10, nq=256),
        # making a road network resident: the device CCSR builder and its copies
        dict(name="grid_build", call="build", graph="grid", side=1400, labels=4, vl=1),
        # hub-heavy unlabelled graph: one heavy query
        dict(name="rmat_triangle", call="single", graph="rmat", scale=20, edges=16 << 20, labels=0, vl=0,
             shape="triangle", nq=1),
        # labelled power-law graph: a batch of small queries, each with very many embeddings
        dict(name="rmat_batch_64", call="batch", graph="rmat", scale=20, edges=8 << 20, labels=8, vl=1,
             shape="three", nq=64),
        # Zipf-labelled preferential-attachment graph, order chosen for the data
        dict(name="ba_planned", call="single", graph="ba", n=500_000, m=4, labels=16, vl=1, k=6, planned=1, nq=1),
        # edges with labels, as in RDF data
        dict(name="er_edge_labels", call="batch", graph="er", n=100_000, deg=6.0, labels=3, vl=1, kmin=4, kmax=6,
             elab=1, nq=32),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["er", "er", "mappings", "grid", "batch", "ingest", "serve", "build", "rmat", "rmat_batch", "ba",
                       "edge_labels"])
    if kind == "er":
        if rng.random() < 0.5:
            return dict(call="single", graph="er", n=int(_log(rng, 500, 20000)), deg=rng.uniform(4, 10), labels=4,
                        vl=1, k=rng.randint(3, 7), nq=1)
        return dict(call="single", graph="er", n=int(_log(rng, 500, 5000)), deg=rng.uniform(3, 8), labels=4, vl=0,
                    k=rng.randint(3, 5), nq=1)
    if kind == "mappings":
        return dict(call="mappings", graph="er", n=int(_log(rng, 500, 4000)), deg=rng.uniform(3, 8), labels=4, vl=1,
                    k=rng.randint(3, 6), nq=1)
    side = int(_log(rng, 150, 1400))
    if kind == "grid":
        return dict(call="single", graph="grid", side=side, labels=rng.choice([3, 4, 6]), vl=1, k=rng.randint(4, 10),
                    nq=1)
    if kind == "batch":
        return dict(call="batch", graph="grid", side=side, labels=4, vl=1, kmin=rng.randint(3, 5),
                    kmax=rng.randint(6, 10), nq=int(_log(rng, 2, 1000)))
    if kind == "ingest":
        return dict(call="ingest", graph="grid", side=side, labels=4, vl=1, kmin=4, kmax=rng.randint(7, 10),
                    nq=int(_log(rng, 256, 4096)))
    if kind == "serve":
        return dict(call="serve", graph="grid", side=side, labels=4, vl=1, kmin=4, kmax=rng.randint(6, 10),
                    nq=int(_log(rng, 1, 1024)))
    if kind == "build":
        if rng.random() < 0.5:
            return dict(call="build", graph="grid", side=side, labels=4, vl=1)
        return dict(call="build", graph="ba", n=int(_log(rng, 5_000, 500_000)), m=rng.randint(2, 6), labels=16, vl=1)
    if kind == "rmat":
        shape = rng.choice(["triangle", "triangle", "path3", "4-clique"])
        top = 400_000 if shape == "4-clique" else 16 << 20
        edges = int(_log(rng, 50_000, top))
        return dict(call="single", graph="rmat", scale=max(13, min(20, round(math.log2(edges / rng.uniform(8, 16))))),
                    edges=edges, labels=0, vl=0, shape=shape, nq=1)
    if kind == "rmat_batch":
        edges = int(_log(rng, 100_000, 8 << 20))
        return dict(call="batch", graph="rmat", scale=max(14, round(math.log2(edges / 8))), edges=edges, labels=8, vl=1,
                    shape="three", nq=rng.randint(3, 64))
    if kind == "ba":
        return dict(call="single", graph="ba", n=int(_log(rng, 20_000, 500_000)), m=rng.randint(2, 4), labels=16, vl=1,
                    k=rng.randint(4, 7), planned=rng.randint(0, 1), nq=1)
    return dict(call="batch", graph="er", n=int(_log(rng, 5_000, 100_000)), deg=rng.uniform(4, 7), labels=3, vl=1,
                kmin=4, kmax=rng.randint(5, 6), elab=1, nq=rng.randint(2, 64))


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _rmat(scale, edges, seed):
    gen = torch.Generator("cuda").manual_seed(seed)
    src = torch.zeros(edges, dtype=torch.int64, device="cuda")
    dst = torch.zeros_like(src)
    for bit in range(scale):
        r = torch.rand(edges, device="cuda", generator=gen)
        src |= (r >= 0.76).long() << bit
        dst |= (((r >= 0.57) & (r < 0.76)) | (r >= 0.95)).long() << bit
    key = torch.unique((torch.minimum(src, dst) << 32) | torch.maximum(src, dst))
    a, b = key >> 32, key & 0xFFFFFFFF
    keep = a != b
    to = lambda x: x[keep].to(torch.int32).cpu().numpy().view(np.uint32)
    return synth.UGraph(1 << scale, to(a), to(b))


def _edge_label(a, b):
    """The label of the undirected edge (a, b): the same in data and query."""
    a, b = np.asarray(a, np.uint64), np.asarray(b, np.uint64)
    h = np.minimum(a, b) * np.uint64(0x9E3779B97F4A7C15) + np.maximum(a, b) * np.uint64(0xC2B2AE3D27D4EB4F)
    return ((h >> np.uint64(40)) % np.uint64(EDGE_LABELS) + np.uint64(1)).astype(np.uint32)


def _graph(case, seed):
    kind = case["graph"]
    if kind == "er":
        g = synth.er(case["n"], case["deg"], seed=seed)
    elif kind == "grid":
        g = synth.grid(case["side"], 0.05, 0.02, seed=seed)
    elif kind == "rmat":
        g = _rmat(case["scale"], case["edges"], seed)
    else:
        g = synth.ba(case["n"], case["m"], seed=seed)
    if case["labels"]:
        g.vlabel = synth.vlabels(g.n, case["labels"], 1.0 if kind == "ba" else 0.0, seed=seed + 100)
    return g


def _shape(name, vlabel=None):
    k, e = SHAPES[name]
    e = np.array(e, np.uint32)
    return synth.UGraph(k, e[:, 0], e[:, 1], vlabel)


def _queries(case, g, seed):
    """(query, visited data vertices or None) for every query of the case."""
    rng = np.random.default_rng(seed + 7)
    if case.get("shape") == "three":  # paths and triangles with random labels
        return [(_shape("triangle" if rng.random() < 0.15 else "path3",
                        rng.integers(0, case["labels"], 3).astype(np.uint32)), None) for _ in range(case["nq"])]
    if case.get("shape"):
        return [(_shape(case["shape"]), None)]
    out = []
    for i in range(case["nq"]):
        k = case["k"] if "k" in case else int(rng.integers(case["kmin"], case["kmax"] + 1))
        q, seen = synth.rw_query(g, k, tree=False, seed=1 + i + 1_000_003 * seed)
        if case["graph"] == "ba":  # a program asks for the rarer labels: frequent ones have no end of embeddings
            q.vlabel = rng.integers(4, case["labels"], k).astype(np.uint32)
        out.append((q, seen))
    return out


_CTX = {}


def _ctx(vl):
    """The program's one context for each label mode, kept for its life."""
    if vl not in _CTX:
        _CTX[vl] = gfsm_b200.GFSM(vertex_labels=vl)
    return _CTX[vl]


class _Served:
    """A running server and what it works on; stopped with the state."""

    def __init__(self, ctx, data):
        self.data = data
        self.server = ctx.serve(data, slots=2, max_batch=4096)

    def __del__(self):
        self.server.stop()


def _inputs(case, seed):
    g = _graph(case, seed)
    if case["call"] == "build" and case["graph"] == "grid":  # as many edges whatever the seed
        keep = np.sort(np.random.default_rng(seed).permutation(g.m)[: int(1.9 * case["side"] * (case["side"] - 1))])
        g = synth.UGraph(g.n, g.src[keep], g.dst[keep], g.vlabel)
    src, dst = g.directed()
    elab = _edge_label(src, dst) if case.get("elab") else None
    return g, src, dst, elab, (g.vlabel if case["vl"] else None)


def prepare(case, seed):
    ctx = _ctx(case["vl"])
    g, src, dst, elab, vlabel = _inputs(case, seed)
    if case["call"] == "build":
        return dict(call="build", ctx=ctx, args=(g.n, src, dst, elab, vlabel))
    data = ctx.graph_from_edges(g.n, src, dst, elab, vlabel).to_device()
    flat = []
    for q, seen in _queries(case, g, seed):
        qs, qd = q.directed()
        flat.append((q.n, qs, qd, _edge_label(seen[qs], seen[qd]) if case.get("elab") else None,
                     q.vlabel if case["vl"] else None))
    st = dict(call=case["call"], ctx=ctx, data=data)
    if case["call"] == "ingest":
        cat = lambda i: np.concatenate([f[i] for f in flat])
        eoff = np.zeros(len(flat) + 1, np.uint64)
        np.cumsum([len(f[1]) for f in flat], out=eoff[1:])
        st["flat"] = (np.array([f[0] for f in flat], np.uint32), eoff, cat(1), cat(2), None, cat(4))
    elif case.get("planned"):
        st["plans"] = [ctx.plan_for(ctx.graph_from_edges(*f), data) for f in flat]
    else:
        st["plans"] = ctx.prepare_queries(flat)
    if case["call"] == "serve":
        st["served"] = _Served(ctx, data)
    return st


def _table(rows):
    """A set of embeddings, which has no order of its own, as one table."""
    out = np.full((MAX_ROWS, rows.shape[1]), 0xFFFFFFFF, np.uint32)
    out[: len(rows)] = rows[np.lexsort(rows.T[::-1])]
    return out


def run(st):
    ctx, call = st["ctx"], st["call"]
    if call == "build":
        g = ctx.graph_from_edges(*st["args"]).to_device()
        out = g.download()
        g.close()
        return out
    if call == "single":
        return ctx.match_count(st["plans"][0], st["data"])[0]
    if call == "batch":
        return ctx.batch_count(st["plans"], st["data"])[0]
    if call == "ingest":
        plans = ctx.prepare_queries_flat(*st["flat"])
        counts = ctx.batch_count(plans, st["data"])[0]
        plans.close()
        return counts
    if call == "mappings":
        rows, count = ctx.match_mappings(st["plans"][0], st["data"], max_rows=MAX_ROWS)
        return _table(rows), count
    server = st["served"].server
    for i, p in enumerate(st["plans"]):
        server.submit(p, i)
    server.drain()
    counts = np.zeros(len(st["plans"]), np.uint64)
    for r in server.poll():
        counts[r["req_id"]] = r["count"]
    return counts


def work(case):
    """Each entry of the data graph's rows and row bounds read once, the
    queries' edges read and the counts written; building reads the edge list
    and writes the rows."""
    if case["graph"] == "er":
        n, m = case["n"], case["n"] * case["deg"]
    elif case["graph"] == "grid":
        n = case["side"] ** 2
        m = n * 3.88
    elif case["graph"] == "rmat":
        n, m = 1 << case["scale"], 2.0 * case["edges"]
    else:
        n, m = case["n"], 2.0 * case["m"] * case["n"]
    entry = 5.0 if case.get("elab") else 4.0
    if case["call"] == "build":
        return {"bytes": m * 9.0 + n * 4.0 + m * 5.0 + n * 8.0, "flops": 0}
    return {"bytes": m * entry + n * 4.0 + case["nq"] * (10 * 2 * 8.0 + 8.0), "flops": 0}


# ---------------------------------------------------------------------------
# The same results from numpy and torch alone
# ---------------------------------------------------------------------------
def _rows(n, src, dst, deg_order):
    """CSR by original id; rows sorted by target's place in deg_order."""
    o = np.lexsort((deg_order[dst], src))
    return np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))]), dst[o].astype(np.int64), o


def _join(n, src, dst, q, vl):
    """All embeddings of q, extended vertex by vertex."""
    ptr, adj, _ = _rows(n, src, dst, np.arange(n))
    keys = np.sort(src.astype(np.int64) * n + dst)
    nb = [set() for _ in range(q[0])]
    for a, b in zip(q[1].tolist(), q[2].tolist()):
        nb[a].add(b)
    order = [0]
    while len(order) < q[0]:
        order.append(next(v for v in range(q[0]) if v not in order and nb[v] & set(order)))
    has = np.diff(ptr) > 0
    t = np.flatnonzero(has if vl is None else has & (vl == q[3][0]))[:, None]
    for d in range(1, q[0]):
        v = order[d]
        back = [order.index(u) for u in nb[v] if u in order[:d]]
        a = t[:, back[0]]
        ln = ptr[a + 1] - ptr[a]
        rep = np.repeat(np.arange(len(t)), ln)
        c = adj[np.arange(len(rep)) - np.repeat(np.cumsum(ln) - ln, ln) + np.repeat(ptr[a], ln)]
        ok = np.ones(len(c), bool) if vl is None else vl[c] == q[3][v]
        for j in range(d):
            ok &= t[rep, j] != c
        for b in back[1:]:
            k = t[rep, b] * n + c
            ok &= keys[np.minimum(np.searchsorted(keys, k), len(keys) - 1)] == k
        t = np.concatenate([t[rep[ok]], c[ok][:, None]], 1)
    return t[:, np.argsort(order)]


def exact(case, seed):
    if case["call"] == "build":
        _, src, dst, elab, vlabel = _inputs(case, seed)
        n = case["side"] ** 2 if case["graph"] == "grid" else case["n"]
        deg = np.bincount(src, minlength=n)
        group = np.zeros(n, np.int64) if vlabel is None else vlabel.astype(np.int64)
        order = np.lexsort((np.arange(n), -deg, group))
        place = np.empty(n, np.int64)
        place[order] = np.arange(n)
        o = np.lexsort((place[dst], place[src]))
        rowptr = np.concatenate([[0], np.cumsum(deg[order])])
        return (rowptr.astype(np.uint32), place[dst[o]].astype(np.uint32), np.ones(len(src), np.uint8),
                order.astype(np.uint32))
    if case["call"] not in ("single", "mappings") or case["graph"] not in ("er", "grid") or case.get("elab"):
        return None  # too many embeddings to list here
    if not case["vl"] and case["n"] * case["deg"] ** (case["k"] - 1) > 2e7:
        return None
    g, src, dst, _, vlabel = _inputs(case, seed)
    q = _queries(case, g, seed)[0][0]
    t = _join(g.n, src, dst, (q.n, *q.directed(), q.vlabel), None if vlabel is None else vlabel)
    if case["call"] == "single":
        return len(t)
    return _table(t.astype(np.uint32)), len(t)
