"""The walk's tables (trie of a batch's plans, suffixes of trailing leaves)
and its per-candidate functions, run on the host by a plain depth-first loop
(walk_host.cpp) and compared with the oracle's counts: trees with many
leaves, cycles, equal and overlapping leaf windows, edge labels, repeated
entries, self-loops, one-way edges, shared and unshared."""
import os
import subprocess

import numpy as np
import pytest

from gfsm_b200 import synth
from oracle import oracle as O

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(os.path.dirname(HERE), "gfsm_b200")


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("walk") / "walk_host")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I/usr/local/cuda/include", os.path.join(HERE, "walk_host.cpp"), "-o",
                    out, "-L" + PKG, "-lgfsm", "-Wl,-rpath," + PKG], check=True)
    return out


def _write(path, n, src, dst, lab, vlabel):
    lines = ["t # 0", f"{n} {len(src)} 1 1"] + [f"v {i} {vlabel[i]}" for i in range(n)]
    lines += [f"e {a} {b} {c}" for a, b, c in zip(src, dst, lab)]
    path.write_text("\n".join(lines) + "\nt # -1")


def _tree(k, parent):
    return k, [(p, i + 1) for i, p in enumerate(parent)]


# trees whose trailing leaves hang on one or several anchors
TREES = [_tree(2, [0]), _tree(4, [0, 0, 0]), _tree(5, [0, 0, 1, 1]), _tree(6, [0, 0, 0, 1, 1]), _tree(6, [0, 1, 2, 2, 0]),
         _tree(7, [0, 1, 0, 1, 2, 2]), _tree(5, [0, 1, 2, 3])]
DATA = {
    "er": lambda: synth.er(90, 4.0, seed=3),
    "ba": lambda: synth.ba(70, 2, seed=5),
    "grid": lambda: synth.grid(9, 0.05, 0.1, seed=7),
}


@pytest.mark.parametrize("data", sorted(DATA))
@pytest.mark.parametrize("form", ["plain", "edge_labels", "repeated", "one_way", "loops"])
@pytest.mark.parametrize("vl", [0, 1])
def test_counts(exe, tmp_path, data, form, vl):
    g = DATA[data]()
    rng = np.random.default_rng(17)
    g.vlabel = synth.vlabels(g.n, 2, 0.0, seed=9)
    s, d = g.directed()
    lab = np.ones(len(s), np.uint32)
    if form == "edge_labels":
        half = rng.integers(1, 3, g.m).astype(np.uint32)
        lab = np.concatenate([half, half])
    elif form == "repeated":
        x = rng.integers(0, len(s), 12)
        s, d, lab = np.concatenate([s, s[x]]), np.concatenate([d, d[x]]), np.concatenate([lab, lab[x]])
    elif form == "one_way":
        keep = rng.random(len(s)) < 0.9
        keep[np.unique(s, return_index=True)[1]] = True  # every target keeps a row (the oracle's domain)
        s, d, lab = s[keep], d[keep], lab[keep]
    elif form == "loops":
        x = rng.integers(0, g.n, 8).astype(np.uint32)
        s, d, lab = np.concatenate([s, x]), np.concatenate([d, x]), np.concatenate([lab, np.ones(8, np.uint32)])
    dp = tmp_path / "d.g"
    _write(dp, g.n, s, d, lab, g.vlabel)
    od = O.Graph(path=str(dp))
    qs = []
    for i, (k, e) in enumerate(TREES):
        e = np.array(e, np.uint32).reshape(-1, 2)
        qs.append((k, np.concatenate([e[:, 0], e[:, 1]]), np.concatenate([e[:, 1], e[:, 0]])))
    for i in range(14):
        q, _ = synth.rw_query(g, 3 + i % 4, tree=i % 3 == 0, seed=50 + i)
        qs.append((q.n, *q.directed()))
    if form == "loops":
        qs.append((2, np.array([0, 1, 0], np.uint32), np.array([1, 0, 0], np.uint32)))
    paths, want = [], []
    for i, (k, a, b) in enumerate(qs):
        ql = np.ones(len(a), np.uint32)
        if form == "edge_labels":
            ql = np.array([1 + (int(x) + int(y) + i) % 2 for x, y in zip(a, b)], np.uint32)
        p = tmp_path / f"q{i}.g"
        _write(p, k, a, b, ql, rng.integers(0, 2, k) if vl else np.zeros(k, int))
        oq = O.Graph(path=str(p))
        paths.append(str(p))
        want.append(O.ffs_count(oq, O.Plan(oq), od, vlabel_mode=bool(vl), threads=8))
    assert sum(want) > 0
    for share, leaves, cross, desc in [(0, 0, 0, 0), (1, 0, 0, 1), (0, 1, 1, 0), (1, 1, 1, 1), (1, 1, 0, 1)]:
        r = subprocess.run([exe, str(vl), str(share), str(leaves), str(cross), str(desc), str(dp)] + paths,
                           capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr
        out = r.stdout.strip().split("\n")
        assert [int(x) for x in out[:-1]] == want, (share, leaves, cross, desc)
        assert (int(out[-1].split()[-1]) > 0) == bool(leaves and form != "repeated")
