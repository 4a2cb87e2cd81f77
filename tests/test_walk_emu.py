"""The walk's kernel run on the host, lane by lane (walk_emu.cpp): lanes in a
random order between the warp intrinsics, every array ending at an unmapped
page, clamps counted.  Counts against the oracle's: queues that fill and
drain, batches of up to 300 queries, limited walks that hand work from pass to
pass, and list units with a depth out of range, which must stay in bounds."""
import os
import subprocess

import numpy as np
import pytest

from gfsm_b200 import synth
from oracle import oracle as O
from test_walk_host import _write

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(os.path.dirname(HERE), "gfsm_b200")


def _build(tmp_path_factory, *flags):
    out = str(tmp_path_factory.mktemp("walk") / "walk_emu")
    # (the lanes' stacks are switched by longjmp, which a fortified build forbids)
    subprocess.run(["g++", "-O1", "-std=c++17", "-U_FORTIFY_SOURCE", "-w", "-I/usr/local/cuda/include", *flags,
                    os.path.join(HERE, "walk_emu.cpp"), "-o", out, "-L" + PKG, "-lgfsm", "-Wl,-rpath," + PKG], check=True)
    return out


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    return _build(tmp_path_factory)


@pytest.fixture(scope="module")
def exe_short_list(tmp_path_factory):
    """Lists of 40 units."""
    return _build(tmp_path_factory, "-DGFSM_WALK_LISTED=40")


@pytest.fixture(scope="module")
def exe_spill(tmp_path_factory):
    """A lane's totals are added to the call's from 64 on."""
    return _build(tmp_path_factory, "-DGFSM_SPILL_BITS=6")


def _few_roots():
    """Five vertices of label 1, the rest label 0, rows of about 16; a path
    whose search starts at its one vertex of label 1."""
    g = synth.er(300, 16.0, seed=11)
    g.vlabel = np.zeros(g.n, np.uint32)
    g.vlabel[7:300:60] = 1
    k = 6
    q = synth.UGraph(k, np.arange(k - 1, dtype=np.uint32), np.arange(1, k, dtype=np.uint32))
    q.vlabel = np.array([0, 1] + [0] * (k - 2), np.uint32)
    return g, [(q, np.arange(k))]


def _case(tmp_path, g, nq, sizes, labels, edge_labels=False):
    """Data and queries as files, and the oracle's counts."""
    if isinstance(g, tuple):
        g, queries = g
    else:
        g.vlabel = synth.vlabels(g.n, labels, 0.0, seed=9)
        queries = [synth.rw_query(g, sizes[i % len(sizes)], tree=i % 2 == 0, seed=1 + i) for i in range(nq)]
    s, d = g.directed()
    lab = 1 + (s ^ d) % 2 if edge_labels else np.ones(len(s), np.uint32)
    _write(tmp_path / "d.g", g.n, s, d, lab, g.vlabel)
    od = O.Graph(path=str(tmp_path / "d.g"))
    paths, want = [], []
    for i, (q, seen) in enumerate(queries):
        a, b = q.directed()
        p = tmp_path / f"q{i}.g"
        _write(p, q.n, a, b, 1 + (seen[a] ^ seen[b]) % 2 if edge_labels else np.ones(len(a), np.uint32), q.vlabel)
        oq = O.Graph(path=str(p))
        paths.append(str(p))
        want.append(O.ffs_count(oq, O.Plan(oq), od, vlabel_mode=True, threads=8))
    return paths, want


def _run(exe, tmp_path, paths, form, seed):
    r = subprocess.run([exe, "1", "1", "1", str(int(form == "walk")), "1", form, str(seed), str(tmp_path / "d.g")] + paths,
                       capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr
    out = r.stdout.strip().split("\n")
    last = out[-1].split()
    return [int(x) for x in out[:-1]], dict(zip(last[::2], map(int, last[1::2])))


CASES = {
    "grid": (lambda: synth.grid(30, 0.05, 0.1, seed=7), 40, [3, 5, 7], 3, False),
    "grid_batch": (lambda: synth.grid(40, 0.05, 0.1, seed=7), 300, [4, 5, 6, 7, 8, 9, 10], 3, False),
    "edge_labels": (lambda: synth.grid(24, 0.05, 0.1, seed=8), 24, [2, 4, 6, 9], 3, True),
    "few_roots": (lambda: _few_roots(), 1, [6], 2, False),
    "few_roots_edge_labels": (lambda: _few_roots(), 1, [6], 2, True),
    "ba": (lambda: synth.ba(300, 3, seed=5), 8, [3, 4, 5], 2, False),
}


@pytest.mark.parametrize("case", sorted(CASES))
@pytest.mark.parametrize("seed", [1, 2, 3])
def test_every_lane_order(exe, tmp_path, case, seed):
    make, *rest = CASES[case]
    paths, want = _case(tmp_path, make(), *rest)
    got, st = _run(exe, tmp_path, paths, "walk", seed)
    assert got == want and sum(want) > 0
    assert st["clamped"] == 0 and st["unfinished"] == 0
    if case.startswith("few_roots"):  # a whole walk hands on what its few warps hold
        assert st["passes"] > 1 and st["listed"] > 32  # a unit for each of the chip's warps
        return
    if case == "grid_batch":
        return  # (more work than a limited walk does)
    got, st = _run(exe, tmp_path, paths, "limited", seed)
    assert got == want
    assert st["clamped"] == 0 and st["unfinished"] == 0
    if case != "edge_labels":
        assert st["passes"] > 1 and st["listed"] > 100


def test_depth_out_of_range_stays_in_bounds(exe, tmp_path):
    make, *rest = CASES["grid"]
    paths, _ = _case(tmp_path, make(), *rest)
    _, st = _run(exe, tmp_path, paths, "poison", 1)
    assert st["listed"] > 100 and st["clamped"] > 0


def test_a_full_list(exe_short_list, tmp_path):
    """A whole walk whose list has no room keeps its work; a limited one says
    that it has not finished."""
    make, *rest = CASES["few_roots"]
    paths, want = _case(tmp_path, make(), *rest)
    got, st = _run(exe_short_list, tmp_path, paths, "walk", 1)
    assert got == want and st["unfinished"] == 0 and st["clamped"] == 0
    _, st = _run(exe_short_list, tmp_path, paths, "limited", 1)
    assert st["unfinished"] == 1 and st["clamped"] == 0


@pytest.mark.parametrize("case", ["grid", "few_roots", "ba"])
def test_totals_in_parts(exe, exe_spill, tmp_path, case):
    """A call's totals are the same however often a lane's are added to them."""
    make, *rest = CASES[case]
    paths, want = _case(tmp_path, make(), *rest)
    got, st = _run(exe, tmp_path, paths, "walk", 1)
    parts, sp = _run(exe_spill, tmp_path, paths, "walk", 1)
    assert got == parts == want
    for k in ("candidates", "kept", "bytes", "front"):
        assert st[k] == sp[k] > 0
