"""Waves whose extension records do not fit their buffer, or that have none, make
their children by enumerating again: every instance of that materialise pass,
packed (6- and 8-bit ids, rows of one, two and five planes, a child's row in a
new plane) and on columns (8 to 32 pattern vertices, with the vertex set and
without), by two builds of the library: one whose record buffers begin with less
than any wave writes, and one whose buffers do not grow either."""
import json
import os
import random
import subprocess
import sys

import pytest

from conftest import REPO, run_oracle, to_lines

pytestmark = pytest.mark.gpu

_CHILD = """
import json, sys
import gpu_graph_mining_gb300 as g
g.LIB_PATH = sys.argv[1]
for path, s, me, kw in json.load(sys.stdin):
    db = g.Database.load(path, "txt")
    g.engine_reset()
    pats, st = g.mine(db, s, max_edges=me, label_style=g.LABELS_SEQ, **kw)
    print(json.dumps([[[g.code_to_string(c), n] for c, n in pats], st]), flush=True)
"""


def _write(path, graphs):
    with open(path, "w") as f:
        for i, (vl, edges) in enumerate(graphs):
            f.write("t # %d\n" % i)
            f.writelines("v %d %d\n" % x for x in enumerate(vl))
            f.writelines("e %d %d %d\n" % e for e in edges)


def _tree(r, n, vlabels, elabels):
    e = [(r.randrange(v), v) for v in range(1, n)]
    e += [(a, b) for a, b in (sorted(r.sample(range(n), 2)) for _ in range(n // 6)) if (a, b) not in e]
    return [r.randrange(vlabels) for _ in range(n)], [(a, b, r.randrange(elabels)) for a, b in sorted(set(e))]


def _alphabet(r):
    # labels of which few are frequent: too many label pairs for packed rows
    vl, e = _tree(r, r.randint(3, 24), 300, 40)
    vl = [x if r.random() < 0.5 else x % 3 for x in vl]
    return vl, [(a, b, x if max(vl[a], vl[b]) > 2 else 0) for a, b, x in e]


def _path(nv):
    # vertices that differ, and edges across the path: patterns of up to 27 vertices, with cycles
    return list(range(nv)), [(i, i + 1, 0) for i in range(nv - 1)] + [(i, i + 3, 1) for i in range(0, nv - 3, 24)]


# name: graphs, minsup, edge cap
_DBS = {
    "narrow": (lambda r: [_tree(r, r.randint(20, 64), 3, 2) for _ in range(40)], 15, 5),
    "narrow_long": (lambda r: [_path(48)] * 3, 2, 26),
    "wide": (lambda r: [_tree(r, r.randint(65, 200), 3, 2) for _ in range(20)], 15, 4),
    "wide_long": (lambda r: [_path(72)] * 3, 2, 26),
    "columns": (lambda r: [_tree(r, r.randint(257, 300), 3, 2) for _ in range(10)], 8, 4),
    "columns_long": (lambda r: [_path(60) if i else _tree(r, 257, 1, 1) for i in range(4)], 2, 26),
    "alphabet": (lambda r: [_alphabet(r) for _ in range(5000)], 40, 5),
}
_BUILDS = {"small": ["-DGS_REC_INIT=576"], "off": ["-DGS_REC_INIT=576", "-DGS_REC_MAX=576"]}


@pytest.fixture(scope="module")
def runs(gs, tmp_path_factory):
    """{(build, database, options): (lines, stats)} of both builds, and the databases' files"""
    from gpu_graph_mining_gb300 import build as b
    tmp = tmp_path_factory.mktemp("records")
    files = {}
    for i, (name, (graphs, _, _)) in enumerate(_DBS.items()):
        files[name] = str(tmp / (name + ".txt"))
        _write(files[name], graphs(random.Random(i)))
    jobs = [(n, kw) for n in _DBS for kw in ({}, {"wave_nodes": 1}, {"extension": "lists"})]
    objs = [os.path.join(b.OBJ, s + ".o") for s in b.CU_SRCS + b.CPP_SRCS if s != "gs_engine.cpp"]
    out = {}
    for build, flags in _BUILDS.items():
        obj, so = str(tmp / (build + ".o")), str(tmp / ("libgspan_gb300_%s.so" % build))
        b._run(["g++", "-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-I" + os.path.join(b.CUDA_HOME, "include"),
                "-c", os.path.join(b.CSRC, "gs_engine.cpp"), "-o", obj] + flags)
        b._run([b.NVCC] + b.ARCH + ["-shared", "-cudart", "static", "-o", so, obj] + objs +
               ["-Xlinker", "--exclude-libs,ALL", "-lpthread"])
        r = subprocess.run([sys.executable, "-c", _CHILD, so], cwd=REPO, text=True, capture_output=True, timeout=600,
                           input=json.dumps([(files[n], _DBS[n][1], _DBS[n][2], kw) for n, kw in jobs]))
        assert r.returncode == 0, r.stderr
        for (n, kw), line in zip(jobs, r.stdout.splitlines()):
            pats, st = json.loads(line)
            out[build, n, json.dumps(kw)] = ["%s\t%d" % tuple(p) for p in pats], st
    return files, out


@pytest.mark.parametrize("name", _DBS)
def test_reenumerated(gs, oracle, runs, name):
    files, out = runs
    _, s, me = _DBS[name]
    want = run_oracle(oracle, "txt", files[name], s, ["--max-edges", str(me)])
    assert len(want) > 50
    for (build, n, kw), (lines, _) in out.items():
        if n == name:
            assert lines == want, (build, kw)
    # one node a wave: all but the first are without records once the buffer may
    # not grow (4 bytes an extension less for the count kernel, 16 on columns)
    db = gs.Database.load(files[name], "txt")
    pats, st = gs.mine(db, s, max_edges=me, label_style=gs.LABELS_SEQ, wave_nodes=1)
    off = out["off", name, json.dumps({"wave_nodes": 1})][1]
    assert to_lines(pats, gs) == want and off["extensions"] == st["extensions"] and off["waves"] == st["waves"] > 10
    record = 16 if name.startswith(("columns", "alphabet")) else 4
    less = st["count_bytes"] - off["count_bytes"]
    assert 0.5 * record * st["extensions"] < less < record * st["extensions"]
