"""Packed rows (graphs of at most 256 vertices) against the oracle and against
the column kernels: neighbour lists that end at and past their 8-entry blocks,
databases on either side of the rule that chooses the row format, batches of
both, and the re-enumerating materialise after a record overflow."""
import random

import pytest

from conftest import run_oracle, to_lines

pytestmark = pytest.mark.gpu


def _write(path, graphs):
    """graphs: (vertex labels, [(a, b, edge label)])"""
    with open(path, "w") as f:
        for i, (vl, edges) in enumerate(graphs):
            f.write("t # %d\n" % i)
            f.writelines("v %d %d\n" % x for x in enumerate(vl))
            f.writelines("e %d %d %d\n" % e for e in edges)


def _lines(gs, db, s, **kw):
    return to_lines(gs.mine(db, s, label_style=gs.LABELS_SEQ, **kw)[0], gs)


# a list of d entries: one block up to 8, then 7 and a continuation (8 again, or 7 and another)
@pytest.mark.parametrize("degree", [1, 7, 8, 9, 15, 16, 22, 23, 62, 63])
def test_list_lengths(gs, oracle, tmp_path, degree):
    r = random.Random(degree)
    graphs = []
    for g in range(6):
        # a hub with `degree` leaves and some edges between them; the leaves' labels decide
        # where in the hub's sorted list an entry stands
        vl = [0] + [r.randrange(1, 5) for _ in range(degree)]
        edges = [(0, v, r.randrange(3)) for v in range(1, degree + 1)]
        edges += [(v, v + 1, r.randrange(3)) for v in range(1, degree) if r.random() < 0.3]
        graphs.append((vl, edges))
    p = str(tmp_path / "hub.txt")
    _write(p, graphs)
    db = gs.Database.load(p, "txt")
    want = run_oracle(oracle, "txt", p, 4, ["--max-edges", "3"])
    assert _lines(gs, db, 4, max_edges=3) == want
    # the same from host arrays converted on the device
    q = str(tmp_path / "hub.cudabin")
    db.write(q, "cudabin")
    import numpy as np
    raw = np.fromfile(q, dtype=np.int32)
    n, esz, maxv = (int(x) for x in raw[:3])
    cuts = np.cumsum([4, esz, esz, n * maxv, n * maxv + 1])
    e, el, vl, vo = (raw[a:b] for a, b in zip(cuts[:-1], cuts[1:]))
    dev = gs.Database.from_arrays(n, maxv, e, el, vl, vo, device=True)
    assert _lines(gs, dev, 4, max_edges=3) == want


def _random_graphs(r, count, nv, vlabels, elabels):
    graphs = []
    for _ in range(count):
        n = r.randint(*nv)
        edges = {(r.randrange(v), v) for v in range(1, n)}
        for _ in range(n // 4):
            a, b = sorted(r.sample(range(n), 2))
            edges.add((a, b))
        graphs.append(([r.randrange(vlabels) for _ in range(n)], [(a, b, r.randrange(elabels)) for a, b in sorted(edges)]))
    return graphs


# one label (no label bits), alphabets of powers of two and one more, and one whose label pairs
# are too many for the 4-byte entries and items (mined on columns)
@pytest.mark.parametrize("vlabels,elabels,count", [(1, 1, 30), (2, 4, 60), (32, 3, 200), (33, 3, 200), (300, 40, 2500)])
def test_alphabets(gs, oracle, tmp_path, vlabels, elabels, count):
    r = random.Random(vlabels)
    p = str(tmp_path / "db.txt")
    _write(p, _random_graphs(r, count, (3, 24), vlabels, elabels))
    s = max(2, count // 10) if vlabels <= 33 else 3
    want = run_oracle(oracle, "txt", p, s, ["--max-edges", "4"])
    assert _lines(gs, gs.Database.load(p, "txt"), s, max_edges=4) == want


def test_batch_of_both_formats(gs, tmp_path):
    r = random.Random(3)
    dbs = []
    for i, nv in enumerate([(4, 20), (60, 64), (60, 90), (4, 30), (66, 70)]):
        p = str(tmp_path / ("b%d.txt" % i))
        _write(p, _random_graphs(r, 40, nv, 3, 2))
        dbs.append(gs.Database.load(p, "txt"))
    sups = [12, 25, 25, 10, 25]
    got, _ = gs.mine_batch(dbs, sups, max_edges=4)
    for db, s, pats in zip(dbs, sups, got):
        assert pats == gs.mine(db, s, max_edges=4)[0]
        # the lists strategy mines every database on columns
        assert pats == gs.mine(db, s, max_edges=4, extension="lists")[0]


def test_record_overflow(gs):
    # the first waves of a fresh engine write more extension items than its
    # record buffer holds (they are enumerated again); small waves never do
    db = gs.Database.generate(5, scale=0.25)
    s = int(0.01 * len(db))
    gs.engine_reset()
    first, _ = gs.mine_collect(db, s)
    again, _ = gs.mine_collect(db, s)
    small, _ = gs.mine_collect(db, s, wave_rows=1 << 20)
    assert first == again == small
    gs.engine_reset()


@pytest.mark.parametrize("kw", [{}, {"launch_mode": 1}, {"serial": 1}, {"min_check": 1}, {"extension": "lists"}])
def test_more_results_than_room(gs, kw):
    # a fresh engine has room for 4,096 selected candidates per wave in pinned
    # memory (the rest of a larger wave's come by a second copy); waves of 64
    # nodes never fill it
    db = gs.Database.generate(1, scale=1.0)
    s = 2
    gs.engine_reset()
    small, _ = gs.mine_collect(db, s, wave_nodes=64, max_edges=7)
    gs.engine_reset()
    large, st = gs.mine_collect(db, s, max_edges=7, **kw)
    assert st["candidates"] > 4 * 4096 and large == small
    # one wave after another: the kernels' stamped times fit in the call
    if kw.get("serial"):
        parts = [st[k] for k in ("count_ms", "sel_ms", "min_ms", "mat_ms", "root_ms")]
        assert min(parts) > 0 and sum(parts) <= st["wall_ms"]
    gs.engine_reset()


def test_nodes_reused_across_formats(gs, tmp_path):
    # the engine keeps its DFS-tree nodes between runs: packed and column runs
    # of different depth, one after the other, take each other's nodes
    r = random.Random(11)
    small, large = str(tmp_path / "s.txt"), str(tmp_path / "l.txt")
    _write(small, _random_graphs(r, 60, (10, 40), 2, 2))
    _write(large, _random_graphs(r, 40, (66, 80), 2, 2))
    a, b = gs.Database.load(small, "txt"), gs.Database.load(large, "txt")
    runs = [(a, 30, {"max_edges": 6}), (b, 30, {"max_edges": 4}), (a, 30, {"max_edges": 6, "extension": "lists"}),
            (a, 20, {"max_edges": 4, "wave_nodes": 7})]
    gs.engine_reset()
    want = [gs.mine(d, s, **kw)[0] for d, s, kw in runs]
    for (d, s, kw), pats in list(zip(runs, want))[::-1]:
        assert gs.mine(d, s, **kw)[0] == pats
    assert want[0] == want[2]


def _shape(name):
    """One pattern family per graph: its edges, and a label per vertex."""
    kind, n, labels = name
    if kind == "path":
        e = [(i, i + 1) for i in range(n - 1)]
    elif kind == "cycle":
        e = [(i, (i + 1) % n) for i in range(n)]
    else:
        e = [(i, j) for i in range(n) for j in range(i + 1, n)]
    return [i % labels for i in range(n)], [(a, b, 0) for a, b in e]


# the canonicality kernel's edges: one pass of 32 directed edges and several (past 16 edges),
# up to its 32 vertices and past them, backward edges, and embeddings that outgrow its buffer
# (6 vertices all joined, one label: 720), each against the host's check and the oracle
@pytest.mark.parametrize("shape", [("path", 17, 1), ("path", 18, 3), ("path", 32, 2), ("path", 34, 1), ("cycle", 9, 3),
                                   ("cycle", 32, 1), ("cycle", 33, 1), ("complete", 5, 1), ("complete", 6, 1)])
def test_canonicality(gs, oracle, tmp_path, shape):
    p = str(tmp_path / "shape.txt")
    _write(p, [_shape(shape)] * 3)
    db = gs.Database.load(p, "txt")
    got = _lines(gs, db, 2)
    assert got == _lines(gs, db, 2, min_check=1)
    assert got == run_oracle(oracle, "txt", p, 2)


# graph-local ids of 6 bits (up to 64 vertices), of 8 (up to 256), and columns beyond; rows of one, two
# and five planes; the hub's list has up to 37 blocks
@pytest.mark.parametrize("nv", [64, 65, 128, 255, 256, 257])
def test_graph_sizes(gs, oracle, tmp_path, nv):
    r = random.Random(nv)
    p = str(tmp_path / "sizes.txt")
    hub = [(0, v, r.randrange(3)) for v in range(1, nv)] + [(v, v + 1, 0) for v in range(1, nv - 1, 5)]
    graphs = _random_graphs(r, 9, (nv - 3, nv), 4, 3) + [([0] + [r.randrange(1, 5) for _ in range(nv - 1)], hub)] * 3
    _write(p, graphs)
    db = gs.Database.load(p, "txt")
    want = run_oracle(oracle, "txt", p, 3, ["--max-edges", "3"])
    assert _lines(gs, db, 3, max_edges=3) == want
    # a path of vertices that differ, and edges across it
    n = nv // 4 * 4
    path = [(i, i + 1, 0) for i in range(n - 1)] + [(i, i + 3, 1) for i in range(0, n - 3, 40)]
    _write(p, [(list(range(n)), path)] * 3)
    want = run_oracle(oracle, "txt", p, 2, ["--max-edges", "26"])
    assert _lines(gs, gs.Database.load(p, "txt"), 2, max_edges=26) == want


def test_batch_of_id_widths(gs, tmp_path):
    r = random.Random(5)
    dbs = []
    for i, nv in enumerate([(4, 20), (60, 64), (65, 90), (250, 256), (257, 260), (4, 30)]):
        p = str(tmp_path / ("w%d.txt" % i))
        _write(p, _random_graphs(r, 40, nv, 3, 2))
        dbs.append(gs.Database.load(p, "txt"))
    sups = [12, 25, 25, 30, 30, 10]
    for kw in ({}, {"launch_mode": 1}):
        got, _ = gs.mine_batch(dbs, sups, max_edges=4, **kw)
        for db, s, pats in zip(dbs, sups, got):
            assert pats == gs.mine(db, s, max_edges=4)[0]
            assert pats == gs.mine(db, s, max_edges=4, extension="lists")[0]


# selection in one kernel (waves of up to 2^21 bitmap words) and in two, by graph replay and direct
# launches; keys of at most 256 words and of more
@pytest.mark.parametrize("launch_mode", [0, 1])
def test_selection_forms(gs, launch_mode):
    db = gs.Database.generate(5, scale=0.2)
    s = int(0.01 * len(db))
    large, sl = gs.mine_collect(db, s, launch_mode=launch_mode)
    small, ss = gs.mine_collect(db, s, launch_mode=launch_mode, wave_words=1 << 20)
    assert large == small and len(large) > 500
    # waves limited to 2^20 words take one kernel less each
    assert sl["launches"] / sl["waves"] > ss["launches"] / ss["waves"]
