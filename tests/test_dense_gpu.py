"""Counting nodes with many rows a graph: their bitmap words are read before a bit is
set.  Rows around the line of that rule, packed rows of one, two and five planes and
of 6- and 8-bit ids, columns, graphs over several bitmap words, against the oracle."""
import pytest

from conftest import run_oracle, to_lines

pytestmark = pytest.mark.gpu


def _broom(path, leaves, size):
    # a path of labels that differ, at its end so many leaves of one label, at every
    # third leaf a vertex more; isolated vertices up to the size
    vl = list(range(path)) + [path] * leaves
    e = [(v, v + 1, 0) for v in range(path - 1)] + [(path - 1, path + v, 0) for v in range(leaves)]
    for v in range(0, leaves, 3):
        e.append((path + v, len(vl), 1))
        vl.append(path + 1)
    return vl + [0] * (size - len(vl)), e


# path: rows of one, two and five planes where the leaves begin; leaves: rows a graph of the
# node that ends in one, the line is at 16
@pytest.mark.parametrize("size", [0, 70, 300])
@pytest.mark.parametrize("path", [2, 8, 24])
@pytest.mark.parametrize("leaves", [15, 16, 17])
def test_rows_a_graph(gs, oracle, tmp_path, path, leaves, size):
    p = str(tmp_path / "brooms.txt")
    graphs = 70
    with open(p, "w") as f:
        for g in range(graphs):
            # every third graph ends before the leaves
            vl, e = _broom(path, leaves, size)
            e = e[:path - 1] if g % 3 == 1 else e
            f.write("t # %d\n" % g)
            f.writelines("v %d %d\n" % x for x in enumerate(vl))
            f.writelines("e %d %d %d\n" % x for x in e)
    db = gs.Database.load(p, "txt")
    # the subtree of the path's first edge
    me = path + 1
    want = run_oracle(oracle, "txt", p, 30, ["--max-edges", str(me), "--roots", "0/1000"])
    for opts in ({}, {"wave_nodes": 1}, {"extension": "lists"}):
        pats, _ = gs.mine(db, 30, max_edges=me, root_part=0, root_parts=1000, label_style=gs.LABELS_SEQ, **opts)
        assert to_lines(pats, gs) == want
