"""Extension records of the column kernels (graphs of more than 256 vertices):
waves of few rows whose right-most path has a vertex of thousands of neighbours,
so that one warp writes most of the wave's records."""
import pytest

from conftest import run_oracle, to_lines

pytestmark = pytest.mark.gpu

_LEAVES = 3000


@pytest.fixture(scope="module")
def hubs(gs, tmp_path_factory):
    # a path 0-1-2-3 and leaves 4..7 at its end, in every graph, and there too
    # leaves of a label that no other graph has: every pattern with vertex 3 has
    # one row a graph, one tile, and that many extensions a row
    p = str(tmp_path_factory.mktemp("hubs") / "hubs.txt")
    with open(p, "w") as f:
        for g in range(32):
            f.write("t # %d\n" % g)
            f.writelines("v %d %d\n" % (v, v) for v in range(8))
            f.writelines("v %d %d\n" % (v, 100 + g) for v in range(8, 8 + _LEAVES))
            f.writelines("e %d %d 0\n" % (v, v + 1) for v in range(3))
            f.writelines("e 3 %d 0\n" % v for v in range(4, 8 + _LEAVES))
    db = gs.Database.load(p, "txt")
    db.upload()
    return p, db


def test_hub_lists(gs, oracle, hubs):
    p, db = hubs
    want = run_oracle(oracle, "txt", p, 20)
    gs.engine_reset()
    runs = [gs.mine(db, 20, label_style=gs.LABELS_SEQ, extension="lists") for _ in range(3)]
    for pats, _ in runs:
        assert to_lines(pats, gs) == want
    # the first run's records fit as well as the later ones': every node that
    # can join its parent's lists does
    joins = [st["join_nodes"] for _, st in runs]
    assert joins[0] == joins[1] == joins[2] > 0


def test_hub_default(gs, oracle, hubs):
    torch = pytest.importorskip("torch")
    p, db = hubs
    small = gs.Database.generate(1, scale=0.2)

    def held(d, s):
        # device memory that an engine holds after mining: its record buffers among it
        gs.engine_reset()
        free = torch.cuda.mem_get_info()[0]
        pats = [gs.mine(d, s, label_style=gs.LABELS_SEQ)[0] for _ in range(2)]
        assert pats[0] == pats[1]
        return free - torch.cuda.mem_get_info()[0], to_lines(pats[0], gs)

    small.upload()
    gs.set_pool_bytes(1 << 28)  # one chunk of embedding rows, the same for both
    try:
        base, _ = held(small, 20)
        used, lines = held(db, 20)
    finally:
        gs.set_pool_bytes(0)
        gs.engine_reset()
    assert lines == run_oracle(oracle, "txt", p, 20)
    # 2 M records of 16 bytes at most in a wave: the buffers that every engine begins with take them
    assert used - base < 64 << 20
