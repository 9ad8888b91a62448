"""Mining under a limit of the embedding pool: where packed rows (32 bytes a row
from 9 pattern vertices on, 48 from 25) do not fit and columns do, the call
mines on columns instead of failing."""
import pytest

pytestmark = pytest.mark.gpu


def _brush(gs, tmp_path, graphs, path, leaves):
    """A path of so many labels, whose last vertex has leaves of one label."""
    p = str(tmp_path / ("brush%d_%d.txt" % (path, leaves)))
    with open(p, "w") as f:
        for g in range(graphs):
            f.write("t # %d\n" % g)
            f.writelines("v %d %d\n" % (v, min(v, path)) for v in range(path + leaves))
            f.writelines("e %d %d 0\n" % (v, v + 1) for v in range(path - 1))
            f.writelines("e %d %d 0\n" % (path - 1, v) for v in range(path, path + leaves))
    return gs.Database.load(p, "txt")


def _limited(gs, limit, call):
    gs.engine_reset()
    gs.set_pool_bytes(limit)
    try:
        return call()
    finally:
        gs.set_pool_bytes(0)
        gs.engine_reset()


# the subtree of the path's first edge: its prefixes, then two of 40 leaves (1,560 rows a
# graph); the whole takes 3.3 and 4.9 MB packed, 1.2 on columns
@pytest.mark.parametrize("path", [9, 25])
def test_columns_where_packed_rows_do_not_fit(gs, tmp_path, path):
    db = _brush(gs, tmp_path, 64, path, 40)
    kw = dict(max_edges=path + 2, root_part=0, root_parts=1000)
    want, st = gs.mine_collect(db, 32, **kw)
    got, sl = _limited(gs, 60000, lambda: gs.mine_collect(db, 32, **kw))
    assert got == want and len(want) == path + 2
    assert sl["patterns"] == st["patterns"] and sl["peak_pool_bytes"] < st["peak_pool_bytes"]
    # a call with room is on packed rows again
    again, sa = gs.mine_collect(db, 32, **kw)
    assert again == want and sa["peak_pool_bytes"] == st["peak_pool_bytes"]


# on columns from 1.3 MB on, on packed rows from 3.5
@pytest.mark.parametrize("schedulers", [1, 2])
def test_batch(gs, tmp_path, schedulers):
    dbs = [_brush(gs, tmp_path, 64, path, 40) for path in (9, 12, 9)]
    kw = dict(max_edges=11, root_part=0, root_parts=1000, schedulers=schedulers)
    want, _ = gs.mine_batch(dbs, [32] * 3, **kw)
    got, st = _limited(gs, 2300000, lambda: gs.mine_batch(dbs, [32] * 3, **kw))
    assert got == want and st["patterns"] == sum(len(w) for w in want)


def test_limit_that_neither_fits(gs, tmp_path):
    db = _brush(gs, tmp_path, 64, 9, 40)
    with pytest.raises(gs.GSpanError) as e:
        _limited(gs, 1, lambda: gs.mine_collect(db, 32, max_edges=11, root_part=0, root_parts=1000))
    assert e.value.status == 5
    emitted = []
    gs.mine(db, 32, max_edges=3, collect=False, sink=lambda code, sup: emitted.append(code))
    assert emitted and len(set(emitted)) == len(emitted)


def test_server(gs, tmp_path):
    # up to 40,320 rows a graph for a pattern: mined on columns from 433 MB on, on packed rows from 450
    db = _brush(gs, tmp_path, 64, 9, 8)
    small = gs.Database.generate(1, scale=1.0)
    want, _ = gs.mine_collect(db, 32)
    other, _ = gs.mine_collect(small, 60)
    with gs.Server(max_active=1, pool_bytes=436000000) as srv:
        a, b = srv.add_db(db), srv.add_db(small)
        rids = [srv.submit(b, 60), srv.submit(a, 32), srv.submit(b, 60)]
        res = [srv.result(r) for r in rids]
    assert [i["state"] for _, i in res] == [gs.REQ_DONE] * 3
    assert res[1][0] == want and res[0][0] == res[2][0] == other


def test_neighbour_blocks_make_room(gs):
    # a second database fits beside the first one, but not beside its neighbour
    # blocks: those are given up, and the first is mined on columns
    torch = pytest.importorskip("torch")
    gs.engine_reset()
    a, b, c = (gs.Database.generate(5, seed=s, scale=0.25) for s in (1, 2, 2))
    s = int(0.02 * len(a))
    a.upload()
    want_a, want_b = (gs.mine_collect(d, s, max_edges=4)[0] for d in (a, c))
    c.free()
    info = a.info()
    blocks = 32 * (info["vertices"] + info["adjacency_entries"] // 7 + 256)
    base = info["device_bytes"] - blocks
    assert base > 0.5 * blocks > 64 << 20
    gs.engine_reset()
    torch.cuda.empty_cache()
    room = int(base - 0.4 * min(base, blocks))
    hold = torch.empty(torch.cuda.mem_get_info()[0] - room, dtype=torch.uint8, device="cuda")
    try:
        b.upload()
        assert a.info()["device_bytes"] == base
    finally:
        del hold
        torch.cuda.empty_cache()
    for d, want in ((a, want_a), (b, want_b)):
        assert gs.mine_collect(d, s, max_edges=4)[0] == want
    gs.engine_reset()
