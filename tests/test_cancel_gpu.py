"""Cancelling requests while others are mined: memory of a cancelled request goes
to the others only when nothing queued for it can write it any more."""
import pytest

pytestmark = pytest.mark.gpu


def _wait_admitted(srv):
    while srv.stats()["queued"]:
        pass


def test_cancelled_at_once_beside_another(gs):
    # a request cancelled as soon as it runs: its root phase may still be queued
    # behind the other's waves when its memory is given back
    big = gs.Database.generate(5, scale=0.1)
    small = gs.Database.generate(2, scale=0.2)
    s = int(0.005 * len(big))
    want, _ = gs.mine_collect(big, s, max_edges=8)
    with gs.Server(max_active=8) as srv:
        a, b = srv.add_db(big), srv.add_db(small)
        for _ in range(3):
            rid = srv.submit(a, s, 8)
            _wait_admitted(srv)
            cancelled = []
            while srv.status(rid) is None and len(cancelled) < 200:
                c = srv.submit(b, max(2, int(0.02 * len(small))), 4)
                _wait_admitted(srv)
                srv.cancel(c)
                cancelled.append(c)
            pats, info = srv.result(rid)
            for c in cancelled:
                assert srv.result(c)[1]["state"] in (gs.REQ_CANCELLED, gs.REQ_DONE)
            assert info["state"] == gs.REQ_DONE and pats == want
