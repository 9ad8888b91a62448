"""gs_support_count_noalloc's launch paths: four records a step and one at a
time (16-byte aligned arrays or not, record counts around multiples of four), a
warp and a block per key (rows of at most and more than 256 words)."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


def _call(gs, keys, gids, n_keys, n_graphs, out, stream):
    st = gs.lib().gs_support_count_noalloc(ctypes.c_void_p(keys.data_ptr()), ctypes.c_void_p(gids.data_ptr()),
                                           keys.numel(), n_keys, n_graphs, ctypes.c_void_p(out.data_ptr()),
                                           ctypes.c_void_p(stream))
    assert st == 0, gs.lib().gs_last_error()


def _want(torch, keys, gids, n_keys, n_graphs):
    ok = (keys >= 0) & (keys < n_keys) & (gids >= 0) & (gids < n_graphs)
    pairs = torch.unique(keys[ok].long() * n_graphs + gids[ok].long())
    return torch.bincount(torch.div(pairs, n_graphs, rounding_mode="floor"), minlength=n_keys).int()


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("n", [1, 3, 4, 5, 1023, 40001])
@pytest.mark.parametrize("n_graphs", [31, 8192, 8193])
def test_paths(gs, offset, n, n_graphs):
    torch = pytest.importorskip("torch")
    g = torch.Generator(device="cuda").manual_seed(n)
    keys = torch.randint(-2, 62, (n + offset,), generator=g, device="cuda", dtype=torch.int32)[offset:]
    gids = torch.randint(-9, n_graphs + 9, (n + offset,), generator=g, device="cuda", dtype=torch.int32)[offset:]
    out = torch.full((60,), -1, dtype=torch.int32, device="cuda")
    _call(gs, keys, gids, 60, n_graphs, out, torch.cuda.current_stream().cuda_stream)
    assert torch.equal(out, _want(torch, keys, gids, 60, n_graphs))

