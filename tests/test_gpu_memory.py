"""Calls while the device memory is nearly used up: what cannot be had is an
error or another driver, never a wrong result, and the calls after it work."""
import numpy as np
import pytest

from graptor_b200 import gg
from oracle import oracle as O

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

MB = 1 << 20


class Fill:
    """Device memory held so that about `left` bytes stay free."""

    def __init__(self, left):
        self.held = []
        for size in (1 << k for k in range(34, 20, -1)):
            while torch.cuda.mem_get_info()[0] >= left + size:
                try:
                    self.held.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
                except torch.OutOfMemoryError:
                    break

    def __enter__(self):
        return self

    def __exit__(self, *a):
        self.held.clear()
        torch.cuda.empty_cache()


@pytest.fixture(scope="module", autouse=True)
def loaded(ctx):
    """Kernels are loaded on first use, which takes memory too."""
    g = ctx.rmat(10, 8 << 10, seed=1)
    old = gg.tuning_get("resident")
    for res in (1, 0):
        gg.tuning_set("resident", res)
        g.bfs_level(0), g.cc(), g.kcore(), g.pagerank(maxiter=2)
    gg.tuning_set("resident", old)
    g.close()


def test_an_error_is_reported_once(ctx):
    g = ctx.rmat(22, 1 << 22, seed=2)
    want = g.bfs_level(0)
    with Fill(8 * MB):
        with pytest.raises(gg.GGError) as e:
            g.prop(gg.F64)  # 32 MiB
        assert e.value.status == gg.GG_ERR_OOM
        assert np.array_equal(g.bfs_level(0), want)
    g.close()


@pytest.mark.parametrize("resident", [0, 1])
def test_buffers_that_fit_in_part(ctx, resident):
    """First calls with room for ever more of their buffers: the levels or
    GG_ERR_OOM, and the levels from the next call, whichever buffer was the
    one that did not fit (two frontiers of 50 MiB, two candidate lists, level
    and prev of 17 MiB each, 34 MiB of items)."""
    n = 1 << 22
    old = gg.tuning_get("resident")
    gg.tuning_set("resident", resident)
    try:
        want, kept = None, 0
        for left in range(4, 232, 12):
            g = ctx.rmat(22, n, seed=2)
            with Fill(left * MB):
                try:
                    kept = g.bfs_level(0)
                except gg.GGError as e:
                    assert e.status == gg.GG_ERR_OOM
                    kept = None
            got = g.bfs_level(0)
            want = got if want is None else want
            assert np.array_equal(got, want)
            assert kept is None or np.array_equal(kept, want), left
            g.close()
        assert kept is not None
        g = ctx.rmat(22, n, seed=2)
        off, adj = g.download()
        assert np.array_equal(want, O.bfs_level(O.Graph(n, off, adj), 0))
        g.close()
    finally:
        gg.tuning_set("resident", old)


@pytest.mark.parametrize("extra", [-30, 2, 8, 40])  # no items; no bitmaps or levels of the search; all of it
def test_cc_takes_the_other_driver_where_its_buffers_do_not_fit(ctx, extra):
    """A CC that had run in this memory runs in it still: the search's levels
    (17 MiB) or items (34 MiB) do not fit, label propagation does."""
    n = 1 << 22
    g = ctx.rmat(22, n, seed=3)
    old = gg.tuning_get("resident")
    try:
        gg.tuning_set("resident", 0)
        want = g.cc()
        gg.tuning_set("resident", 1)
        items = 8 * (n + g.m // 32 + g.m // 256 + 2 * (g.m // 4096) + 5)
        with Fill(items + 3 * n // 8 + extra * MB):
            for _ in range(2):
                assert np.array_equal(g.cc(), want)
        assert np.array_equal(g.cc(), want)
        assert np.array_equal(gg.batch_bfs_cc(g, np.array([0], dtype=np.uint32))[1], want)
    finally:
        gg.tuning_set("resident", old)
    g.close()
