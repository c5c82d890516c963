"""Downloads into pageable and page-locked memory at the sizes where the path
changes: below and from 4 MiB on, pieces of 1 MiB with a ragged last one, fewer
and more pieces than copiers have slots."""
import numpy as np
import pytest

from graptor_b200 import gg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, (4 << 20) - 1, 4 << 20, (4 << 20) + 1, (6 << 20) + 12345, (41 << 20) + 7])
@pytest.mark.parametrize("pinned", [False, True])
def test_download_every_byte(ctx, n, pinned):
    torch = pytest.importorskip("torch")
    g = ctx.from_edges(n, np.zeros(0, np.uint32), np.zeros(0, np.uint32))
    p = g.prop(gg.U8)
    a = np.random.default_rng(n).integers(0, 256, n, dtype=np.uint8)
    p.upload(a)
    for _ in range(2):
        out = torch.zeros(n, dtype=torch.uint8, pin_memory=pinned).numpy()
        assert gg.lib().gg_prop_download(p.h, out.ctypes.data) == gg.GG_OK
        assert np.array_equal(out, a)
    g.close()


@pytest.mark.parametrize("k", [1, 7, 63, 64])
def test_msbfs_rows_packed(ctx, k):
    g = ctx.rmat(13, 16 << 13, seed=31)
    roots = np.arange(k, dtype=np.uint32) * 3
    lv = gg.msbfs(g, roots)
    for i in (0, k - 1):
        assert np.array_equal(lv[:, i], g.bfs_level(int(roots[i])))
    g.close()


def test_download_leaves_the_current_device(ctx):
    """From a context on another device than the thread's current one."""
    torch = pytest.importorskip("torch")
    if torch.cuda.device_count() < 2:
        pytest.skip("two devices")
    c = gg.Context(1)
    n = 6 << 20
    g = c.from_edges(n, np.zeros(0, np.uint32), np.zeros(0, np.uint32))
    p = g.prop(gg.U8)
    a = np.random.default_rng(n).integers(0, 256, n, dtype=np.uint8)
    p.upload(a)
    torch.cuda.set_device(0)
    for _ in range(2):
        assert np.array_equal(p.download(), a)
        assert torch.cuda.current_device() == 0
    c.close()


@pytest.mark.parametrize("n", [(8 << 20) - 1, 8 << 20, (8 << 20) + 1, (9 << 20) + 5])
def test_download_where_threads_take_over(ctx, n):
    g = ctx.from_edges(n, np.zeros(0, np.uint32), np.zeros(0, np.uint32))
    p = g.prop(gg.U8)
    a = np.random.default_rng(n).integers(0, 256, n, dtype=np.uint8)
    p.upload(a)
    for _ in range(3):
        assert np.array_equal(p.download(), a)
    g.close()
