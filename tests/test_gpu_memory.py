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
