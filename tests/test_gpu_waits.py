"""The bounded waits of the resident kernels: a grid-barrier wait that runs out
(limit 1 ns) ends the call with GG_ERR_TIMEOUT, without a trap or a hang, and
the context and the graph keep working."""
import numpy as np
import pytest

from graptor_b200 import gg
from oracle import oracle as O

pytestmark = pytest.mark.gpu

CALLS = {
    "bfs": lambda g: g.bfs_level(0),
    "bfs_multi": lambda g: gg.bfs_level_multi(g, np.array([0, 3], dtype=np.uint32)),
    "kcore": lambda g: g.kcore()[0],
    "msbfs": lambda g: gg.msbfs(g, np.array([0, 3], dtype=np.uint32)),
    "batch": lambda g: gg.batch_bfs_cc(g, np.array([0, 3], dtype=np.uint32))[1],
}


@pytest.fixture
def short_wait():
    old = gg.tuning_get("barrier_timeout_ns")
    yield lambda on: gg.tuning_set("barrier_timeout_ns", 1 if on else old)
    gg.tuning_set("barrier_timeout_ns", old)


def graph(kind):
    return O.rmat(15, 16 << 15, seed=8) if kind == "rmat" else O.grid(300, 311, seed=9, del_bp=200)


def runs_out(ctx, short_wait, kind, call):
    og = graph(kind)
    g = ctx.upload(og.off, og.adj)
    want = call(g)
    for _ in range(3):
        short_wait(True)
        with pytest.raises(gg.GGError) as e:
            call(g)
        assert e.value.status == gg.GG_ERR_TIMEOUT
        short_wait(False)
        assert np.array_equal(call(g), want)
    g.close()


@pytest.mark.parametrize("kind", ["rmat", "grid"])
@pytest.mark.parametrize("call", list(CALLS))
def test_wait_that_runs_out_is_reported(ctx, short_wait, kind, call):
    runs_out(ctx, short_wait, kind, CALLS[call])


@pytest.mark.parametrize("kind", ["rmat", "grid"])  # with the search, and hooking alone
def test_cc_wait_that_runs_out_is_reported(ctx, short_wait, kind):
    """Labels are not returned as good where any CTA of the run or of its
    search gave up, though the first one may have come through."""
    runs_out(ctx, short_wait, kind, lambda g: g.cc())
