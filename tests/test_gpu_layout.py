"""The blocked PageRank gather's layout as a thing that a graph holds: how much
memory it takes, when it is built and which gather runs with it."""
import numpy as np
import pytest

from graptor_b200 import gg

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

MB = 1 << 20
ROWS, BLOCKS = (3, 2), 4  # kernels per iteration: gather (+ heavy totals) + update; values, bins, spans, update


@pytest.fixture
def knob():
    old = gg.tuning_get("pr_blocked")
    yield lambda v: gg.tuning_set("pr_blocked", v)
    gg.tuning_set("pr_blocked", old)


def free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def local_sources(ctx, n, m, sources, seed=5):
    """m edges from the first `sources` ids to all."""
    rng = np.random.default_rng(seed)
    src = rng.integers(0, sources, m, dtype=np.uint32)
    dst = rng.integers(0, n, m, dtype=np.uint32)
    return ctx.from_edges(n, src, dst, symmetrise=False)


def test_layout_takes_its_chunks_and_goes_with_a_retune(ctx, knob):
    """512 source blocks of which one has edges: a chunk for every 8 edges of a
    bin, not one more for each of its 512 tiles (175 k chunks, 6 MB here)."""
    g = local_sources(ctx, 1 << 24, 8_000_000, 32768)
    knob(2)
    want = g.pagerank(maxiter=2)
    held = free()
    gg.graph_retune(g)
    layout = free() - held
    bins = -(-g.m // 24576)
    chunks = g.m // 8 + bins
    bound = 36 * chunks + bins * (768 * 4 + 8)
    assert bound - 4 * MB <= layout <= bound + 4 * MB, (layout / MB, bound / MB)
    np.testing.assert_allclose(g.pagerank(maxiter=2), want, rtol=1e-6, atol=0)
    assert abs(held - free()) <= 2 * MB
    g.close()


def test_a_new_graph_gets_the_memory_that_others_can_do_without(ctx, knob):
    """A graph that fits in what a layout and its values hold: they go, the
    ranks come back the same, and the layout once there is room again."""
    from test_gpu_memory import Fill
    g = ctx.er(1 << 16, 256.0, seed=4, symmetric=False)  # 75 MB of layout, 84 of values
    run = dict(maxiter=2, accum_f64=True)
    knob(0)
    rows = g.pagerank(**run)
    knob(2)
    st = gg.RunStats()
    want = g.pagerank(stats=st, **run)
    assert st.kernels >= BLOCKS * 2
    n = 1 << 20  # keys 17 MB, sorted 17, rows: 60 MB at its most
    src = np.arange(n, dtype=np.uint32)
    with Fill(16 * MB):
        h = ctx.from_edges(n, src, (src + 1) % n, symmetrise=False)
        assert h.m == n
        h.close()
    np.testing.assert_allclose(g.pagerank(**run), want, rtol=1e-6, atol=0)
    np.testing.assert_allclose(want, rows, rtol=1e-6, atol=0)
    g.close()
