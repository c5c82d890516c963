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
    knob(0)
    gg.graph_retune(g)
    layout = free() - held
    knob(2)
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


def star(ctx, n):
    leaves = np.arange(1, n, dtype=np.uint32)
    return ctx.from_edges(n, np.zeros_like(leaves), leaves)


FROM = 3 << 23  # edges from which the default asks for the blocked gather
GRAPHS = {  # what the rule looks at: shared sectors, few vertices, few edges
    "er": (lambda ctx: ctx.er(1 << 20, 26.0, seed=3, symmetric=False), True),
    "rmat": (lambda ctx: ctx.rmat(20, 15 << 20, seed=3), True),
    "grid": (lambda ctx: ctx.grid(2600, 2600, seed=3), False),
    "star": (lambda ctx: star(ctx, (FROM >> 1) + 10), False),
    "dense": (lambda ctx: ctx.er(50000, 520.0, seed=3, symmetric=False), False),
    "fewer": (lambda ctx: ctx.er(1 << 20, 23.0, seed=3, symmetric=False), False),
}


@pytest.mark.parametrize("kind", list(GRAPHS))
@pytest.mark.parametrize("fmt,acc64", [(gg.F32, True), (gg.BF16, False)])
def test_default_takes_the_faster_gather(ctx, knob, kind, fmt, acc64):
    make, blocks = GRAPHS[kind]
    g = make(ctx)
    assert (g.m >= FROM) == (kind != "fewer")
    k, st = 16, gg.RunStats()
    run = dict(maxiter=k, tol=-1.0, contrib=fmt, accum_f64=acc64)
    knob(0)
    rows = g.pagerank(stats=st, **run)
    by_rows = st.kernels
    knob(1)
    g.pagerank(**run)
    got = g.pagerank(stats=st, **run)
    assert st.kernels - by_rows == (k * (BLOCKS - ROWS[0 if by_rows > 2.5 * k else 1]) if blocks else 0)
    # double sums: eight roundings an iteration; float ones of 16-bit values: those of a step of the format
    np.testing.assert_allclose(got, rows, rtol=k * 8 * 2.0 ** -24 if acc64 else 2.0 ** -8, atol=0)
    g.close()


def test_layout_waits_for_iterations_that_are_run(ctx, knob):
    """A tolerance met after a few of the iterations allowed does not build the
    layout; runs do, once they have come to 16 iterations together, and a run
    without a tolerance that takes as many."""
    g = ctx.er(1 << 20, 26.0, seed=3, symmetric=False)
    st = gg.RunStats()

    def kernels(k, **run):
        g.pagerank(stats=st, host=False, **run)
        g.pagerank_iters = st.iterations
        return (st.kernels - 3) / k  # per iteration enqueued

    knob(0)
    assert kernels(100, maxiter=100, tol=1e-2) < BLOCKS
    few = g.pagerank_iters
    assert few < 8
    knob(1)
    done = few
    while done < 16:
        assert kernels(100, maxiter=100, tol=1e-2) < BLOCKS
        done += few
    assert kernels(100, maxiter=100, tol=1e-2) >= BLOCKS
    g.close()

    for parts in ((8, 7, 8), (15, 1), (16,)):
        g = ctx.er(1 << 20, 26.0, seed=3, symmetric=False)
        for k in parts[:-1]:
            assert kernels(k, maxiter=k, tol=0.0) < BLOCKS, parts
        assert kernels(parts[-1], maxiter=parts[-1], tol=0.0) >= BLOCKS, parts
        x = g.pagerank(maxiter=10, tol=0.0)
        knob(0)
        np.testing.assert_allclose(x, g.pagerank(maxiter=10, tol=0.0), rtol=80 * 2.0 ** -24, atol=0)
        knob(1)
        g.close()


def test_run_that_builds_the_layout_reports_it(ctx, knob):
    g = ctx.er(1 << 20, 26.0, seed=3, symmetric=False)
    knob(2)
    first, next_ = gg.RunStats(), gg.RunStats()
    g.pagerank(maxiter=2, host=False, stats=first)
    g.pagerank(maxiter=2, host=False, stats=next_)
    assert next_.kernels == 3 + 2 * BLOCKS
    assert first.kernels >= next_.kernels + 5  # counts, scans, row ends, the sorting pass
    assert first.total_ms > next_.total_ms
    g.close()
