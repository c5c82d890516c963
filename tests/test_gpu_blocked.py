"""The PageRank gather by blocks of sources against the gather by rows: rows
around the lengths at which a bin's sums change hands (4 lanes, the warp at
256 edges, pieces at 1024, the next bin at 24576), rows that fill bins
exactly, several source blocks (32768 ids), and a last block, bin and chunk
that are not full."""
import numpy as np
import pytest

from graptor_b200 import gg
from oracle import oracle as O

pytestmark = pytest.mark.gpu

LENGTHS = [1, 3, 4, 5, 7, 8, 9, 255, 256, 257, 1023, 1024, 1025, 2049, 24575, 24576, 24577, 50000, 60001]
KNOB = "pr_blocked"


@pytest.fixture
def knob():
    old = gg.tuning_get(KNOB)
    yield
    gg.tuning_set(KNOB, old)


def edges(kind, rng):
    if kind == "short":  # a row ends every few edges; more rows than edges in places
        n = 40003
        deg = rng.integers(0, 6, n)
        deg[5000:9000] = 0
    elif kind == "lengths":
        n = 70001
        deg = np.zeros(n, dtype=np.int64)
        deg[rng.permutation(n)[: len(LENGTHS)]] = LENGTHS
        deg[-1] = 300
    elif kind == "full":  # rows that begin and end with bins, and rows of whole bins
        n = 65536
        deg = np.zeros(n, dtype=np.int64)
        deg[10:34] = 1024
        deg[40], deg[50], deg[60], deg[61] = 24576, 49152, 24000, 576
        deg[70] = 24577
    else:  # one bin and a single source block
        n = 999
        deg = rng.integers(0, 20, n)
    dst = np.repeat(np.arange(n), deg)
    if kind in ("lengths", "full"):
        src = np.concatenate([(d + 1 + rng.permutation(n - 1)[:k]) % n for d, k in enumerate(deg) if k])
    else:
        src = (dst + rng.integers(1, n, len(dst))) % n
    return n, src.astype(np.uint32), dst.astype(np.uint32)


@pytest.mark.parametrize("kind", ["short", "lengths", "full", "small"])
@pytest.mark.parametrize("fmt,acc64", [(gg.F32, True), (gg.F32, False), (gg.BF16, True), (gg.F16, False)])
def test_blocked_equals_row_gather(ctx, knob, kind, fmt, acc64):
    n, src, dst = edges(kind, np.random.default_rng(len(kind)))
    g = ctx.from_edges(n, src, dst, symmetrise=False)
    run = dict(contrib=fmt, accum_f64=acc64, tol=0.0)
    gg.tuning_set(KNOB, 0)
    want = g.pagerank(maxiter=1, **run).astype(np.float64)
    again = g.pagerank(maxiter=5, **run).astype(np.float64)
    gg.tuning_set(KNOB, 2)
    got = g.pagerank(maxiter=1, **run)
    # one iteration: the same terms summed in another order.  Double sums
    # round once to float, as do the three steps after it; float sums take at
    # most 200 additions one after the other on either side
    eps = 2.0 ** -24
    assert np.all(np.abs(got - want) <= want * eps * (8 if acc64 else 400))
    # then the contributions are rounded again each time: to 8 or 11 bits (a
    # float16 run whose contributions outgrow its range is NaN on both sides)
    rel = {gg.F32: 5 * 400 * eps, gg.BF16: 2.0 ** -8, gg.F16: 2.0 ** -10}[fmt]
    np.testing.assert_allclose(g.pagerank(maxiter=5, **run), again, rtol=rel, atol=0)
    g.close()


@pytest.mark.parametrize("fmt,acc64", [(gg.F32, True), (gg.F32, False), (gg.BF16, False)])
def test_rows_over_many_bins(ctx, knob, fmt, acc64):
    """Rows over 2 to 6 bins (summed by a lane up to 4) and over 33, 34, 129,
    130 and 300 (by a warp, 128 bins at a time), the first one from bin 0, with
    short rows before, between and after them."""
    rng = np.random.default_rng(11)
    n = 1 << 23
    bins = [300, 2, 3, 4, 5, 6, 33, 34, 129, 130]
    deg = np.zeros(n, dtype=np.int64)
    at = 0
    for k in bins:  # k - 1 whole bins and some edges before and after them
        deg[at] = (k - 1) * 24576 + 7
        deg[at + 1: at + 40] = rng.integers(1, 5, 39)
        at += 60
    dst = np.repeat(np.arange(n, dtype=np.int64), deg)
    first = np.repeat(np.cumsum(deg) - deg, deg)
    src = (dst + 1 + (np.arange(len(dst)) - first)) % n  # distinct within a row
    g = ctx.from_edges(n, src.astype(np.uint32), dst.astype(np.uint32), symmetrise=False)
    assert g.m == len(dst)
    run = dict(contrib=fmt, accum_f64=acc64, tol=0.0, maxiter=1)
    gg.tuning_set(KNOB, 0)
    want = g.pagerank(**run).astype(np.float64)
    gg.tuning_set(KNOB, 2)
    got = g.pagerank(**run)
    # the same terms in another order: double sums round once, float sums take
    # at most 32 + 5 + 24 + 4 + 300 / 32 + 5 + 1 additions one after the other by
    # blocks, and 1024 / 32 + 5 + 7200 / 32 + 5 by rows
    eps = 2.0 ** -24
    assert np.all(np.abs(got - want) <= want * eps * (8 if acc64 else 400))
    g.close()


@pytest.mark.parametrize("kind", ["short", "lengths", "full", "small"])
def test_knob_decides_which_gather_runs(ctx, knob, kind):
    """Told apart by their kernels: four per iteration by blocks, two or three
    (heavy rows) by rows."""
    n, src, dst = edges(kind, np.random.default_rng(len(kind)))
    g = ctx.from_edges(n, src, dst, symmetrise=False)
    st = gg.RunStats()
    for fmt, acc64 in ((gg.F32, True), (gg.F32, False), (gg.BF16, False), (gg.F16, False), (gg.CFP_6_10, False),
                       (gg.BF16_TRUNC, False)):
        for value, kernels in ((2, {4}), (0, {2, 3})):
            gg.tuning_set(KNOB, value)
            for _ in range(2):  # (the first also builds the layout)
                g.pagerank(maxiter=3, tol=0.0, contrib=fmt, accum_f64=acc64, host=False, stats=st)
            assert st.kernels - 3 in {3 * k for k in kernels}, (fmt, value)
    for fmt, acc64 in ((gg.F64, True), (gg.FP8E4M3, False)):  # never by blocks
        gg.tuning_set(KNOB, 2)
        g.pagerank(maxiter=3, tol=0.0, contrib=fmt, accum_f64=acc64, host=False, stats=st)
        assert st.kernels - 3 in (6, 9)
    g.close()


@pytest.mark.parametrize("blocked", [0, 2])
def test_both_gathers_give_the_references_ranks(ctx, knob, blocked):
    """PRv's answer by rows and by blocks, and PR_vary's with customfp<6,10>
    storage, as the row gather's tests have it."""
    og = O.rmat(15, 16 << 15, seed=9)
    g = ctx.upload(og.off, og.adj)
    gg.tuning_set(KNOB, blocked)
    st = gg.RunStats()
    xo, _, _ = O.pagerank(og, maxiter=20, tol=0)
    x = g.pagerank(maxiter=20, tol=0, stats=st)
    assert (st.kernels >= 3 + 20 * 4) == (blocked == 2)
    assert np.abs(x.astype(np.float64) - xo).sum() <= 1e-6
    xo, _, _ = O.pagerank_vary(og, O.CFP_6_10, accum_f64=False, maxiter=20, tol=0)
    x = g.pagerank(maxiter=20, tol=0, contrib=gg.CFP_6_10, accum_f64=False, renorm_f32=False)
    assert np.abs(x.astype(np.float64) - xo).sum() <= 1e-5
    g.close()
