"""Full dense pulls around the sizes at which rows change hands: settled by
the per-vertex record (three in-neighbours at most), put aside 32 at a time,
walked by a lane (8 edges) or by the warp, on vertex counts that leave the last
word and the last set of open rows ragged."""
import numpy as np
import pytest

from graptor_b200 import gg

pytestmark = pytest.mark.gpu


@pytest.fixture
def pull_first():
    old = gg.tuning_get("pull_first")
    yield
    gg.tuning_set("pull_first", old)


@pytest.mark.parametrize("records", [0, 1, 3, 4])
@pytest.mark.parametrize("n", [31, 33, 1000, 4133])
def test_full_pull_counts_and_levels(ctx, pull_first, n, records):
    gg.tuning_set("pull_first", records)
    rng = np.random.default_rng(n)
    deg = np.minimum(rng.choice([0, 1, 2, 3, 4, 7, 8, 9, 31, 40, 300], n), n - 1)
    dst = np.repeat(np.arange(n), deg)
    src = np.concatenate([(d + 1 + rng.permutation(n - 1)[:k]) % n for d, k in enumerate(deg)]).astype(np.int64)
    g = ctx.from_edges(n, src.astype(np.uint32), dst.astype(np.uint32), symmetrise=False)
    fin, fout = g.frontier(), g.frontier()
    active = rng.random(n) < 0.4
    fin.set_list(np.flatnonzero(active))
    hits = np.bincount(dst[active[src]], minlength=n)
    out_deg = np.bincount(src, minlength=n)
    # counting down to a floor of 3: every row is walked until it gets there
    count = rng.integers(0, 30, n).astype(np.uint32)
    a = g.prop(gg.U32)
    a.upload(count)
    g.edgemap(gg.EmapDesc(relax=gg.RELAX_COUNT_DOWN_U32, a=a.h, dst_filter=gg.FILTER_GT_CONST, dst_filter_k=3,
                          record=gg.RECORD_AT_FLOOR, variant=gg.VAR_PULL_DENSE), fin, fout)
    want = np.where(count > 3, np.maximum(3, count.astype(np.int64) - hits), count)
    down = (count > 3) & (want == 3)
    assert np.array_equal(a.download(), want)
    assert np.array_equal(np.sort(fout.download()), np.flatnonzero(down))
    assert fout.counts() == (int(down.sum()), int(out_deg[down].sum()))
    # a level: rows stop at their first active in-neighbour
    level, prev = g.prop(gg.I32), g.prop(gg.I32)
    lv = np.where(active, 0, n + 1).astype(np.int32)
    level.upload(lv)
    prev.upload(lv)
    g.edgemap(gg.EmapDesc(relax=gg.RELAX_MIN_PLUS1_I32, a=level.h, dst_filter=gg.FILTER_GT_CONST, dst_filter_k=1,
                          record=gg.RECORD_NE_PREV, prev=prev.h, variant=gg.VAR_PULL_DENSE), fin, fout)
    new = ~active & (hits > 0)
    assert np.array_equal(level.download(), np.where(new, 1, lv))
    assert np.array_equal(prev.download(), np.where(new, 1, lv))
    assert np.array_equal(np.sort(fout.download()), np.flatnonzero(new))
    g.close()
