"""Sparse pushes from frontiers around the sizes at which a warp takes one
source, several, or 32 of them (148 SMs x 8 CTAs x 8 warps take one each)."""
import numpy as np
import pytest

from graptor_b200 import gg
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 7, 8, 9, 33, 9471, 9472, 9473, 40000])
def test_push_from_small_sources(ctx, k):
    og = O.rmat(16, 3 << 16, seed=5)
    G = ctx.upload(og.off, og.adj, True)
    deg = np.diff(og.off.astype(np.int64))
    rng = np.random.default_rng(k)
    small = np.flatnonzero(deg <= 32)
    src = np.sort(rng.choice(small, k, replace=False)).astype(np.uint32)
    a, prev = G.prop(gg.U32), G.prop(gg.U32)
    fin, fout = G.frontier(), G.frontier()
    fin.set_list(src)
    a.upload(np.full(og.n, 0xFFFFFFFF, dtype=np.uint32))
    prev.upload(np.full(og.n, 0xFFFFFFFF, dtype=np.uint32))
    G.edgemap(gg.EmapDesc(relax=gg.RELAX_SETIF_U32, a=a.h, dst_filter=gg.FILTER_MSB_SET, record=gg.RECORD_NE_PREV,
                          prev=prev.h, variant=gg.VAR_PUSH_SPARSE), fin, fout)
    got = a.download()
    edge_src = np.repeat(np.arange(og.n), deg)
    active = np.zeros(og.n, dtype=bool)
    active[src] = True
    reached = np.zeros(og.n, dtype=bool)
    reached[og.adj[active[edge_src]]] = True
    assert np.array_equal(got != 0xFFFFFFFF, reached)
    # every taken value is an active in-neighbour of its vertex
    pairs = set(zip(edge_src[active[edge_src]].tolist(), og.adj[active[edge_src]].tolist()))
    assert all((int(got[d]), int(d)) in pairs for d in np.flatnonzero(reached))
    assert np.array_equal(np.sort(fout.download()), np.flatnonzero(reached))
    assert fout.counts() == (int(reached.sum()), int(deg[reached].sum()))
    G.close()


@pytest.mark.parametrize("deg", [1, 5, 40])
@pytest.mark.parametrize("k", [4095, 4096, 4097, 8193, 131073])
def test_push_where_warps_take_several(ctx, k, deg):
    """Sources per warp by what fills it: graphs of few edges, some and many a
    vertex, around the 4096 warps beyond which they count."""
    n = 140003
    src = np.repeat(np.arange(n), deg)
    dst = (src + 1 + np.arange(len(src)) % (deg * 7 + 1) * 3) % n
    G = ctx.from_edges(n, src.astype(np.uint32), dst.astype(np.uint32), symmetrise=False)
    rng = np.random.default_rng(k)
    active = np.zeros(n, dtype=bool)
    active[rng.choice(n, k, replace=False)] = True
    a, prev = G.prop(gg.U32), G.prop(gg.U32)
    fin, fout = G.frontier(), G.frontier()
    fin.set_list(np.flatnonzero(active))
    lab = rng.integers(0, 1 << 30, n).astype(np.uint32)
    a.upload(lab)
    prev.upload(lab)
    G.edgemap(gg.EmapDesc(relax=gg.RELAX_OR_U32, a=a.h, src=prev.h, prev=prev.h, record=gg.RECORD_NE_PREV,
                          variant=gg.VAR_PUSH_SPARSE), fin, fout)
    want = lab.copy()
    on = active[src]
    np.bitwise_or.at(want, dst[on], lab[src[on]])
    changed = np.flatnonzero(want != lab)
    assert np.array_equal(a.download(), want)
    assert np.array_equal(np.sort(fout.download()), changed)
    assert fout.counts() == (len(changed), int(np.bincount(src, minlength=n)[changed].sum()))
    G.close()
