"""The resident BFS against the oracle's levels and the other drivers' records:
rows at the item boundaries (32, 256 and 4096 edges), vertex counts that are
no multiple of a word or of 16 bytes of bits, pushes after pulls, frontiers
too large to list, hand-overs to the one-cluster kernel and back, and many
roots at once."""
import numpy as np
import pytest

from graptor_b200 import gg
from oracle import oracle as O

pytestmark = pytest.mark.gpu

KNOBS = ("resident", "graph_handoff", "small_frontier")


@pytest.fixture
def knobs():
    old = {k: gg.tuning_get(k) for k in KNOBS}
    yield
    for k, v in old.items():
        gg.tuning_set(k, v)


def graph(kind):
    if kind == "rows":  # hubs over common leaves, the leaves chained
        degs = [1, 31, 32, 33, 255, 256, 257, 4095, 4096, 4097, 9001]
        h = len(degs)
        edges = [(i, h + j) for i, d in enumerate(degs) for j in range(d)]
        edges += [(h + j, h + j + 1) for j in range(9100)]
        return O.from_edges(h + 9105, edges), True
    if kind == "rmat":
        og = O.rmat(13, 16 << 13, seed=91)
        perm = np.random.default_rng(5).permutation(og.n)  # ids in no order of degree
        src = np.repeat(np.arange(og.n), np.diff(og.off.astype(np.int64)))
        return O.from_edges(og.n, list(zip(perm[src].tolist(), perm[og.adj].tolist()))), True
    if kind == "er_directed":
        return O.er(10007, 6.0, seed=92, dangling_bp=200, symmetric=False), False
    return O.grid(61, 83, seed=93, del_bp=300), True


def records(st):
    k = min(st.iterations, gg.MAX_ITERS)
    return (st.iterations, [st.nactv[i] for i in range(k)], [st.nacte[i] for i in range(k)],
            [st.variant[i] for i in range(k)], st.edges_reached, st.vertices_reached)


@pytest.mark.parametrize("kind", ["rows", "rmat", "er_directed", "grid"])
def test_resident_equals_other_drivers(ctx, knobs, kind):
    og, sym = graph(kind)
    g = ctx.upload(og.off, og.adj, symmetric=sym)
    deg = og.outdeg()
    roots = [int(np.argmax(deg)), int(np.flatnonzero(deg)[-1]), og.n - 1]
    for threshold, k in ((gg.THRESH_DEFAULT, 0), (gg.THRESH_FRAC, 1), (gg.THRESH_ALWAYS_SPARSE, 0),
                         (gg.THRESH_ALWAYS_DENSE, 0)):
        opts = gg.default_opts(threshold, k)
        for r in roots:
            want = O.bfs_level(og, r)
            rec = {}
            for res in (0, 1):
                gg.tuning_set("resident", res)
                st = gg.RunStats()
                assert np.array_equal(g.bfs_level(r, opts=opts, stats=st), want), (kind, threshold, r, res)
                rec[res] = records(st)
            assert rec[0] == rec[1], (kind, threshold, r)
    g.close()


@pytest.mark.parametrize("kind", ["rows", "rmat", "er_directed", "grid"])
def test_resident_hand_over_and_back(ctx, knobs, kind):
    og, sym = graph(kind)
    g = ctx.upload(og.off, og.adj, symmetric=sym)
    r = int(np.flatnonzero(og.outdeg())[-1])
    want = O.bfs_level(og, r)
    gg.tuning_set("resident", 1)
    gg.tuning_set("small_frontier", 0)
    st = gg.RunStats()
    assert np.array_equal(g.bfs_level(r, stats=st), want)
    ref = records(st)
    gg.tuning_set("small_frontier", 1)
    for h in (1, 2, 5):
        gg.tuning_set("graph_handoff", h)
        assert np.array_equal(g.bfs_level(r, stats=st), want), (kind, h)
        assert records(st) == ref, (kind, h)
    g.close()


@pytest.mark.parametrize("kind", ["rows", "rmat", "er_directed", "grid"])
@pytest.mark.parametrize("k", [1, 33, 2000])
def test_resident_many_roots(ctx, knobs, kind, k):
    og, sym = graph(kind)
    g = ctx.upload(og.off, og.adj, symmetric=sym)
    roots = np.random.default_rng(k).choice(og.n, min(k, og.n), replace=False).astype(np.uint32)
    gg.tuning_set("resident", 0)
    want = gg.bfs_level_multi(g, roots)
    gg.tuning_set("resident", 1)
    assert np.array_equal(gg.bfs_level_multi(g, roots), want)
    if k == 1:
        assert np.array_equal(want, O.bfs_level(og, int(roots[0])))
    g.close()
