"""The resident BFS and CC against the oracle and the other drivers' records:
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


def cc_graph(kind):
    rng = np.random.default_rng(7)
    if kind == "core_and_tail":
        # a dense core that the search reaches at once, and a path whose small
        # ids (0 at its far end) are farther than the search goes
        core = [(int(a), int(b)) for a, b in rng.integers(1000, 4000, (30000, 2)) if a != b]
        path = [(i, i + 1) for i in range(60)] + [(60, 1500)]
        return O.from_edges(4100, core + path)
    if kind == "giant_without_0":
        # vertex 0 in a small component; stars of 257 and 3000 leaves (rows
        # above the heavy-row threshold) outside the giant one
        core = [(int(a), int(b)) for a, b in rng.integers(5000, 13000, (60000, 2)) if a != b]
        stars = [(10, 20 + i) for i in range(257)] + [(15, 600 + i) for i in range(3000)]
        return O.from_edges(13100, core + stars + [(0, 4), (4, 1)])
    if kind == "many":
        # no giant component: stars, paths and cliques of growing size
        edges, at = [], 3
        for k in range(1, 40):
            edges += [(at + k, at + j) for j in range(k)] + [(at + k + j, at + k + j + 1) for j in range(37 * k)]
            at += 38 * k + 2
        edges += [(at, at + 1 + j) for j in range(1500)] + [(at + 2000, at + 1 + 2 * j) for j in range(700)]
        return O.from_edges(at + 2010, edges)
    return O.from_edges(77, [])


@pytest.mark.parametrize("kind", ["core_and_tail", "giant_without_0", "many", "edgeless"])
def test_resident_cc_exact(ctx, knobs, kind):
    og = cc_graph(kind)
    g = ctx.upload(og.off, og.adj)
    want = O.cc(og)
    for res in (0, 1):
        gg.tuning_set("resident", res)
        for _ in range(3):
            assert np.array_equal(g.cc(), want), (kind, res)
    lv, lb, _, _ = gg.batch_bfs_cc(g, np.array([0, 5], dtype=np.uint32))
    assert np.array_equal(lb, want)
    assert np.array_equal(lv, np.minimum(O.bfs_level(og, 0), O.bfs_level(og, 5)))
    g.close()


@pytest.mark.parametrize("kind", ["core_and_tail", "giant_without_0", "many", "edgeless", "star"])
def test_resident_cc_counts_the_edges_it_examines(ctx, knobs, kind):
    """scanned[0]: the search's edges (as a BFS of at most ten steps counts
    them) and, where it found no giant component, every vertex's first edge;
    scanned[1]: those of the rows that hook."""
    if kind == "star":
        og = O.from_edges(3001, [(7, i) for i in range(3001) if i != 7])
    else:
        og = cc_graph(kind)
    g = ctx.upload(og.off, og.adj)
    gg.tuning_set("resident", 1)
    st, bfs = gg.RunStats(), gg.RunStats()
    assert np.array_equal(g.cc(stats=st), O.cc(og))
    assert st.iterations == 2
    assert st.scanned_edges == st.scanned[0] + st.scanned[1]
    deg = og.outdeg()
    hub = int(np.argmax(deg))
    level = g.bfs_level(hub, stats=bfs)
    searched = int(deg[hub]) * (og.m / og.n) ** 2 >= 1024 if og.n else False
    giant = 2 * int((level <= og.n).sum()) >= int((deg > 0).sum())
    if kind == "star":  # the search reaches all of it: nothing left to hook
        assert searched and bfs.iterations <= 10
        assert (st.scanned[0], st.scanned[1]) == (bfs.scanned_edges, 0)
    elif kind == "edgeless":
        assert (st.scanned[0], st.scanned[1]) == (0, 0)
    elif not giant:  # (the hub of giant_without_0 is a star's): every edge is looked at
        assert st.scanned[1] == og.m
        assert st.scanned[0] >= int((deg > 0).sum())
    else:
        # rows outside the part reached (the search may stop before its end)
        out = int(deg[level > og.n].sum())
        assert searched and out <= st.scanned[1] < og.m // 2
        assert 0 < st.scanned[0] <= bfs.scanned_edges
    g.close()


def test_huge_rows_are_listed_together(ctx, knobs):
    """Rows of 1 to 40 huge items, many in one warp, beside rows with long and
    short items: BFS (the hubs are one level) and k-core."""
    rng = np.random.default_rng(12)
    hubs, n = 70, 200000
    deg = [int(d) for d in rng.choice([3, 40, 300, 4096, 4097, 8192, 8193, 40000, 163840, 163841], hubs)]
    src = np.repeat(np.arange(1, hubs + 1), deg)
    dst = np.concatenate([hubs + 1 + rng.permutation(n - hubs - 1)[:d] for d in deg])
    src = np.concatenate([src, np.zeros(hubs, dtype=np.int64)])
    dst = np.concatenate([dst, np.arange(1, hubs + 1)])
    g = ctx.from_edges(n, src.astype(np.uint32), dst.astype(np.uint32))
    off, adj = g.download()
    og = O.Graph(n, off, adj)
    for threshold in (gg.THRESH_DEFAULT, gg.THRESH_ALWAYS_SPARSE):
        for r in (0, 1, n - 1):
            assert np.array_equal(g.bfs_level(r, opts=gg.default_opts(threshold)), O.bfs_level(og, r))
    st = gg.RunStats()
    core, largest = g.kcore(stats=st)
    want, wl = g.kcore(opts=gg.default_opts(gg.THRESH_ALWAYS_SPARSE, collect=True))  # host-driven
    assert np.array_equal(core, want) and largest == wl
    assert np.array_equal(g.cc(), O.cc(og))
    g.close()


@pytest.mark.parametrize("width,deg", [(20, 3), (1000, 8), (7000, 1)])
def test_resident_cc_local_ids(ctx, knobs, width, deg):
    """Chains of trees that many edges merge at once: neighbours within `width`
    ids, components cut every 9973 vertices."""
    n = 60000
    rng = np.random.default_rng(width)
    src = np.repeat(np.arange(n), deg)
    dst = np.minimum(src + rng.integers(1, width, len(src)), (src // 9973 + 1) * 9973 - 1).clip(max=n - 1)
    g = ctx.from_edges(n, src.astype(np.uint32), dst.astype(np.uint32))
    off, adj = g.download()
    want = O.cc(O.Graph(n, off, adj))
    for res in (1, 0):
        gg.tuning_set("resident", res)
        for _ in range(5):
            assert np.array_equal(g.cc(), want), res
    g.close()
