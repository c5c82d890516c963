"""Timed cases: what programs built on this library have it do.

A case names an analytic (or a loop of a program's own over the operators), a
family of graphs with its size, and the options the call takes.  Graphs come
as edge lists made from the seed and go through the library's own ingest, as
a program's data do.  Traversals deliver levels, labels and core numbers in
device properties; the batched calls, whose results exist in host memory
only, deliver host arrays.
"""
import math

import numpy as np
import torch

from graptor_b200 import gg
from graptor_b200.selector_train import load_selector

DEV = "cuda"
DAMPING = 0.85
FORMATS = {"f32": gg.F32, "bf16": gg.BF16, "f16": gg.F16, "f64": gg.F64}

_context = None


def context():
    """One library context per process, as a program keeps it."""
    global _context
    if _context is None:
        _context = gg.Context(0)
    return _context


# --------------------------------------------------------------------------
# The cases
# --------------------------------------------------------------------------
def listed():
    return [
        # the smallest call: levels of one root on a graph that fits any cache (latency of a call)
        dict(name="bfs_rmat12", op="bfs", graph="rmat", scale=12, ef=16, relabel=False, learned=False),
        # the benchmark's step: one root of an R-MAT 24 graph, variants chosen by the shipped network
        dict(name="bfs_rmat24_learned", op="bfs", graph="rmat", scale=24, ef=16, relabel=False, learned=True),
        # ids as real data have them, in no order of degree; density threshold alone
        dict(name="bfs_rmat22_relabelled", op="bfs", graph="rmat", scale=22, ef=16, relabel=True, learned=False),
        # road-like graph, thousands of small levels
        dict(name="bfs_grid2896", op="bfs", graph="grid", rows=2896, cols=2893, deleted=0.01, learned=False),
        # connected components of a power-law graph
        dict(name="cc_rmat24", op="cc", graph="rmat", scale=24, ef=16, relabel=False),
        # many small graphs (power-law and grids) served as one batch: levels and labels to the host
        dict(name="batch_100_graphs", op="batch", parts=100, low=10.0, high=18.0),
        # core decomposition: a thousand dependent peel steps
        dict(name="kcore_rmat20", op="kcore", graph="rmat", scale=20, ef=16, relabel=False),
        # PageRank as the reference computes it: FP32 values, double sums, 20 iterations
        dict(name="pagerank_f32_rmat24", op="pagerank", graph="rmat", scale=24, ef=16, relabel=False, fmt="f32",
             iters=20),
        # the reduced-precision format that is used in earnest, on a directed graph with sinks
        dict(name="pagerank_bf16_er24", op="pagerank", graph="er", n=16777259, deg=32.0, sinks=0.01, directed=True,
             fmt="bf16", iters=20),
        # 64 searches and 128 personalised rankings at once, results to the host
        dict(name="msbfs64_rmat18", op="msbfs", graph="rmat", scale=18, ef=16, relabel=False, k=64),
        dict(name="ppr128_rmat18", op="ppr", graph="rmat", scale=18, ef=16, relabel=False, k=128, iters=20),
        # a program's own loop over edgemap and vertexmap: frontier steps on a directed graph of odd size
        dict(name="operators_bfs_er", op="operators_bfs", graph="er", n=3000017, deg=16.0, sinks=0.01,
             directed=True),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    op = rng.choice(["bfs", "bfs", "bfs", "cc", "cc", "pagerank", "pagerank", "pagerank", "kcore", "msbfs", "ppr",
                     "batch", "operators_bfs", "operators_pagerank"])
    if op == "batch":
        low = rng.uniform(8.0, 11.0)
        return dict(op=op, parts=_log_int(rng, 3, 100), low=low, high=low + rng.uniform(1.0, 7.0))
    batched = op in ("msbfs", "ppr")
    family = rng.choice(["rmat", "rmat", "er"] if batched or op == "kcore" else ["rmat", "rmat", "er", "grid"])
    case = dict(op=op, graph=family)
    if family == "rmat":
        case.update(scale=rng.randint(8, 18 if batched else 23 if op != "kcore" else 20), ef=rng.randint(4, 24),
                    relabel=rng.random() < 0.5)
    elif family == "er":
        n = _log_int(rng, 301, 262145 if batched else 4194305)
        directed = op != "kcore" and rng.random() < 0.5
        # components are of interest where a graph is sparse enough to have several
        deg = rng.uniform(0.5, 2.0) if op == "cc" else rng.uniform(2.0, 32.0)
        case.update(n=n, deg=round(deg, 2), sinks=0.01 if directed else 0.0, directed=directed)
    else:
        deleted = rng.uniform(0.3, 0.45) if op == "cc" else rng.uniform(0, 0.1)
        case.update(rows=_log_int(rng, 17, 2048), cols=_log_int(rng, 17, 2048), deleted=round(deleted, 3))
    if op == "bfs":
        case["learned"] = rng.random() < 0.5
    if op == "pagerank":
        case.update(fmt=rng.choice(["f32", "f32", "bf16", "f16", "f64"]), iters=rng.randint(5, 20))
    if op == "msbfs":
        case["k"] = rng.randint(1, 64)
    if op == "ppr":
        case.update(k=rng.randint(1, 128), iters=rng.randint(5, 20))
    if op == "operators_pagerank":
        case["iters"] = rng.randint(2, 10)
    return case


# --------------------------------------------------------------------------
# Graphs from the seed: edge lists on the device
# --------------------------------------------------------------------------
def _rmat_edges(scale, ef, relabel, gen):
    """Endpoints of ef * 2^scale R-MAT edges, quadrants 0.57 / 0.19 / 0.19 / 0.05; `relabel` shuffles the ids."""
    count = ef << scale
    src = torch.zeros(count, dtype=torch.int32, device=DEV)
    dst = torch.zeros(count, dtype=torch.int32, device=DEV)
    for _ in range(scale):
        u = torch.rand(count, device=DEV, generator=gen)
        src.mul_(2).add_(u >= 0.76)
        dst.mul_(2).add_(((u >= 0.57) & (u < 0.76)) | (u >= 0.95))
    if relabel:
        perm = torch.randperm(1 << scale, device=DEV, generator=gen, dtype=torch.int32)
        src, dst = perm[src], perm[dst]
    return src, dst


def _er_edges(n, deg, sinks, gen):
    """n * deg uniform endpoint pairs; a share `sinks` of the vertices has no out-edges."""
    count = max(1, int(n * deg))
    src = torch.randint(n, (count,), device=DEV, generator=gen, dtype=torch.int32)
    dst = torch.randint(n, (count,), device=DEV, generator=gen, dtype=torch.int32)
    if sinks:
        keep = (torch.rand(n, device=DEV, generator=gen) >= sinks)[src]
        src, dst = src[keep], dst[keep]
    return src, dst


def _grid_edges(rows, cols, deleted, gen):
    """Right and down neighbours of a rows x cols grid, a share `deleted` of them left out."""
    ids = torch.arange(rows * cols, device=DEV, dtype=torch.int32).view(rows, cols)
    src = torch.cat([ids[:, :-1].reshape(-1), ids[:-1, :].reshape(-1)])
    dst = torch.cat([ids[:, 1:].reshape(-1), ids[1:, :].reshape(-1)])
    keep = torch.rand(src.numel(), device=DEV, generator=gen) >= deleted
    return src[keep].contiguous(), dst[keep].contiguous()


def _edges(case, gen):
    """(n, src, dst, symmetric) of the case's graph."""
    if case["graph"] == "rmat":
        return (1 << case["scale"],) + _rmat_edges(case["scale"], case["ef"], case["relabel"], gen) + (True,)
    if case["graph"] == "er":
        return (case["n"],) + _er_edges(case["n"], case["deg"], case["sinks"], gen) + (not case["directed"],)
    return (case["rows"] * case["cols"],) + _grid_edges(case["rows"], case["cols"], case["deleted"], gen) + (True,)


def _ingest(n, src, dst, symmetric):
    torch.cuda.synchronize()
    return context().from_edges(n, (src.data_ptr(), src.numel()), (dst.data_ptr(), dst.numel()), symmetrise=symmetric,
                                device=True)


def _pick(n, src, dst, count, gen):
    """`count` vertices with out-edges (endpoints of seeded edges that are no self-loops)."""
    at = torch.randint(src.numel(), (64 * count,), device=DEV, generator=gen)
    a, b = src[at], dst[at]
    a = a[a != b]
    a = a if a.numel() else torch.zeros(1, dtype=torch.int32, device=DEV)
    return a.repeat(-(-count // a.numel()))[:count].cpu().numpy().astype(np.uint32)


class _DeviceArray:
    """A property's storage for torch, which keeps this object and with it the property and its graph
    (uint32 ids are seen as int32)."""

    def __init__(self, prop):
        self.prop = prop
        typestr = {gg.F32: "<f4", gg.F64: "<f8"}.get(prop.dtype, "<i4")
        self.__cuda_array_interface__ = dict(shape=(prop.g.n,), typestr=typestr, data=(prop.device_ptr(), False),
                                             version=3)


def _view(prop):
    return torch.as_tensor(_DeviceArray(prop), device=DEV)


# --------------------------------------------------------------------------
# What a program has in hand before the call
# --------------------------------------------------------------------------
def _batch_parts(case, gen):
    """Edge lists of the batch's small graphs, power-law and grids in turn, sizes spread over their logarithm (the
    sizes belong to the case, a few of the grids' edges are left out at random)."""
    rng = np.random.default_rng(case["parts"])
    for i in range(case["parts"]):
        lg = rng.uniform(case["low"], case["high"])
        if i % 2 == 0:
            scale = int(round(lg))
            ef = int(rng.integers(8, 33))
            yield (1 << scale,) + _rmat_edges(scale, ef, False, gen)
        else:
            side = int(2 ** (lg / 2))
            rows, cols = side, max(2, int(2 ** lg) // side)
            yield (rows * cols,) + _grid_edges(rows, cols, 0.01, gen)


def prepare(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    op = case["op"]
    state = dict(op=op, case=case)
    if op == "batch":
        parts = [_ingest(n, src, dst, True) for n, src, dst in _batch_parts(case, gen)]
        state["graph"], base = gg.graph_union(context(), parts)
        state["roots"] = base[:-1].copy()
        for p in parts:
            p.close()
        torch.cuda.empty_cache()
        return state
    n, src, dst, symmetric = _edges(case, gen)
    state["graph"] = g = _ingest(n, src, dst, symmetric)
    roots = _pick(n, src, dst, max(1, case.get("k", 1)), gen)
    del src, dst
    torch.cuda.empty_cache()
    if op in ("bfs", "operators_bfs"):
        state["root"] = int(roots[0])
        state["out"] = g.prop(gg.I32)
    if op == "bfs":
        state["opts"] = None
        if case["learned"]:
            gg.attach_selector(g, load_selector(context()))
            state["opts"] = gg.default_opts(gg.THRESH_LEARNED)
    elif op in ("cc", "kcore"):
        state["out"] = g.prop(gg.U32)
    elif op == "pagerank":
        state["out"] = g.prop(gg.F64 if case["fmt"] == "f64" else gg.F32)
    elif op in ("msbfs", "ppr"):
        state["roots"] = roots
    elif op == "operators_bfs":
        state["prev"] = g.prop(gg.I32)
        state["frontiers"] = [g.frontier(), g.frontier()]
    elif op == "operators_pagerank":
        for p in ("out", "y", "contrib"):
            state[p] = g.prop(gg.F32)
    if "out" in state:
        state["view"] = _view(state["out"])
    return state


# --------------------------------------------------------------------------
# One pass
# --------------------------------------------------------------------------
def _program(g, props, consts, code, nreduce=0):
    """vertexmap of [(opcode, argument), ...]."""
    d = gg.VmapDesc(ncode=len(code), nreduce=nreduce)
    for i, (op, arg) in enumerate(code):
        d.code[i], d.arg[i] = op, arg
    for i, p in enumerate(props):
        d.props[i] = p.h
    for i, c in enumerate(consts):
        d.consts[i] = c
    return g.vertexmap(d)


def _operators_bfs(state):
    """Level-synchronous search over edgemap, one call a level, the library choosing push or pull."""
    g, level, prev, root = state["graph"], state["out"], state["prev"], state["root"]
    fin, fout = state["frontiers"]
    level.fill(g.n + 1)
    prev.fill(g.n + 1)
    level.set(root, 0)
    prev.set(root, 0)
    fin.set_single(root)
    step = 0
    while fin.counts()[0]:
        g.edgemap(gg.EmapDesc(relax=gg.RELAX_MIN_PLUS1_I32, a=level.h, dst_filter=gg.FILTER_GT_CONST,
                              dst_filter_k=step + 1, record=gg.RECORD_NE_PREV, prev=prev.h, variant=gg.VAR_AUTO,
                              threshold=gg.THRESH_DEFAULT), fin, fout)
        fin, fout = fout, fin
        step += 1


def _operators_pagerank(state):
    """The reference's PageRank loop written over edgemap and vertexmap."""
    g, x, y, contrib, n = state["graph"], state["out"], state["y"], state["contrib"], state["graph"].n
    scatter = [(gg.VM_LOAD, 0), (gg.VM_CONST, 0), (gg.VM_MUL, 0), (gg.VM_DEGREE, 0), (gg.VM_DIV, 0), (gg.VM_STORE, 2)]
    _program(g, [x, y, contrib], [DAMPING, 1.0 / n, 0.0],
             [(gg.VM_CONST, 1), (gg.VM_STORE, 0), (gg.VM_CONST, 2), (gg.VM_STORE, 1)] + scatter)
    for _ in range(state["case"]["iters"]):
        g.edgemap(gg.EmapDesc(relax=gg.RELAX_ADD_GATHER, a=y.h, src=contrib.h, accum_f64=1, record=gg.RECORD_NONE,
                              variant=gg.VAR_AUTO))
        s = _program(g, [y], [], [(gg.VM_LOAD, 0), (gg.VM_REDUCE_ADD, 0)], 1)[0]
        s = _program(g, [y], [(1.0 - s) / n],
                     [(gg.VM_LOAD, 0), (gg.VM_CONST, 0), (gg.VM_ADD, 0), (gg.VM_STORE, 0), (gg.VM_LOAD, 0),
                      (gg.VM_REDUCE_ADD, 0)], 1)[0]
        delta = _program(g, [x, y, contrib], [DAMPING, 1.0 / s, 0.0],
                         [(gg.VM_LOAD, 1), (gg.VM_CONST, 1), (gg.VM_MUL, 0), (gg.VM_DUP, 0), (gg.VM_LOAD, 0),
                          (gg.VM_SUB, 0), (gg.VM_ABS, 0), (gg.VM_REDUCE_ADD, 0), (gg.VM_STORE, 0), (gg.VM_CONST, 2),
                          (gg.VM_STORE, 1)] + scatter, 1)[0]
        if not delta > 0:
            break


def run(state):
    op, g, case = state["op"], state["graph"], state["case"]
    if op == "bfs":
        g.bfs_level(state["root"], level=state["out"], host=False, opts=state["opts"])
    elif op == "cc":
        g.cc(label=state["out"], host=False)
    elif op == "kcore":
        _, largest = g.kcore(coreness=state["out"], host=False)
        return [state["view"], largest]
    elif op == "pagerank":
        # a negative tolerance runs every iteration; sums in double for FP32 and FP64, in float for the
        # reduced formats, as the benchmark runs them
        g.pagerank(maxiter=case["iters"], tol=-1.0, contrib=FORMATS[case["fmt"]],
                   accum_f64=case["fmt"] in ("f32", "f64"), renorm_f32=case["fmt"] == "f32", x=state["out"],
                   host=False)
    elif op == "batch":
        levels, labels, _, _ = gg.batch_bfs_cc(g, state["roots"])
        return [levels, labels.view(np.int32)]
    elif op == "msbfs":
        return gg.msbfs(g, state["roots"])
    elif op == "ppr":
        return gg.ppr(g, state["roots"], alpha=0.15, iters=case["iters"])
    elif op == "operators_bfs":
        _operators_bfs(state)
    else:
        _operators_pagerank(state)
    return state["view"]


# --------------------------------------------------------------------------
# What a pass cannot do without
# --------------------------------------------------------------------------
def _size(case):
    """(vertices, directed edges) of the case's graph, duplicates and self-loops not taken off."""
    if case["op"] == "batch":
        spread = case["high"] - case["low"]
        mean = (2 ** case["high"] - 2 ** case["low"]) / (spread * math.log(2))
        return case["parts"] * mean, case["parts"] * mean * (20 * 2 + 4) / 2
    if case["graph"] == "rmat":
        return 1 << case["scale"], 2 * (case["ef"] << case["scale"])
    if case["graph"] == "er":
        return case["n"], case["n"] * case["deg"] * (1 if case["directed"] else 2)
    return case["rows"] * case["cols"], 4 * case["rows"] * case["cols"]


def work(case):
    n, m = _size(case)
    op = case["op"]
    if op in ("bfs", "operators_bfs", "cc"):
        # every vertex's row bound, one edge that reaches it, its result
        return {"bytes": 8 * n + 4 * n + 4 * n, "flops": 0}
    if op == "batch":
        return {"bytes": 2 * (8 * n + 4 * n + 4 * n), "flops": 0}
    if op == "kcore":
        # every edge is counted down once
        return {"bytes": 8 * n + 4 * m + 4 * n, "flops": m}
    if op == "msbfs":
        return {"bytes": 8 * n + 4 * m + 4 * n * case["k"], "flops": 0}
    if op == "ppr":
        # the edges and, per iteration, contributions of two bytes a seed read and written
        return {"bytes": case["iters"] * (8 * n + 4 * m + 4 * n * case["k"]) + 4 * n * case["k"],
                "flops": 2 * case["iters"] * m * case["k"]}
    # an iteration reads the edges and the contributions, and reads and writes ranks
    size = {"f32": 4, "f64": 8}.get(case.get("fmt", "f32"), 2)
    rank = 8 if case.get("fmt") == "f64" else 4
    return {"bytes": case["iters"] * (8 * n + 4 * m + 2 * size * n + 2 * rank * n), "flops": 2 * case["iters"] * m}


# --------------------------------------------------------------------------
# The same in 64 bits
# --------------------------------------------------------------------------
def _unique(n, src, dst, symmetric):
    """Distinct edges without self-loops, as (src, dst) of 64-bit ids."""
    src, dst = src.long(), dst.long()
    if symmetric:
        src, dst = torch.cat([src, dst]), torch.cat([dst, src])
    keys = src * n + dst
    keys = torch.unique(keys[src != dst])
    return keys // n, keys % n


def exact(case, seed):
    op = case["op"]
    if op not in ("pagerank", "operators_pagerank", "ppr"):
        return None  # whole numbers
    gen = torch.Generator(device=DEV).manual_seed(seed)
    n, src, dst, symmetric = _edges(case, gen)
    roots = _pick(n, src, dst, max(1, case.get("k", 1)), gen)
    src, dst = _unique(n, src, dst, symmetric)
    deg = torch.bincount(src, minlength=n).double()
    if op == "ppr":
        k = case["k"]
        rows = torch.sparse_coo_tensor(torch.stack([dst, src]), 1.0 / deg[src], (n, n)).coalesce().to_sparse_csr()
        seeds = torch.zeros(n, k, dtype=torch.float64, device=DEV)
        seeds[torch.from_numpy(roots.astype(np.int64)).to(DEV), torch.arange(k, device=DEV)] = 1.0
        x = seeds
        for _ in range(case["iters"]):
            x = 0.15 * seeds + 0.85 * (rows @ x)
        return x
    x = torch.full((n,), 1.0 / n, dtype=torch.float64, device=DEV)
    for _ in range(case["iters"]):
        contrib = DAMPING * x / deg.clamp(min=1.0)
        y = torch.zeros_like(x).index_add_(0, dst, contrib[src])
        y += (1.0 - y.sum()) / n
        x = y / y.sum()
    return x
