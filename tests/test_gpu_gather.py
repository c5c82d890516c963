"""The contribution gather at the sizes where its paths meet: rows around the
heavy-row threshold (256), its chunks (1024) and the shared-memory stage (512
or 1024 values), words with several heavy rows, empty rows and words, and a
vertex count that is no multiple of 32."""
import numpy as np
import pytest

from graptor_b200 import gg

pytestmark = pytest.mark.gpu

EDGES = [0, 1, 2, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 512, 513, 1023, 1024, 1025,
         2048, 3001]


def in_degrees(kind, n, rng):
    deg = np.zeros(n, dtype=np.int64)
    if kind == "edges":      # every boundary length, in words of their own and mixed with empty rows
        deg[rng.permutation(n)[: 8 * len(EDGES)]] = np.tile(EDGES, 8)
    elif kind == "full":     # words whose light rows fill many stages: 32 rows of 250..256
        deg[:160] = rng.integers(250, 257, 160)
    elif kind == "heavy":    # words of heavy rows with a light row between two of them
        deg[32:96] = rng.integers(257, 2500, 64)
        deg[40], deg[41], deg[95] = 3, 256, 200
    else:                    # short rows only
        deg[:] = rng.integers(0, 6, n)
    return deg


@pytest.mark.parametrize("kind", ["edges", "full", "heavy", "short"])
@pytest.mark.parametrize("dtype,acc64", [(gg.F32, 1), (gg.F32, 0), (gg.BF16, 0), (gg.F64, 1)])
def test_gather_rows(ctx, kind, dtype, acc64):
    rng = np.random.default_rng(len(kind))
    n = 4133
    deg = in_degrees(kind, n, rng)
    dst = np.repeat(np.arange(n), deg).astype(np.uint32)
    # a row's sources: distinct vertices other than the row's own
    src = np.concatenate([(d + 1 + rng.permutation(n - 1)[:k]) % n for d, k in enumerate(deg) if k]).astype(np.uint32)
    g = ctx.from_edges(n, src, dst, symmetrise=False)
    assert g.m == len(src)
    c = rng.uniform(0.5, 1.5, n).astype(np.float32)
    if dtype == gg.BF16:
        raw = (c.view(np.uint32) >> 16).astype(np.uint16)
        c = (raw.astype(np.uint32) << 16).view(np.float32)
    else:
        raw = c.astype(np.float64) if dtype == gg.F64 else c
    want = np.bincount(dst, weights=c[src].astype(np.float64), minlength=n)
    contrib, y = g.prop(dtype), g.prop(gg.F64 if dtype == gg.F64 else gg.F32)
    contrib.upload(raw)
    y.fill(0)
    g.edgemap(gg.EmapDesc(relax=gg.RELAX_ADD_GATHER, a=y.h, src=contrib.h, accum_f64=acc64, record=gg.RECORD_NONE,
                          variant=gg.VAR_AUTO))
    got = y.download().astype(np.float64)
    # double sums: one rounding to the stored type; float sums: half an ulp of the sum per addition
    eps = 2.0 ** -52 if dtype == gg.F64 else 2.0 ** -24
    tol = want * eps * (np.maximum(deg, 1) if dtype == gg.F64 or not acc64 else 1.001)
    assert np.all(np.abs(got - want) <= tol)
    g.close()


@pytest.mark.parametrize("n", [5920 * 32 - 1, 5920 * 32 + 1, 400003, 2200001])
@pytest.mark.parametrize("deg", [0, 1, 3])
def test_gather_ranges_of_several_words(ctx, n, deg):
    """Sparse rows, whose ranges are of several words: up to and beyond a word
    per warp, none and few edges, and a stretch of longer rows."""
    rng = np.random.default_rng(n + deg)
    degs = np.full(n, deg, dtype=np.int64)
    degs[n // 3: n // 3 + 2000] = 40
    dst = np.repeat(np.arange(n), degs)
    src = (dst + 1 + np.arange(len(dst)) % 977) % n
    g = ctx.from_edges(n, src.astype(np.uint32), dst.astype(np.uint32), symmetrise=False)
    assert g.m == len(dst)
    c = rng.uniform(0.5, 1.5, n)
    contrib, y = g.prop(gg.F64), g.prop(gg.F64)
    contrib.upload(c)
    y.fill(0)
    g.edgemap(gg.EmapDesc(relax=gg.RELAX_ADD_GATHER, a=y.h, src=contrib.h, accum_f64=1, record=gg.RECORD_NONE,
                          variant=gg.VAR_AUTO))
    want = np.bincount(dst, weights=c[src], minlength=n)
    assert np.all(np.abs(y.download() - want) <= want * 2.0 ** -52 * np.maximum(degs, 1))
    g.close()
