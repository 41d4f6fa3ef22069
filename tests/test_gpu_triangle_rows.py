"""Rows of a two-adjacency intersection written from the candidates' bits: lists around
a word, a step of 64 and a warp's 1,024 candidates, tuples without a list or a match,
a base no multiple of a task, and lists too long for the bits' scratch."""
import numpy as np
import pytest

from vertexsurge_gb300 import graphgen

pytestmark = pytest.mark.gpu

SIZES = [0, 1, 31, 32, 33, 63, 64, 65, 127, 128, 129, 500, 1023, 1024, 1025, 2000]


@pytest.fixture(scope="module")
def lists(vs):
    """Vertex i has SIZES[i] out-neighbours above 100; vertex 20 + i every third of them and others."""
    rng = np.random.default_rng(4)
    src, dst = [], []
    for i, n in enumerate(SIZES):
        nb = rng.choice(4000, n, replace=False) + 100
        other = np.unique(np.concatenate([nb[::3], rng.choice(4000, n // 2, replace=False) + 100]))
        src += [i] * n + [20 + i] * len(other)
        dst += list(nb) + list(other)
    g = graphgen.from_edges(4200, np.array(src, np.uint32), np.array(dst, np.uint32))
    return g, vs.DeviceGraph.from_host(g)


def expected(g, a, b):
    out = []
    for x, y in zip(a, b):
        nx, ny = (g.fwd_dst[g.fwd_off[v]:g.fwd_off[v + 1]] for v in (int(x), int(y)))
        out += [(x, y, z) for z in np.intersect1d(nx, ny)]
    return np.array(out, np.uint32).reshape(-1, 3)


def listing(vs, dg, a, b, **kw):
    base = vs.FlatTable.from_columns([a, b])
    deps = [dict(graph=dg, direction="forward", base_col=c) for c in (0, 1)]
    t, n, cut = vs.mintersect(base, deps, 4200, **kw)
    return np.stack(t.columns(), 1).astype(np.uint32).reshape(-1, 3), n, cut


@pytest.mark.parametrize("n", [1, 7, 8, 9, 200])
@pytest.mark.parametrize("long_only", [False, True])
def test_rows_and_bound(vs, lists, n, long_only):
    g, dg = lists
    rng = np.random.default_rng(n)
    pick = [len(SIZES) - 1] if long_only else range(len(SIZES))  # long_only: more bits than 512 a tuple
    i = np.array(rng.choice(pick, n), np.uint32)
    a, b = (i, i + 20) if n % 2 else (i + 20, i)
    exp = expected(g, a, b)
    rows, count, cut = listing(vs, dg, a, b)
    assert count == len(exp) and not cut and np.array_equal(rows, exp)
    if len(exp) > 2:
        bound = len(exp) // 2
        rows, count, cut = listing(vs, dg, a, b, max_rows=bound)
        assert count == len(exp) and cut and np.array_equal(rows, exp[:bound])
