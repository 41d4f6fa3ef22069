"""Glue operators at the edges of their kernels' tiles, against numpy: the
transposed TableConvert (512 x 512 bit tiles), column counts and their ranking
(groups of 1 to 32 lanes, four columns each; with and without a column map), and
the row listing of a two-adjacency intersection (64 candidates a step, chunks of
8 tuples, lists with and without a bitmap)."""
import numpy as np
import pytest

from tests.conftest import bool_to_words, words_to_bool
from vertexsurge_gb300 import graphgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 31, 64, 65, 511, 512, 513, 1100])
@pytest.mark.parametrize("cols", [1, 32, 127, 129, 512, 513, 1537])
def test_transpose_tile_edges(vs, rows, cols):
    b = np.random.default_rng(rows * 10007 + cols).random((rows, cols)) < 0.4
    m = vs.BitMatrix.from_logical(bool_to_words(b), rows, cols)
    t = m.convert(True)
    assert t.shape == (cols, rows)
    assert np.array_equal(words_to_bool(t.download(), cols), b.T)
    assert t.count() == int(b.sum())  # padding words are zero
    assert np.array_equal(words_to_bool(m.convert(False).download(), rows), b)


@pytest.mark.parametrize("rows,cols", [(1, 5), (128, 9), (129, 1000), (500, 37), (2049, 300), (5000, 133)])
@pytest.mark.parametrize("mapped", [False, True])
def test_column_counts_and_ranking(vs, rows, cols, mapped):
    rng = np.random.default_rng(rows + cols)
    b = rng.random((rows, cols)) < rng.choice([0.0, 0.1, 0.5], cols)
    cmap = rng.permutation(10 * cols)[:cols].astype(np.uint32) if mapped else None
    m = vs.BitMatrix.from_logical(bool_to_words(b), rows, cols, col_map=cmap)
    val, cnt = (cmap if mapped else np.arange(cols)).astype(np.int64), b.sum(axis=0)
    for order in (None, "asc", "desc"):
        v, c = vs.matrix_column_count(m, order).columns()
        k = np.arange(cols) if order is None else np.lexsort((val, cnt))
        k = k[::-1] if order == "desc" else k
        assert np.array_equal(v, val[k]) and np.array_equal(c, cnt[k]), order
    assert m.count() == int(cnt.sum())


@pytest.mark.parametrize("direction", ["forward", "backward"])
def test_pair_rows(vs, direction):
    g = graphgen.rmat(11, 24, 0.57, 0.19, 0.19, seed=5)  # lists from 1 entry to several hundred
    dg = vs.DeviceGraph.from_host(g)
    u = np.repeat(np.arange(g.V, dtype=np.uint32), np.diff(g.fwd_off))
    off, adj = (g.fwd_off, g.fwd_dst) if direction == "forward" else (g.rev_off, g.rev_src)
    pick = np.random.default_rng(1).choice(g.E, 5003, replace=False)  # not a multiple of the chunk
    a, b = u[pick], g.fwd_dst[pick]
    base = vs.FlatTable.from_columns([a, b])
    deps = [dict(graph=dg, direction=direction, base_col=0), dict(graph=dg, direction=direction, base_col=1)]
    want = []
    for x, y in zip(a, b):
        for w in np.intersect1d(adj[off[x]:off[x + 1]], adj[off[y]:off[y + 1]]):
            want.append((x, y, w))
    t, n, cut = vs.mintersect(base, deps, g.V)
    assert n == len(want) and not cut
    assert sorted(zip(*(c.tolist() for c in t.columns()))) == sorted(want)
    for algo in ("binary", "bitmap", "merge"):
        t2, n2, _ = vs.mintersect(base, [dict(d, algo=algo) for d in deps], g.V)
        assert n2 == n and all(np.array_equal(p, q) for p, q in zip(t.columns(), t2.columns())), algo
    lim = n // 3
    t3, n3, cut = vs.mintersect(base, deps, g.V, max_rows=lim)
    assert cut and n3 == n and all(np.array_equal(p, q[:lim]) for p, q in zip(t3.columns(), t.columns()))
