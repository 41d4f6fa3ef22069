"""Rows of a two-adjacency intersection over bases around the sizes at which a warp takes one, two, four and
eight tuples."""
import numpy as np
import pytest

from vertexsurge_gb300 import graphgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [9727, 9728, 9729, 19457, 38911, 38912, 38915, 60_001])
def test_rows(vs, n):
    rng = np.random.default_rng(n)
    sizes = [0, 1, 5, 31, 33, 64, 65, 130, 200]
    src = np.repeat(np.arange(90, dtype=np.uint32), np.tile(sizes, 10))
    g = graphgen.from_edges(700, src, np.concatenate([rng.choice(600, k, replace=False) + 100 for k in np.tile(sizes, 10)]))
    dg = vs.DeviceGraph.from_host(g)
    both = {}
    for x in range(90):
        for y in range(90):
            li = [g.fwd_dst[g.fwd_off[v]:g.fwd_off[v + 1]] for v in (x, y)]
            both[x, y] = np.intersect1d(*li)
    a, b = rng.integers(0, 90, n).astype(np.uint32), rng.integers(0, 90, n).astype(np.uint32)
    per = [both[p] for p in zip(a.tolist(), b.tolist())]
    cnt = np.array([len(z) for z in per])
    want = np.stack([np.repeat(a, cnt), np.repeat(b, cnt), np.concatenate(per)], 1).astype(np.uint32)
    base = vs.FlatTable.from_columns([a, b])
    deps = [dict(graph=dg, direction="forward", base_col=c) for c in (0, 1)]
    t, count, _ = vs.mintersect(base, deps, 700, False)
    assert count == len(want) and np.array_equal(np.stack(t.columns(), 1), want)
    t, count, cut = vs.mintersect(base, deps, 700, False, max_rows=len(want) // 3)
    assert count == len(want) and cut and np.array_equal(np.stack(t.columns(), 1), want[:len(want) // 3])
