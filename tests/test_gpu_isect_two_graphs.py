"""Adjacency dependencies on two graphs of different vertex counts: candidates of the
larger graph's lists lie past the end of the smaller graph's bitmaps (lists of 64
and of 1,024 entries and more), and are in none of its lists."""
import numpy as np
import pytest

from vertexsurge_gb300 import graphgen

pytestmark = pytest.mark.gpu


def star(V, deg, n, seed):
    """The first n vertices have deg out-neighbours each, spread up to the last vertex."""
    rng = np.random.default_rng(seed)
    dst = np.concatenate([np.sort(np.append(rng.choice(V - 1, deg - 1, replace=False), V - 1)) for _ in range(n)])
    return graphgen.from_edges(V, np.repeat(np.arange(n, dtype=np.uint32), deg), dst.astype(np.uint32))


@pytest.mark.parametrize("small_deg", [40, 64, 100, 1500])
@pytest.mark.parametrize("algo", ["auto", "binary", "bitmap"])
@pytest.mark.parametrize("ndeps", [2, 3])
def test_candidates_past_the_smaller_graph(vs, small_deg, algo, ndeps):
    n, Vs, Vl = 12, 1601, 9001
    big, small = star(Vl, 35 if small_deg < 1000 else 1200, n, 1), star(Vs, small_deg, n, 2)
    dgs = {id(g): vs.DeviceGraph.from_host(g) for g in (big, small)}
    rng = np.random.default_rng(small_deg)
    cols = [rng.integers(0, n, 50).astype(np.uint32) for _ in range(ndeps)]
    base = vs.FlatTable.from_columns(cols)
    for graphs in ([big, small, big], [small, big, small]):
        deps = [dict(graph=dgs[id(g)], direction="forward", base_col=c, algo=algo) for c, g in enumerate(graphs[:ndeps])]
        want = []
        for t in zip(*(c.tolist() for c in cols)):
            z = None
            for u, g in zip(t, graphs):
                li = g.fwd_dst[g.fwd_off[u]:g.fwd_off[u + 1]]
                z = li if z is None else np.intersect1d(z, li)
            want += [(*t, x) for x in z.tolist()]
        t, count, _ = vs.mintersect(base, deps, Vl, False)
        assert count == len(want) and sorted(zip(*(c.tolist() for c in t.columns()))) == sorted(want)
        assert vs.mintersect(base, deps, Vl, True)[1] == len(want)
