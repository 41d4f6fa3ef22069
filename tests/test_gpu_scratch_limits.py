"""Calls whose optional scratch does not fit: they give the same rows without it."""
import numpy as np
import pytest

from tests.small_pool import small_pool
from vertexsurge_gb300 import graphgen

pytestmark = pytest.mark.gpu


def test_adjacency_bitmaps_without_room(vs):
    """3,000 lists of 1,100 entries on 1M vertices (375 MB of bitmaps): a call in a pool of 64 MB tests by binary
    search, and the next call builds them."""
    V, n, deg = 1_000_000, 3000, 1100
    dst = (np.arange(deg)[None, :] * 900 + np.arange(n)[:, None] % 90 * 10).astype(np.uint32)
    g = graphgen.from_edges(V, np.repeat(np.arange(n, dtype=np.uint32), deg), dst.ravel())
    dg = vs.DeviceGraph.from_host(g)
    a, b = np.arange(0, 200, dtype=np.uint32), np.arange(90, 290, dtype=np.uint32)
    base = vs.FlatTable.from_columns([a, b])  # pairs of equal lists, but for an edge of a vertex to itself
    nb = [g.fwd_dst[g.fwd_off[v]:g.fwd_off[v + 1]] for v in range(290)]
    want = sum(len(np.intersect1d(nb[x], nb[y])) for x, y in zip(a, b))
    deps = [dict(graph=dg, direction="forward", base_col=c) for c in (0, 1)]
    counts, launches = [], []
    for limit in (64 << 20, None, None):
        n0 = vs.kernel_launches()
        if limit:
            with small_pool(limit):
                counts.append(vs.mintersect(base, deps, V, True)[1])
        else:
            counts.append(vs.mintersect(base, deps, V, True)[1])
        launches.append(vs.kernel_launches() - n0)
    assert counts == [want] * 3
    # degree bins by both dependencies; bins, slots and bitmaps; the count alone
    assert [n - launches[2] for n in launches] == [2, 3, 0]
