"""Triangle rows whose output fits only without the scratch that keeps the candidates' bits."""
import numpy as np
import pytest

from tests.small_pool import small_pool
from vertexsurge_gb300 import graphgen

pytestmark = pytest.mark.gpu


def test_output_takes_the_room_of_the_bits(vs):
    """2M tuples of four common members each: 128 MB of bits, 96 MB of rows, 48 MB of counts and places."""
    n, members = 2_000_000, np.array([70, 81, 95, 99], np.uint32)
    g = graphgen.from_edges(100, np.repeat(np.arange(64, dtype=np.uint32), 4), np.tile(members, 64))
    dg = vs.DeviceGraph.from_host(g)
    rng = np.random.default_rng(1)
    a, b = rng.integers(0, 64, n).astype(np.uint32), rng.integers(0, 64, n).astype(np.uint32)
    base = vs.FlatTable.from_columns([a, b])
    deps = [dict(graph=dg, direction="forward", base_col=c) for c in (0, 1)]
    vs.mintersect(base, deps, 100, True)  # the graph's bitmaps, if any
    with small_pool(224 << 20):
        t, count, cut = vs.mintersect(base, deps, 100, False)
        cols = t.columns()
        t.free()
    assert count == 4 * n and not cut
    for got, want in zip(cols, (np.repeat(a, 4), np.repeat(b, 4), np.tile(members, n))):
        assert np.array_equal(got, want)
