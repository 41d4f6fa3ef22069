"""What runs between hops, at its sizes' edges: cleared rows of every narrow width
over reused buffers, and the SPARSE degree scan around a tile of 1,024 pairs and
beyond 1,024 tiles."""
import numpy as np
import pytest

from oracle import pyoracle as O
from vertexsurge_gb300 import graphgen

pytestmark = pytest.mark.gpu


def random_graph(V, E, seed):
    rng = np.random.default_rng(seed)
    e = rng.integers(0, V, (2, E)).astype(np.uint32)
    return graphgen.from_edges(V, e[0], e[1])


@pytest.mark.parametrize("S", [1, 128, 129, 300, 400, 513, 700, 800, 900, 1024, 1025])
@pytest.mark.parametrize("path", ["shortest", "any"])
def test_narrow_rows_are_clean_for_the_next_run(vs, S, path):
    """Rows of 1 to 9 16-byte cells (a range up to 8, rows above), V no multiple of a range of 128 rows."""
    g = random_graph(1337, 4000, 5)
    dg = vs.DeviceGraph.from_host(g)
    for strategy in ("sparse", "push", "auto"):
        plan = vs.ExpandPlan(dg, S, vs.make_params(1, 3, path, "forward", strategy=strategy))
        for seed in (1, 2, 3):
            src = np.random.default_rng(seed).integers(0, g.V, S).astype(np.uint32)
            plan.run(src)
            assert np.array_equal(plan.result().download(), O.vexpand(g, src, 1, 3, path, "forward")[0]), (strategy, seed)


@pytest.mark.parametrize("S", [1, 1023, 1024, 1025, 2049])
def test_sparse_scan_around_a_tile(vs, S):
    g = random_graph(3000, 9000, 6)
    dg = vs.DeviceGraph.from_host(g)
    src = np.resize(graphgen.sample_sources(g.V, min(S, g.V), seed=S), S).astype(np.uint32)
    m, _, _ = vs.expand(dg, src, 1, 2, "shortest", "both", strategy="sparse")
    assert np.array_equal(m.download(), O.vexpand(g, src, 1, 2, "shortest", "both")[0])


def test_sparse_scan_beyond_1024_tiles(vs):
    g = random_graph(40_000, 1_600_000, 7)
    dg = vs.DeviceGraph.from_host(g)
    src = graphgen.sample_sources(g.V, 1024, seed=8)
    a, _, st = vs.expand(dg, src, 1, 3, "shortest", "forward", strategy="sparse", stats=True,
                         pair_capacity=4_000_000)
    b, _, _ = vs.expand(dg, src, 1, 3, "shortest", "forward", strategy="pull")
    assert list(st["strategy"][1:4]) == [3, 3, 3] and st["new_bits"][2] > 1024 * 1024, st
    assert np.array_equal(a.download(), b.download())
