"""The dense PULL's target groups, list pieces and early exit against the
oracle, bit for bit: every row width of a group (1 to 32 lanes, several words
per lane), in-lists of no entry, of a few, around the chunk and piece sizes and
of several pieces, saturated rows, sources that reach nothing."""
import numpy as np
import pytest

from oracle import pyoracle as O
from vertexsurge_gb300 import graphgen

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def listy(vs):
    """Vertex v < 40 has an in-list and an out-list of a length at or beside a
    chunk, threshold or piece size; a dense core saturates; 300 vertices are
    isolated."""
    V = 2400
    rng = np.random.default_rng(3)
    src, dst = [], []
    sizes = [1, 2, 7, 8, 9, 31, 32, 33, 63, 64, 65, 255, 256, 257, 511, 512, 513, 1023, 1024, 1025]
    for v, n in enumerate(sizes):
        peers = rng.choice(2000, n, replace=False) + 40
        src += list(peers) + [20 + v] * n
        dst += [v] * n + list(peers)
    core = rng.integers(40, 2100, (2, 12000))
    src += list(core[0])
    dst += list(core[1])
    g = graphgen.from_edges(V, np.array(src, np.uint32), np.array(dst, np.uint32))
    return g, vs.DeviceGraph.from_host(g)


@pytest.mark.parametrize("S", [1, 64, 129, 300, 513, 1025, 2049, 4097, 8193, 16385])
@pytest.mark.parametrize("path,k0,k1", [("shortest", 1, 5), ("shortest", 2, 4), ("any", 1, 3), ("any", 3, 3)])
def test_dense_pull_widths_and_pieces(vs, listy, S, path, k0, k1):
    g, dg = listy
    src = np.resize(graphgen.sample_sources(g.V, min(S, g.V), seed=S), S).astype(np.uint32)
    for direction in ("forward", "both"):
        exp, _, ost = O.vexpand(g, src, k0, k1, path, direction, hop_stats=True)
        for hub in (0, 5):
            m, _, st = vs.expand(dg, src, k0, k1, path, direction, strategy="pull", hub_threshold=hub, stats=True,
                                 short_share=-1.0)
            assert np.array_equal(m.download(), exp), (direction, hub)
            assert st["active_edges"][1:] == ost["active_edges"][1:]
            if path == "shortest":
                assert st["visit_count"] == ost["visit_count"][-1]
            m.free()


def test_dense_pull_reused_plan_and_row_limits(vs, listy):
    """Piece counters and unions are back at their start after every hop and run."""
    g, dg = listy
    S = 700
    plan = vs.ExpandPlan(dg, S, vs.make_params(1, 4, "shortest", "both", strategy="pull", hub_threshold=6))
    for seed in (1, 2, 3):
        src = graphgen.sample_sources(g.V, S, seed=seed)
        lim = np.random.default_rng(seed).integers(0, 5, S).astype(np.uint8)
        plan.set_row_limits(None if seed == 1 else lim)
        plan.run(src)
        got = plan.result().download()
        exp = O.vexpand(g, src, 1, 4, "shortest", "both")[0]
        if seed != 1:
            exp = np.zeros_like(exp)
            for k in range(1, 5):
                keep = np.packbits(np.resize(np.append(lim == k, np.zeros(4, bool)), 704), bitorder="little").view(np.uint64)
                exp |= O.vexpand(g, src, 1, k, "shortest", "both")[0] & keep
            # a row that never grows keeps nothing: its source bit is not part of hops 1..k
        assert np.array_equal(got, exp), seed
