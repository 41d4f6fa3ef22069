"""The dense PULL with its row flags as bits in shared memory: vertex counts around the
smallest it takes, a word and a 16-byte cell, the row widths it takes, layers below and
above the share of active rows at which it is left, word slices, rows of one and two
cells on a long edge list, and the largest vertex count."""
import numpy as np
import pytest

from oracle import pyoracle as O
from vertexsurge_gb300 import graphgen

pytestmark = pytest.mark.gpu

V0 = 128 * 1024


def graph(V, E, seed):
    e = np.random.default_rng(seed).integers(0, V, (2, E)).astype(np.uint32)
    return graphgen.from_edges(V, e[0], e[1])


@pytest.mark.parametrize("V", [V0 - 1, V0, V0 + 1, V0 + 31, V0 + 33, V0 + 127])
@pytest.mark.parametrize("S", [300, 1000, 2000])
def test_vertex_counts_and_widths(vs, V, S):
    g = graph(V, 2 * V, V)
    dg = vs.DeviceGraph.from_host(g)
    src = np.append(np.random.default_rng(S).integers(0, V, S - 1), V - 1).astype(np.uint32)
    for path, direction, kw in (("shortest", "forward", {}), ("any", "both", {}), ("shortest", "both", {"slice_words": 6})):
        m, _, _ = vs.expand(dg, src, 1, 4, path, direction, strategy="pull", **kw)
        assert np.array_equal(m.download(), O.vexpand(g, src, 1, 4, path, direction)[0]), (path, direction)
        m.free()


@pytest.mark.parametrize("S", [3, 128, 129, 256])
def test_narrow_rows(vs, S):
    V = 200_001
    g = graph(V, 17_500_000, 5)
    dg = vs.DeviceGraph.from_host(g)
    src = np.random.default_rng(S).integers(0, V, S).astype(np.uint32)
    for strategy in ("pull", "auto"):
        m, _, _ = vs.expand(dg, src, 1, 3, "shortest", "forward", strategy=strategy)
        assert np.array_equal(m.download(), O.vexpand(g, src, 1, 3, "shortest", "forward")[0]), strategy
        m.free()


@pytest.mark.parametrize("V", [160 * 1024 * 8, 160 * 1024 * 8 + 1])
def test_largest_vertex_count(vs, V):
    g = graph(V, V // 2, 9)
    dg = vs.DeviceGraph.from_host(g)
    src = np.unique(g.rev_src)[-300:].astype(np.uint32)  # the last vertices with an out-list
    m, _, st = vs.expand(dg, src, 1, 3, "shortest", "forward", strategy="pull", stats=True)
    ref, _, ost = O.vexpand(g, src, 1, 3, "shortest", "forward", hop_stats=True)
    assert np.array_equal(m.download(), ref) and st["active_edges"][1:] == ost["active_edges"][1:]
