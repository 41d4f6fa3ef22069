"""The dense PULL of rows of 32 lanes takes the non-empty rows of 32 list entries in rounds of 8, 4 or 2:
lists with every number of them, over one and two batches of entries, with and without room to gain."""
import numpy as np
import pytest

from oracle import pyoracle as O
from vertexsurge_gb300 import graphgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S", [2176, 4096, 4100, 9000, 16400])  # 17, 32, 34, 72 and 130 cells a row
@pytest.mark.parametrize("path,k0", [("shortest", 1), ("any", 2)])
def test_every_number_of_rows(vs, S, path, k0):
    """Target t's list has t % 67 entries with a row after the first hop and up to 40 without one, in random order."""
    rng = np.random.default_rng(S)
    A, D, T = 3000, 4000, 5000  # first active middle, first vertex without a row, first target
    V = T + 200
    src, dst = list(rng.integers(0, 2900, 6 * (D - A))), list(np.repeat(np.arange(A, D), 6))
    for t in range(200):
        li = np.concatenate([rng.choice(np.arange(A, D), t % 67, replace=False),
                             rng.choice(np.arange(D, T), (t * 7) % 41, replace=False)])
        src += list(li)
        dst += [T + t] * len(li)
    g = graphgen.from_edges(V, np.array(src, np.uint32), np.array(dst, np.uint32))
    dg = vs.DeviceGraph.from_host(g)
    sources = np.resize(np.arange(2900), S).astype(np.uint32)
    m, _, _ = vs.expand(dg, sources, k0, 2, path, "forward", strategy="pull", short_share=-1.0)
    assert np.array_equal(m.download(), O.vexpand(g, sources, k0, 2, path, "forward")[0])
    m.free()
