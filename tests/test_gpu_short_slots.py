"""Short-mode PULL over rows around one and two 32-byte pieces of a slot and its end
(15, 16, 31, 32 and 63 ids), for slots of 16, 32 and 64 entries."""
import numpy as np
import pytest

from oracle import pyoracle as O
from vertexsurge_gb300 import graphgen

pytestmark = pytest.mark.gpu

COUNTS = [1, 2, 3, 14, 15, 16, 17, 30, 31, 32, 33, 62, 63, 64, 65, 100]


@pytest.mark.parametrize("S", [4096, 4097, 8192, 8193, 20000])
@pytest.mark.parametrize("k", [3, 4])
def test_rows_of_every_slot_length(vs, S, k):
    """Source i points at a middle vertex chosen so that middle vertex j gathers COUNTS[j % 16] sources; a second
    middle layer copies those rows, and targets mix several of them."""
    rng = np.random.default_rng(S)
    V, M = 30_000, 400
    src, dst = [], []
    for j in range(M):  # sources 0..19999, middles 20000.., copies 21000.., targets 22000..
        n = COUNTS[j % len(COUNTS)]
        src += list(rng.choice(min(S, 20_000), n, replace=False))
        dst += [20_000 + j] * n
        src.append(20_000 + j)
        dst.append(21_000 + j)
    t = rng.integers(22_000, V, 60_000)
    src += list(21_000 + rng.integers(0, M, len(t)))
    dst += list(t)
    src += list(rng.integers(22_000, V, 20_000))
    dst += list(rng.integers(22_000, V, 20_000))
    g = graphgen.from_edges(V, np.array(src, np.uint32), np.array(dst, np.uint32))
    dg = vs.DeviceGraph.from_host(g)
    sources = np.resize(np.arange(min(S, 20_000)), S).astype(np.uint32)
    exp = O.vexpand(g, sources, 1, k, "shortest", "forward")[0]
    for share in (2.0, 0.0):  # always short, and by the rule
        m, _, st = vs.expand(dg, sources, 1, k, "shortest", "forward", strategy="pull", short_share=share, stats=True)
        assert np.array_equal(m.download(), exp), share
        assert share == 0.0 or any(st["short_pull"]), st["short_pull"]
        m.free()
