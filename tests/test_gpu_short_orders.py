"""Short-mode PULL where lanes write a target's bitmap in turn: long lists that come in
pieces, read from slots, and ids between whole rows in the in-neighbours put aside."""
import numpy as np
import pytest

from oracle import pyoracle as O
from vertexsurge_gb300 import graphgen

pytestmark = pytest.mark.gpu

MID, COPY, TGT = 5000, 7500, 10000  # first ids of the layers after the sources
V = 10200


def layered(rows, lists):
    """Middle vertex j gathers the sources rows[j], its copy the same a hop later; target t has the copies lists[t]."""
    src, dst = [], []
    for j, r in enumerate(rows):
        src += list(r) + [MID + j]
        dst += [MID + j] * len(r) + [COPY + j]
    for t, li in enumerate(lists):
        src += [COPY + int(j) for j in li]
        dst += [TGT + t] * len(li)
    return graphgen.from_edges(V, np.array(src, np.uint32), np.array(dst, np.uint32))


def check(vs, g, S, k_min, short, **kw):
    """Three hops from S sources, all pulled, the third in short mode `short`, against the oracle."""
    sources = np.arange(S, dtype=np.uint32)
    dg = vs.DeviceGraph.from_host(g)
    m, _, st = vs.expand(dg, sources, k_min, 3, "shortest", "forward", strategy="pull", short_share=2.0, stats=True, **kw)
    assert st["short_pull"][3] == short or (short is None and st["short_pull"][3]), st["short_pull"]
    assert np.array_equal(m.download(), O.vexpand(g, sources, k_min, 3, "shortest", "forward")[0])
    m.free()


@pytest.mark.parametrize("S", [2048, 4096])
@pytest.mark.parametrize("deg", [257, 511, 512, 513, 1000, 1999])
def test_pieces_of_rows_read_from_slots(vs, S, deg):
    """Targets of several pieces whose in-neighbours all have 1 to 15 ids: nothing is queued or put aside."""
    rng = np.random.default_rng(deg)
    rows = [rng.choice(S, 1 + j % 15, replace=False) for j in range(2100)]
    check(vs, layered(rows, [rng.choice(len(rows), deg + t, replace=False) for t in range(12)]), S, 1, 2)


@pytest.mark.parametrize("S", [2048, 4096, 8192])
@pytest.mark.parametrize("k_min", [1, 2])  # the last layer of the visited matrix; an accumulator
@pytest.mark.parametrize("deg", [2, 3, 33, 64, 255, 600])
def test_ids_between_whole_rows(vs, S, k_min, deg):
    """In-lists whose rows alternate between a slot's ids and more than a slot holds, so that ids and whole rows
    of one target follow each other in the list put aside; every copy also has ids in the words of the long rows."""
    rng = np.random.default_rng(deg)
    base = rng.choice(128, 100, replace=False)  # the long rows and half of the short ones share their words
    rows = []
    for j in range(1200):
        if j % 2:
            rows.append(np.concatenate([base, rng.choice(np.arange(128, S), j % 40, replace=False)]))
        else:
            rows.append(rng.choice(128 if j % 4 else S, 3 + j % 12, replace=False))
    lists = [(rng.integers(0, 600) + np.arange(deg)) % 1200 for t in range(100)]
    check(vs, layered(rows, lists), S, k_min, None)
