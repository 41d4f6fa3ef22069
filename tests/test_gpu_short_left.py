"""Rows that a short-mode hop left in their slots, of every length a slot holds and more, written out for a hop
that reads rows."""
import numpy as np
import pytest

from oracle import pyoracle as O
from vertexsurge_gb300 import graphgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S", [2048, 4100, 8200])  # slots of 16, 32 and 64 entries
def test_rows_left_in_slots_before_a_push(vs, S):
    rng = np.random.default_rng(S)
    src, dst = [], []
    for j in range(700):  # middle 9000 + j gathers 1 + j % 70 sources, its copy 10000 + j the same a hop later
        n = 1 + j % 70
        src += list(rng.choice(S, n, replace=False)) + [9000 + j]
        dst += [9000 + j] * n + [10_000 + j]
    src += list(10_000 + rng.integers(0, 700, 2000))
    dst += list(11_000 + rng.integers(0, 200, 2000))
    g = graphgen.from_edges(11_200, np.array(src, np.uint32), np.array(dst, np.uint32))
    sources = np.arange(S, dtype=np.uint32)
    dg = vs.DeviceGraph.from_host(g)
    plan = vs.ExpandPlan(dg, S, vs.make_params(1, 3, "shortest", "forward", strategy="pull", short_share=2.0))
    plan.set_hop_strategies([0, vs.STRAT_PULL, vs.STRAT_PULL, vs.STRAT_PUSH])
    for _ in range(2):
        plan.run(sources)
        st = plan.stats()
        assert st["short_pull"][2] and list(st["strategy"][1:4]) == [1, 1, 2], st
        assert np.array_equal(plan.result().download(), O.vexpand(g, sources, 1, 3, "shortest", "forward")[0])
