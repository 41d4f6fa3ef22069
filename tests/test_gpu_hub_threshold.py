"""hub_threshold above the longest list: no vertex's list is cut, in dense and short-mode hops."""
import numpy as np
import pytest

from oracle import pyoracle as O
from vertexsurge_gb300 import graphgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,share", [(40, 0.0), (700, 0.0), (2200, 2.0)])
def test_no_list_is_cut(vs, S, share):
    V, d = 80_000, 70_000  # vertex 0 has 70,000 in-neighbours
    rng = np.random.default_rng(S)
    src = np.concatenate([np.arange(1, d + 1), rng.integers(0, V, 60_000)]).astype(np.uint32)
    dst = np.concatenate([np.zeros(d), rng.integers(0, V, 60_000)]).astype(np.uint32)
    g = graphgen.from_edges(V, src, dst)
    dg = vs.DeviceGraph.from_host(g)
    sources = graphgen.sample_sources(V, S, seed=2)
    want = O.vexpand(g, sources, 1, 3, "shortest", "forward")[0]
    made = []
    for hub in (0, 69_000, 100_000, 0xFFFFFFFF):
        n0 = vs.kernel_launches()
        plan = vs.ExpandPlan(dg, S, vs.make_params(1, 3, "shortest", "forward", strategy="pull", hub_threshold=hub,
                                                   short_share=share))
        made.append(vs.kernel_launches() - n0)
        plan.run(sources)
        assert np.array_equal(plan.result().download(), want), hub
        plan.free()
    assert made[0] == made[1] > made[2] == made[3]  # with pieces to write, and without
