"""Plans of different widths side by side: the kernels' shared memory is that of the widest."""
import numpy as np
import pytest

from oracle import pyoracle as O
from vertexsurge_gb300 import graphgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("one_shot", [False, True])
def test_wide_plan_after_a_narrower_one(vs, one_shot):
    g = graphgen.zipf(1500, 12_000, 2.0, 400, seed=3)
    dg = vs.DeviceGraph.from_host(g)
    want, plans = {}, {}
    for S in (32_768, 16_000, 16_384, 32_768, 16_000):  # 256, 125 and 128 cells a row
        src = np.resize(np.arange(g.V, dtype=np.uint32), S)
        if S not in want:
            want[S] = O.vexpand(g, src, 1, 3, "shortest", "forward")[0]
        if one_shot:
            m, _, st = vs.expand(dg, src, 1, 3, "shortest", "forward", strategy="pull", short_share=2.0, stats=True)
            assert any(st["short_pull"])
        else:
            if S not in plans:
                plans[S] = vs.ExpandPlan(dg, S, vs.make_params(1, 3, "shortest", "forward", strategy="pull",
                                                               short_share=2.0))
            plans[S].run(src)
            m = plans[S].result()
        assert np.array_equal(m.download(), want[S]), S
        m.free()
