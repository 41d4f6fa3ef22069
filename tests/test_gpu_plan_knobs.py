"""Knobs of an expand plan that no longer choose a kernel."""
import numpy as np
import pytest

from oracle import pyoracle as O
from vertexsurge_gb300 import autotune, graphgen

pytestmark = pytest.mark.gpu


def test_calls_that_differ_in_the_kernel_kind_share_a_plan(vs):
    g = graphgen.rmat(10, 8, seed=5)
    dg = vs.DeviceGraph.from_host(g)
    src = graphgen.sample_sources(g.V, 60, seed=1)
    vs.release_cached()
    launches = []
    for kind in (0, 0, 3, 7):
        n0 = vs.kernel_launches()
        m, _, _ = vs.expand(dg, src, 1, 2, "shortest", "forward", pull_kernel=kind)
        launches.append(vs.kernel_launches() - n0)
        m.free()
    assert launches[0] > launches[1] == launches[2] == launches[3]  # the first made the plan


def test_tune_times_a_kernel_once(vs):
    g = graphgen.rmat(10, 8, seed=6)
    dg = vs.DeviceGraph.from_host(g)
    src = graphgen.sample_sources(g.V, 33, seed=1)
    out = autotune.tune(dg, src, 1, 2, repeats=1, pull_kinds=(0, 1, 2, 3), sparse_fracs=(0.002, 0.02), hub_thresholds=(0,),
                        short_shares=(0.0,))
    times = {}
    for row in out["table"]:
        times.setdefault(row["sparse_frac"], set()).add(row["ms"])
    assert len(out["table"]) == 8 and [len(t) for t in times.values()] == [1, 1] and out["pull_kind"] == 0
    with pytest.raises(vs.VsError):
        autotune.tune(dg, src[:9], 1, 2, repeats=1, pull_kinds=(8,))
