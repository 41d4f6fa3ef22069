"""What a plan allocates stays within its footprint, which the serving loop admits by."""
import ctypes as C

import numpy as np
import pytest

from vertexsurge_gb300 import graphgen
from vertexsurge_gb300._abi import plan_footprint

pytestmark = pytest.mark.gpu


def used():
    """Bytes in use in the device's default pool."""
    cu = C.CDLL("libcuda.so.1")
    pool, n = C.c_void_p(), C.c_uint64()
    assert cu.cuDeviceGetDefaultMemPool(C.byref(pool), 0) == 0
    assert cu.cuMemPoolGetAttribute(pool, 7, C.byref(n)) == 0  # used, current
    return n.value


@pytest.mark.parametrize("direction", ["forward", "both"])
@pytest.mark.parametrize("S,slice_words", [(100, 0), (512, 0), (512, 2), (2048, 0), (4096, 0)])
@pytest.mark.parametrize("hub", [0, 3, 600])
def test_plan_within_its_footprint(vs, direction, S, slice_words, hub):
    """20,000 vertices of 33 entries in either list: both together exceed the threshold of narrow rows, and are two
    pieces, neither longer than one."""
    V, d = 20_000, 33
    src = np.repeat(np.arange(V), d)
    g = graphgen.from_edges(V, src.astype(np.uint32), ((src + np.tile(np.arange(1, d + 1) * 577, V)) % V).astype(np.uint32))
    dg = vs.DeviceGraph.from_host(g)
    p = vs.make_params(1, 3, "shortest", direction, slice_words=slice_words, hub_threshold=hub)
    vs.release_cached()
    before = used()
    plan = vs.ExpandPlan(dg, S, p)
    got = used() - before
    assert got <= plan_footprint(dg, S, p) + 40 * 512  # an allocation is rounded up to 512 bytes
    plan.free()
