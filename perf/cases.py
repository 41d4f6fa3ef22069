"""The work whose speed this framework is judged by: calls a user's program makes through the
public entry points, on graphs and tables generated on the GPU from a seed.

Graphs follow the repository's two families: "zipf" (out-degree ~ Zipf(2.1) capped at 50,000, uniform
targets: the power-law social graphs of the pattern query and the batches) and "rmat" (R-MAT,
a=0.57 b=c=0.19, edge factor 16).  A program keeps the graph resident and, where it repeats one query
shape, an expand plan; sources, targets, pairs and key tables are new per query.

Results are bit matrices, vertex ids and counts: whole numbers that have to come out the same.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import vertexsurge_gb300 as vs
from vertexsurge_gb300 import batch

DEV = "cuda"
_ready = {}


def _stream():
    """The stream captured batches run on (capture refuses the default stream)."""
    if "stream" not in _ready:
        _ready["stream"] = torch.cuda.Stream()
    return _ready["stream"]


def _init():
    if "init" not in _ready:
        vs.init(torch.cuda.current_device())
        _ready["init"] = True


# ---- inputs -------------------------------------------------------------------------------------


def _gen(seed, salt=0):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 1000003 + salt)
    return g


def _lists(V, major, minor):
    """CSR of distinct (major, minor) pairs without self-loops: int64 offsets, sorted 32-bit ids."""
    key = (major * V + minor)[major != minor]
    key = torch.sort(key).values
    keep = torch.ones_like(key, dtype=torch.bool)
    keep[1:] = key[1:] != key[:-1]
    key = key[keep]
    del keep
    major = key // V
    off = torch.zeros(V + 1, dtype=torch.int64, device=DEV)
    off[1:] = torch.cumsum(torch.bincount(major, minlength=V), 0)
    return off, (key - major * V).to(torch.int32), major


def _zipf_edges(V, E, seed, alpha=2.1, cap=50_000):
    inv = -1.0 / (alpha - 1.0)
    cap = min(cap, V - 1)
    grid = ((torch.arange(1 << 18, device=DEV, dtype=torch.float64) + 0.5) / (1 << 18)).pow(inv)
    lo, hi = 0.01, 1000.0
    for _ in range(30):  # the scale that gives E edges
        mid = 0.5 * (lo + hi)
        if float((grid * mid).floor().clamp_(max=cap).mean()) * V < E:
            lo = mid
        else:
            hi = mid
    g = _gen(seed, 1)
    u = torch.rand(V, device=DEV, dtype=torch.float64, generator=g).clamp_(min=1e-12)
    deg = (u.pow(inv) * lo).floor().clamp_(max=cap).to(torch.int64)
    src = torch.repeat_interleave(torch.arange(V, device=DEV), deg)
    return src, torch.randint(0, V, (src.numel(),), device=DEV, generator=g)


def _rmat_edges(scale, ef, seed, a=0.57, b=0.19, c=0.19):
    g = _gen(seed, 2)
    m = ef << scale
    u = torch.zeros(m, dtype=torch.int64, device=DEV)
    v = torch.zeros(m, dtype=torch.int64, device=DEV)
    for _ in range(scale):
        r = torch.rand(m, device=DEV, generator=g)
        u = (u << 1) | (r >= a + b)
        v = (v << 1) | (((r >= a) & (r < a + b)) | (r >= a + b + c))
    return u, v


def _graph(case, seed, edges=False):
    """A directed graph resident on the GPU with both list directions, and its edge table if wanted."""
    V = case["V"]
    if case["graph"] == "zipf":
        src, dst = _zipf_edges(V, V * case["degree"], seed)
    else:
        src, dst = _rmat_edges(V.bit_length() - 1, case["degree"], seed)
    off, adj, src = _lists(V, src, dst)
    del dst
    roff, radj, _ = _lists(V, adj.to(torch.int64), src)
    torch.cuda.synchronize()
    dg = vs.DeviceGraph(V, adj.numel(), off, adj, roff, radj)
    table = [t.to(torch.int32).cpu().numpy().view(np.uint32) for t in (src, adj)] if edges else None
    del off, adj, src, roff, radj
    torch.cuda.empty_cache()  # the framework has an allocator of its own
    return (dg, table) if edges else dg


def _ids(V, n, seed, salt):
    """n distinct vertex ids, ascending, as a program samples its start vertices (host uint32)."""
    rng = np.random.default_rng([int(seed), salt])
    return np.sort(rng.choice(V, n, replace=False)).astype(np.uint32)


def _keys(V, n, seed, salt, skew=1.2):
    """n vertex ids, rank r of a random order (the seed's) drawn with probability ~ r^-skew (host uint32)."""
    u = torch.rand(n, device=DEV, dtype=torch.float64, generator=_gen(seed, salt))
    r = (1.0 - u).pow_(-1.0 / (skew - 1.0)).clamp_(max=1e15).to(torch.int64).sub_(1).remainder_(V)
    return torch.randperm(V, device=DEV, generator=_gen(seed, 10))[r].to(torch.int32).cpu().numpy().view(np.uint32)


# ---- device results as tensors ------------------------------------------------------------------


class _Mem:
    """Device memory of a framework handle, which lives as long as this does."""

    def __init__(self, ptr, shape, typestr, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (int(ptr), False), "version": 2}


def _matrix(m):
    """A bit matrix's words: int64 [cols, words per column]."""
    i = m.info()
    return torch.as_tensor(_Mem(i.words, (i.cols, i.wpc), "<i8", m), device=DEV)


def _columns(t):
    """A flat table's columns as tensors (vertex ids as int32)."""
    out = []
    _, rows, types = t.info()
    for c, kind in enumerate(types):
        p = ctypes.c_void_p()
        vs.check(vs.lib().vs_flat_column(t.h, c, ctypes.byref(p)))
        wide = kind == vs.T_I64
        out.append(torch.as_tensor(_Mem(p.value, (rows,), "<i8" if wide else "<i4", t), device=DEV) if rows else
                   torch.empty(0, dtype=torch.int64 if wide else torch.int32, device=DEV))
    return out


# ---- the cases ----------------------------------------------------------------------------------


def listed():
    return [
        # an interactive query on a small resident graph: one call, everything stays in L2, latency counts
        dict(name="expand_small", kind="expand", api="call", graph="rmat", V=1 << 16, degree=16, S=512, path="any",
             k_min=1, k_max=3, direction="forward"),
        # few start vertices on a million-vertex social graph: the narrowest rows, one call
        dict(name="expand_narrow", kind="expand", api="call", graph="zipf", V=1_000_000, degree=30, S=64,
             path="shortest", k_min=1, k_max=4, direction="forward"),
        # a deep neighbourhood, both directions, an odd source count; the reach saturates before the last hop
        dict(name="expand_both", kind="expand", api="plan", graph="rmat", V=1 << 20, degree=16, S=1_001,
             path="shortest", k_min=1, k_max=5, direction="both"),
        # walks of two or three steps against the edges: layers accumulated into a union, no visited set
        dict(name="expand_walks", kind="expand", api="plan", graph="zipf", V=1_000_000, degree=30, S=2_048,
             path="any", k_min=2, k_max=3, direction="backward"),
        # the headline expand: 4,096 sources, four hops, 10M vertices and 300M edges
        dict(name="expand_wide", kind="expand", api="plan", graph="zipf", V=10_000_000, degree=30, S=4_096,
             path="shortest", k_min=1, k_max=4, direction="forward"),
        # hop distances of pairs (who is how far from whom), up to six hops
        dict(name="pair_distances", kind="pairs", graph="rmat", V=1 << 18, degree=16, S=3_000, k_max=6),
        # the whole pattern query (two expands, join count, triangle closing) on the million-vertex graph
        dict(name="pattern", kind="pattern", graph="zipf", V=1_000_000, degree=30, S=4_096, k_max=4),
        # a batch of uneven queries (sources, depths, key tables) replayed as one captured launch
        dict(name="batch", kind="batch", graph="zipf", V=1_000_000, degree=30, queries=16, s_max=4_096, l_max=5,
             rows=1_000_000),
        # exact count of a join of two skewed key tables
        dict(name="join_count", kind="join_count", V=10_000_000, rows_a=10_000_000, rows_b=10_000_000),
        # tuples joined with the vertices' property table (a row per vertex, in no order), rows written out
        dict(name="join_rows", kind="join_rows", V=1_000_000, rows_a=4_000_000),
        # directed triangles a->b, a->c, b->c from the edge table: their number, and rows up to the caller's bound
        dict(name="triangle_rows", kind="triangles", graph="rmat", V=1 << 16, degree=16, limit=20_000_000),
        # the report after an expand: chosen columns, their transpose, vertices ranked by how many reach them
        dict(name="report", kind="report", graph="zipf", V=1_000_000, degree=30, S=4_096, k_max=3, targets=200_000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _odd_graph(rng, v_lo, v_hi):
    if rng.random() < 0.5:
        s = rng.randint(v_lo.bit_length(), v_hi.bit_length() - 1)
        return dict(graph="rmat", V=1 << s, degree=rng.choice([8, 16]))
    return dict(graph="zipf", V=_log(rng, v_lo, v_hi), degree=rng.randint(8, 30))


def draw(rng):
    kind = rng.choice(["expand", "expand", "expand", "expand", "pairs", "pattern", "batch", "join_count", "join_rows",
                       "triangles", "report"])
    if kind == "expand":
        while True:
            path = rng.choice(["any", "shortest", "shortest"])
            k_max = rng.randint(1, 6)
            c = dict(kind=kind, api=rng.choice(["call", "plan"]), **_odd_graph(rng, 1 << 14, 2_000_000),
                     S=_log(rng, 1, 8_192), path=path, k_min=rng.randint(0, min(2, k_max)), k_max=k_max,
                     direction=rng.choice(["forward", "forward", "backward", "both"]))
            # bounded as a dense pass over every edge of every hop would cost
            if c["V"] * c["degree"] * (2 if c["direction"] == "both" else 1) * k_max * max(32, c["S"] / 8) < 4e10:
                return c
    if kind == "pairs":
        return dict(kind=kind, **_odd_graph(rng, 1 << 14, 1 << 19), S=_log(rng, 16, 4_096), k_max=rng.randint(3, 8))
    if kind == "pattern":
        return dict(kind=kind, **_odd_graph(rng, 1 << 15, 1_000_000), S=_log(rng, 64, 4_096), k_max=rng.randint(2, 4))
    if kind == "batch":
        return dict(kind=kind, **_odd_graph(rng, 1 << 16, 1_000_000), queries=rng.randint(5, 20), s_max=_log(rng, 256, 4_096),
                    l_max=rng.randint(2, 5), rows=_log(rng, 100_000, 1_000_000))
    if kind == "join_count":
        return dict(kind=kind, V=_log(rng, 100_000, 10_000_000), rows_a=_log(rng, 10_000, 10_000_000),
                    rows_b=_log(rng, 10_000, 10_000_000))
    if kind == "join_rows":
        V = _log(rng, 1_000, 2_000_000)
        return dict(kind=kind, V=V, rows_a=V + _log(rng, 1_000, 6_000_000 - V))
    if kind == "triangles":
        c = _odd_graph(rng, 1 << 12, 1 << 16)
        return dict(kind=kind, **c, limit=c["V"] * (4 if c["graph"] == "rmat" else 1))
    c = _odd_graph(rng, 1 << 15, 1_000_000)
    return dict(kind=kind, **c, S=_log(rng, 64, 4_096), k_max=rng.randint(1, 3),
                targets=_log(rng, 1_000, c["V"] // 2))


def prepare(case, seed):
    _init()
    kind = case["kind"]
    st = {"case": case}
    if kind in ("join_count", "join_rows"):
        V, na = case["V"], case["rows_a"]
        rng = np.random.default_rng([int(seed), 5])
        ka = _keys(V, na, seed, 11)
        if kind == "join_count":
            st["a"] = vs.FlatTable.from_columns([ka])
            st["b"] = vs.FlatTable.from_columns([_keys(V, case["rows_b"], seed, 12)])
        else:  # (vertex, amount) tuples against (vertex, property) rows
            st["a"] = vs.FlatTable.from_columns([ka, rng.integers(-(1 << 40), 1 << 40, na)])
            st["b"] = vs.FlatTable.from_columns([rng.permutation(V).astype(np.uint32), rng.integers(0, 1 << 40, V)])
        torch.cuda.empty_cache()
        return st
    if kind == "triangles":  # the edge table a plan's base scan holds: (source, target) rows in list order
        dg, table = _graph(case, seed, edges=True)
        st["g"], st["base"] = dg, vs.FlatTable.from_columns(table)
        st["deps"] = [dict(graph=dg, direction="forward", base_col=0), dict(graph=dg, direction="forward", base_col=1)]
        return st
    dg = st["g"] = _graph(case, seed)
    if kind == "expand":
        src = _ids(dg.V, case["S"], seed, 1)
        if case["api"] == "plan":
            st["plan"] = vs.ExpandPlan(dg, case["S"], vs.make_params(case["k_min"], case["k_max"], case["path"],
                                                                     case["direction"]))
            st["src"] = torch.from_numpy(src.view(np.int32)).to(DEV)
        else:
            st["src"] = src
    elif kind == "pairs":
        rng = np.random.default_rng([int(seed), 2])
        st["src"] = rng.integers(0, dg.V, case["S"], dtype=np.uint32)
        st["dst"] = rng.integers(0, dg.V, case["S"], dtype=np.uint32)
    elif kind == "pattern":
        S = case["S"]
        st["A"] = vs.ExpandPlan(dg, S, vs.make_params(1, case["k_max"], "shortest"))
        st["B"] = vs.ExpandPlan(dg, S, vs.make_params(1, 2, "shortest"))
        st["P"] = vs.ExpandPlan(dg, S, vs.make_params(1, 1, "any"))
        st["sa"] = torch.from_numpy(_ids(dg.V, S, seed, 3).view(np.int32)).to(DEV)
        st["sb"] = torch.from_numpy(_ids(dg.V, S, seed, 4).view(np.int32)).to(DEV)
    elif kind == "batch":
        shape = np.random.default_rng([case["queries"], case["s_max"], case["l_max"], case["rows"]])
        qs = []
        for i in range(case["queries"]):
            S = int(np.exp(shape.uniform(np.log(64), np.log(case["s_max"]))))
            rows = int(shape.integers(case["rows"] // 10, case["rows"] + 1))
            qs.append(batch.Query(_ids(dg.V, S, seed, 100 + i), int(shape.integers(2, case["l_max"] + 1)),
                                  _keys(dg.V, rows, seed, 100 + i)))
        st["batch"] = batch.Batch(dg, qs, case["s_max"], _stream())
        st["batch"].capture()
    else:
        st["m"], _, _ = vs.expand(dg, _ids(dg.V, case["S"], seed, 1), 1, case["k_max"], "shortest", "forward")
        st["targets"] = _ids(dg.V, case["targets"], seed, 6)
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "expand":
        if case["api"] == "plan":
            st["plan"].run(st["src"])
            return _matrix(st["plan"].result())
        m, _, _ = vs.expand(st["g"], st["src"], case["k_min"], case["k_max"], case["path"], case["direction"])
        return _matrix(m)
    if kind == "pairs":
        _, dist, _ = vs.expand(st["g"], st["src"], 1, case["k_max"], "find_shortest", "forward", targets=st["dst"])
        return dist
    if kind == "pattern":
        st["A"].run(st["sa"])
        st["B"].run(st["sb"])
        A, B = st["A"].result(), st["B"].result()
        _, joined, _ = vs.hash_join(A, B, 1, 1, only_count=True)
        st["P"].run(st["sa"])
        adj = [dict(graph=st["g"], direction="forward", base_col=0), dict(graph=st["g"], direction="forward", base_col=1)]
        _, triangles, _ = vs.mintersect(st["P"].result(), adj, st["g"].V, only_count=True)
        return {"joined": joined, "triangles": triangles, "A": _matrix(A), "B": _matrix(B)}
    if kind == "batch":
        st["batch"].launch()
        return {"counts": st["batch"].d_counts, "last_wave": _matrix(st["batch"].plans[-1].result())}
    if kind == "join_count":
        return vs.hash_join(st["a"], st["b"], 0, 0, only_count=True)[1]
    if kind == "join_rows":
        t, n, _ = vs.hash_join(st["a"], st["b"], 0, 0)
        return [n] + _columns(t)
    if kind == "triangles":
        t, n, _ = vs.mintersect(st["base"], st["deps"], st["g"].V, max_rows=case["limit"])
        return [n] + _columns(t)
    chosen = st["m"].select(st["targets"])
    by_source = chosen.convert(True)
    ranked = vs.matrix_column_count(st["m"], "desc")
    return {"reached": st["m"].count(), "by_source": _matrix(by_source), "ranked": _columns(ranked)}


def _reach(case, hops):
    """Vertices and edges that hops steps from the sources can touch, in expectation."""
    V, d = case["V"], case["degree"] * (2 if case.get("direction") == "both" else 1)
    pairs = [float(case["S"])]
    for _ in range(hops):
        pairs.append(min(pairs[-1] * d, 1e18))
    rows = min(V, sum(pairs))
    edges = min(V, sum(pairs[:-1])) * d
    return rows, edges


def _words(S):
    return 2 * ((S + 127) // 128)


def _expand_bytes(case, hops, S=None):
    """Offsets and lists of the vertices that are left, the sources, the result's non-zero rows written."""
    c = dict(case, S=S or case["S"])
    rows, edges = _reach(c, hops)
    return 8 * rows + 4 * edges + 4 * c["S"] + 8 * _words(c["S"]) * rows


def work(case):
    kind = case["kind"]
    if kind == "expand":
        b = _expand_bytes(case, case["k_max"])
    elif kind == "pairs":  # a distance per pair; the frontier has to be followed from every source
        rows, edges = _reach(case, min(case["k_max"], 3))
        b = 8 * rows + 4 * edges + 12 * case["S"]
    elif kind == "pattern":
        V, S = case["V"], case["S"]
        b = _expand_bytes(case, case["k_max"]) + _expand_bytes(case, 2)
        b += 8 * _words(S) * _reach(case, 2)[0] * 2  # the join reads the rows both can hold
        b += S * case["degree"] * 4 * 2
    elif kind == "batch":
        per = case["s_max"] / math.log(max(2.0, case["s_max"] / 64))
        b = case["queries"] * (_expand_bytes(case, (2 + case["l_max"]) // 2, S=max(64, int(per))) + 4 * 0.55 * case["rows"])
    elif kind == "join_count":
        b = 4 * (case["rows_a"] + case["rows_b"])
    elif kind == "join_rows":
        b = 12 * (case["rows_a"] + case["V"]) + 20 * case["rows_a"]
    elif kind == "triangles":
        E = case["V"] * case["degree"]
        b = 8 * case["V"] + 4 * E + 8 * E + 12 * case["limit"]
    else:
        W, V = _words(case["S"]), case["V"]
        b = 8 * W * V + 8 * W * case["targets"] + case["S"] * case["targets"] / 8 + 12 * V
    return {"bytes": float(b), "flops": 0.0}


def exact(case, seed):
    """The join count from plain torch; bit matrices and listings have no short 64-bit form."""
    if case["kind"] != "join_count":
        return None
    V, na, nb = case["V"], case["rows_a"], case["rows_b"]
    a, b = _keys(V, na, seed, 11), _keys(V, nb, seed, 12)
    a, b = (torch.bincount(torch.from_numpy(k.astype(np.int64)).to(DEV), minlength=V) for k in (a, b))
    return int((a * b).sum())
