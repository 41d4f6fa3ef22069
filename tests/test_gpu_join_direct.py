"""Flat joins on vertex-id keys around the direct arrays' rule: keys below, at and
above the bound of a few entries per build row, the largest ids, unique and
repeated build keys, row counts around a vector load and a tile, either side
smaller, a row bound; counts and row multisets against numpy, and unique build keys
in probe order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def expect(ka, pa, kb, pb):
    rows = []
    where = {}
    for i, k in enumerate(kb.tolist()):
        where.setdefault(k, []).append(i)
    for i, k in enumerate(ka.tolist()):
        rows += [(k, int(pa[i]), int(pb[j])) for j in where.get(k, ())]
    return rows


@pytest.mark.parametrize("na,nb", [(1, 1), (3, 2), (5, 1023), (1024, 1025), (4097, 300), (2500, 2500), (70001, 20003)])
@pytest.mark.parametrize("top", [7, 65535, (1 << 22) - 1, 1 << 22, 0xFFFFFFFE, 0xFFFFFFFF])
@pytest.mark.parametrize("unique", [True, False])
def test_vid_joins(vs, na, nb, top, unique):
    rng = np.random.default_rng(na * 31 + nb + top % 1000 + unique)
    small, n_small = (min(na, nb), min(na, nb))
    if unique and top + 1 < n_small:
        pytest.skip("fewer keys than rows")
    pool = rng.integers(0, top + 1, 4 * max(na, nb), dtype=np.uint64).astype(np.uint32)
    pool[0] = top
    keys = np.unique(pool)[::-1]  # the largest first
    side = keys[:small] if unique and len(keys) >= small else rng.choice(keys, small)
    side = rng.permutation(side).astype(np.uint32)
    other = rng.choice(keys[: 3 * small], max(na, nb)).astype(np.uint32)
    if na != nb and top <= 7:
        other = other[: max(small + 1, 50)]  # few keys: keep the product small
    ka, kb = (other, side) if na >= nb else (side, other)
    if top <= 7:
        ka, kb = ka[:60], kb[:60]
    pa, pb = rng.integers(-(1 << 40), 1 << 40, len(ka)), rng.integers(0, 1 << 31, len(kb)).astype(np.uint32)
    a, b = vs.FlatTable.from_columns([ka, pa]), vs.FlatTable.from_columns([kb, pb])
    want = expect(ka, pa, kb, pb)
    for x, y in ((a, b), (b, a)):
        assert vs.hash_join(x, y, 0, 0, only_count=True)[1] == len(want)
    t, n, cut = vs.hash_join(a, b, 0, 0)
    assert n == len(want) and not cut
    got = list(zip(*(c.tolist() for c in t.columns())))
    assert sorted(got) == sorted(want)
    if len(np.unique(kb)) == len(kb) and len(kb) <= len(ka):  # b is the build side, one row a key
        assert got == want
    if len(want) > 1:
        t, n, cut = vs.hash_join(a, b, 0, 0, max_rows=len(want) // 2)
        part = list(zip(*(c.tolist() for c in t.columns())))
        assert cut and n == len(want) and len(part) == len(want) // 2 and set(part) <= set(want)
