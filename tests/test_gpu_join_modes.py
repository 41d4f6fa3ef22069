"""Flat joins that list rows, by what their build keys are: unique, repeated (within a warp, beyond the first
rows of the build, one key alone), at or above the array's bound, 64-bit; row counts around the tiles of the
prefix sums, probe rows without a match over more than a block's range."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIRST = 512 * 152  # build rows that are looked at first


def expect(ka, kb):
    """(key, row of a, row of b) of every match, sorted."""
    order = np.argsort(kb, kind="stable")
    lo, hi = np.searchsorted(kb[order], ka, "left"), np.searchsorted(kb[order], ka, "right")
    ia = np.repeat(np.arange(len(ka)), hi - lo)
    at = np.arange(len(ia)) - np.repeat(np.cumsum(hi - lo) - (hi - lo), hi - lo) + np.repeat(lo, hi - lo)
    return np.array(sorted(zip(ka[ia].tolist(), ia.tolist(), order[at].tolist())), dtype=np.int64).reshape(-1, 3)


@pytest.mark.parametrize("nb", [1, 2, 33, 1023, 1024, 1025, FIRST, FIRST + 1, 540_000])
@pytest.mark.parametrize("keys", ["unique", "last", "warp", "one", "mixed", "high", "i64"])
def test_rows(vs, nb, keys):
    rng = np.random.default_rng(nb + len(keys))
    kb = rng.permutation(max(2 * nb, 8))[:nb].astype(np.int64)
    if keys == "last":  # the only repeated key is the last row's
        kb[-1] = kb[0]
    elif keys == "warp":
        kb[nb // 2:nb // 2 + 5] = kb[nb // 2]
    elif keys == "one":
        kb[:] = 5
    elif keys in ("mixed", "i64"):
        kb = rng.integers(0, max(nb // 2, 1), nb)
    elif keys == "high":
        kb[nb // 3] = max(1 << 22, 12 * nb // 4 * 4) + nb % 2
    np_ = 40 if keys == "one" else max(nb + 1, 3000)
    ka = np.where(rng.random(np_) < 0.3, rng.choice(kb, np_), int(kb.max()) + 1 + rng.integers(0, 99, np_))
    if keys == "one":
        nb = min(nb, 2000)
        kb = kb[:nb]
    t = np.int64 if keys == "i64" else np.uint32
    ka, kb = ka.astype(t), kb.astype(t)
    a = vs.FlatTable.from_columns([ka, np.arange(len(ka), dtype=np.uint32)])
    b = vs.FlatTable.from_columns([kb, np.arange(len(kb), dtype=np.int64)])
    want = expect(ka, kb)
    for _ in range(2):
        r, n, cut = vs.hash_join(a, b, 0, 0)
        assert n == len(want) and not cut
        got = np.stack([c.astype(np.int64) for c in r.columns()], 1)
        if len(kb) <= len(ka):
            assert np.all(np.diff(got[:, 1]) >= 0)  # probe order
        assert np.array_equal(got[np.lexsort(got.T[::-1])], want)
    assert vs.hash_join(a, b, 0, 0, only_count=True)[1] == len(want)
    if len(want) > 2:
        r, n, cut = vs.hash_join(a, b, 0, 0, max_rows=len(want) // 2)
        part = np.stack([c.astype(np.int64) for c in r.columns()], 1)
        assert n == len(want) and cut and len(part) == len(want) // 2
        assert len(np.unique(part, axis=0)) == len(part) and set(map(tuple, part[:500].tolist())) <= set(map(tuple, want.tolist()))
