"""Column counts with one and with four columns a group of lanes: matrices around the size between them, tall
ones of few columns."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols", [(64, 622_591), (64, 622_593), (130, 311_297), (1000, 77_830), (200_000, 5), (4100, 19_457)])
def test_counts(vs, rows, cols):
    rng = np.random.default_rng(cols)
    w = rng.integers(0, 1 << 63, (cols, (rows + 63) // 64), dtype=np.uint64) & rng.integers(0, 1 << 63, (cols, 1), dtype=np.uint64)
    if rows % 64:
        w[:, -1] &= np.uint64((1 << (rows % 64)) - 1)
    m = vs.BitMatrix.from_logical(w, rows, cols)
    got = vs.matrix_column_count(m, 0).columns()
    assert np.array_equal(got[-1].astype(np.int64), np.bitwise_count(w).sum(1).astype(np.int64))
