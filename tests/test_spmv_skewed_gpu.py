"""The thread-per-row product where rows do not lie where their share of the entries would put them: no entries at all, all of them in the first or
the last rows, few rows; on both sides of the size from which rows are fetched ahead."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 257, 100_003, 2_000_001])  # the last one above the size from which rows are fetched ahead
@pytest.mark.parametrize("where", ["none", "first", "last", "one"])
def test_skewed_rows(where, n):
    from nangila_spice.gpu import DeviceCsr

    rng = np.random.default_rng(n)
    lengths = np.zeros(n, dtype=np.int64)
    few = max(1, n // 8)
    if where == "first":
        lengths[:few] = min(16, n)
    elif where == "last":
        lengths[-few:] = min(16, n)
    elif where == "one":
        lengths[n // 2] = 1
    row_ptr = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    col = rng.integers(0, n, row_ptr[-1]).astype(np.int32)
    val = rng.standard_normal(col.size)
    x = rng.standard_normal(n)
    rows = np.repeat(np.arange(n), lengths)
    want = np.bincount(rows, val * x[col], minlength=n)
    size = np.bincount(rows, np.abs(val * x[col]), minlength=n)
    got = DeviceCsr(row_ptr, col, val).matvec(x)
    assert (np.abs(got - want) <= 2.3e-16 * 2 * (lengths + 1) * size).all()  # one rounding per product and per sum, on either side
