"""The thread-per-row product and the rule that chooses it: row counts around a CTA, empty rows, rows around the four entries
that are in flight, matrices just inside and just outside the rule (which take the staged kernel)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 255, 256, 257, 20_003])
@pytest.mark.parametrize("longest,mean", [(1, 1), (4, 2), (5, 3), (16, 6), (17, 3), (16, 9)])
def test_product_matches_the_host(n, longest, mean):
    from nangila_spice.gpu import DeviceCsr

    rng = np.random.default_rng(n * 100 + longest + mean)
    lengths = np.minimum(rng.integers(0, 2 * mean + 1, n), min(longest, n))
    lengths[rng.integers(0, n)] = min(longest, n)  # the longest row is there
    row_ptr = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    # (an entry may name a column twice; both count)
    col = rng.integers(0, n, row_ptr[-1]).astype(np.int32)
    val = rng.standard_normal(col.size)
    x = rng.standard_normal(n)
    rows = np.repeat(np.arange(n), lengths)
    prod = val * x[col]
    want = np.bincount(rows, prod, minlength=n)
    size = np.bincount(rows, np.abs(prod), minlength=n)
    # at most one rounding per entry for the product and one for the sum, on either side
    bound = 2.3e-16 * 2 * (lengths + 1) * size
    m = DeviceCsr(row_ptr, col, val)
    assert (np.abs(m.matvec(x) - want) <= bound).all()
    m.update_values(-val)
    assert (np.abs(m.matvec(x) + want) <= bound).all()
