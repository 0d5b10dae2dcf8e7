"""The solver gathers as many entries of a row at once as the longest row of a warp has (three, five, or four at a time beyond): rows of every length
around these lines, alone and mixed, long rows that a whole warp sums among them, on one CTA and on many."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _matrix(n, lengths, rng):
    """Row i has lengths[i] entries (itself and neighbours to both sides), diagonally dominant, not symmetric."""
    rows = np.repeat(np.arange(n), lengths)
    row_ptr = np.concatenate([[0], np.cumsum(lengths)])
    place = np.arange(rows.size) - row_ptr[rows]
    col = np.clip(rows - lengths[rows] // 2, 0, n - lengths[rows]) + place
    val = -np.exp(0.3 * rng.standard_normal(rows.size))
    own = col == rows
    val[own] = 0.0
    val[own] = 0.05 + 1.1 * np.bincount(rows, -val, minlength=n)
    return row_ptr.astype(np.int32), col.astype(np.int32), val, rows


@pytest.mark.parametrize("n", [600, 40_001])
@pytest.mark.parametrize("lengths", [(1,), (2, 3), (3,), (4,), (3, 4), (5,), (5, 6), (6, 7, 8, 9), (64,), (65, 3), (1, 3, 5, 20, 70)])
def test_residual(lengths, n):
    from nangila_spice.gpu import DeviceCsr

    rng = np.random.default_rng(n + sum(lengths))
    row_ptr, col, val, rows = _matrix(n, rng.choice(lengths, n), rng)
    b = rng.standard_normal(n)
    m = DeviceCsr(row_ptr, col, val)
    x, iterations, _, converged = m.solve(b, tol=1e-11)
    assert converged and iterations < 400
    residual = b - np.bincount(rows, val * x[col], minlength=n)
    assert np.linalg.norm(residual) <= 1e-10 * np.linalg.norm(b)  # (the solver's own residual drifts by rounding only)
    assert np.array_equal(x, m.solve(b, tol=1e-11)[0])  # the same bits from run to run
