"""The one-launch BiCGSTAB where its split of the rows changes: one CTA, a few, one per SM, a slice too large for shared
memory; rows that a whole warp sums; rows without a diagonal. Checked through the residual of the returned vector in 64
bits and against the host-driven loop."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _random(n, per_row, seed, dense_rows=0):
    """Diagonally dominant CSR matrix: `per_row` random entries a row, `dense_rows` rows and columns that touch every 3rd node."""
    import scipy.sparse as sp

    rng = np.random.default_rng(seed)
    i = np.repeat(np.arange(n), per_row)
    j = rng.integers(0, n, i.size)
    keep = i != j
    a = sp.coo_matrix((-rng.random(keep.sum()), (i[keep], j[keep])), shape=(n, n)).tocsr()
    for k in range(dense_rows):
        hub = (k * 7919) % n
        others = np.arange(hub % 3, n, 3)
        others = others[others != hub]
        spoke = sp.coo_matrix((-rng.random(others.size) * 0.1, (np.full(others.size, hub), others)), shape=(n, n))
        a = a + spoke + spoke.T
    a = a + sp.diags(np.asarray(abs(a).sum(1)).ravel() * 1.1 + 0.5)
    a = a.tocsr()
    a.sort_indices()
    return a


@pytest.mark.parametrize("n,per_row,dense", [(1, 1, 0), (7, 2, 0), (500, 3, 0), (1023, 4, 2), (2049, 2, 1), (30_000, 1, 0), (30_000, 40, 0), (20_000, 3, 5),
                                             (60_000, 60, 0)])
def test_solution_satisfies_the_system(monkeypatch, n, per_row, dense):
    from nangila_spice.gpu import DeviceCsr

    a = _random(n, per_row, n + per_row, dense)
    b = np.random.default_rng(n).standard_normal(n)
    m = DeviceCsr(a.indptr, a.indices, a.data)
    x, it, rel, ok = m.solve(b, tol=1e-11, max_iter=400)
    assert ok and rel < 1e-11
    # the recurrence's residual drifts from the true one by rounding: a few units in the last place per iteration
    assert np.linalg.norm(b - a @ x) <= (1e-11 + 100 * (it + 1) * 2.3e-16) * np.linalg.norm(b)
    again, it2, _, _ = m.solve(b, tol=1e-11, max_iter=400)
    assert it2 == it and np.array_equal(x, again)
    # new values for the same pattern: the preconditioner on the device follows
    m.update_values(2.0 * a.data)
    half, _, _, ok = m.solve(b, tol=1e-11, max_iter=400)
    assert ok and np.linalg.norm(x - 2.0 * half) <= 1e-8 * np.linalg.norm(x)
    monkeypatch.setenv("NANGILA_SPMV_GRAPH", "0")
    host, it_host, _, ok = m.solve(b, tol=1e-11, max_iter=400)
    assert ok and np.linalg.norm(host - half) <= 1e-8 * np.linalg.norm(half)


def test_slices_too_large_for_shared_memory():
    from nangila_spice.gpu import DeviceCsr, tridiagonal

    n = 1_200_000  # 3.6 M entries: 24 K a CTA
    row_ptr, col, val = tridiagonal(n, diag=2.5, off=-1.0)
    b = np.random.default_rng(1).standard_normal(n)
    x, it, rel, ok = DeviceCsr(row_ptr, col, val).solve(b, tol=1e-11, max_iter=400)
    assert ok
    ax = 2.5 * x
    ax[1:] -= x[:-1]
    ax[:-1] -= x[1:]
    assert np.linalg.norm(b - ax) <= (1e-11 + 100 * (it + 1) * 2.3e-16) * np.linalg.norm(b)


def test_breakdown_and_limits():
    from nangila_spice.gpu import DeviceCsr

    # a skew-symmetric matrix: <r0, A r0> = 0, nothing to do
    m = DeviceCsr([0, 1, 2], [1, 0], [1.0, -1.0])
    x, it, _, ok = m.solve([1.0, 1.0])
    assert not ok and it == 0 and not x.any()
    a = _random(5000, 4, 3)
    m = DeviceCsr(a.indptr, a.indices, a.data)
    b = np.ones(5000)
    assert m.solve(b, max_iter=0)[1] == 0
    _, it, rel, ok = m.solve(b, tol=1e-30, max_iter=2)
    assert not ok and it == 4 and rel < 1.0
    x, it, _, ok = m.solve(np.zeros(5000))
    assert ok and it == 0 and not x.any()
