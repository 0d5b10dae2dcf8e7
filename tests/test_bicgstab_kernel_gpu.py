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


def _one_way_chain(rng, n, gain=None, back=None):
    """Stages that drive the next one and feel little of it, as amplifiers do: lower bidiagonal but for a small reverse coupling."""
    a = np.eye(n)
    for i in range(1, n):
        a[i, i - 1] = -(gain or rng.uniform(1.0, 3.2))
        a[i - 1, i] = -(back or 10.0 ** rng.uniform(-10, -6))
    b = np.zeros(n)
    b[0] = 1.0
    return a, b


def _driven(rng, n):
    """One node drives all others and none drives it (a controlled source)."""
    a = np.diag(rng.uniform(0.5, 4.0, n))
    a[1:, 0] = rng.uniform(-3.0, 3.0, n - 1)
    b = np.zeros(n)
    b[0] = rng.uniform(0.5, 2.0)
    return a, b


def _solve_dense(a, b, **kw):
    from nangila_spice.gpu import DeviceCsr
    import scipy.sparse as sp

    c = sp.csr_matrix(a)
    m = DeviceCsr(c.indptr, c.indices, c.data)
    x, it, rel, ok = m.solve(b, **kw)
    m.close()
    return x, it, rel, ok, np.linalg.norm(b - a @ x) / np.linalg.norm(b)


def _check_residual(a, b, must_converge):
    x, it, rel, ok, true = _solve_dense(a, b, tol=1e-10, max_iter=400)
    assert ok or not must_converge, (it, rel, true)
    if ok:
        # what the recurrence's residual may have drifted by: rounding of the largest iterate, which is of the size of the solution times
        # the matrix (gains multiply along a chain), a few units in the last place per iteration
        size = np.linalg.norm(abs(a) @ abs(np.linalg.solve(a, b))) / np.linalg.norm(b)
        assert rel < 1e-10 and true <= 1e-10 + 100 * (it + 1) * 2.3e-16 * max(size, 1.0), (it, rel, true)


@pytest.mark.parametrize("n", [5, 9])
def test_steps_that_remove_nearly_all_of_the_residual(n):
    # the omega step leaves 1e-8 of s or less: a residual put together from sums of s and t is nothing but rounding there
    a, b = _one_way_chain(None, n, gain=5.0, back=1e-8)
    _check_residual(a, b, must_converge=n == 5)


def test_one_way_systems_end_where_their_residual_says():
    rng = np.random.default_rng(0)
    for _ in range(150):
        _check_residual(*_one_way_chain(rng, int(rng.integers(3, 12))), must_converge=False)
        _check_residual(*_driven(rng, int(rng.integers(2, 4))), must_converge=True)
    # <r0, r> of this one cancels to zero while the residual is far below any tolerance
    a, b = np.array([[2.74424609, 0.0], [0.41547863, 2.90166221]]), np.array([1.27274055, 0.0])
    _check_residual(a, b, must_converge=True)


def test_one_way_chains_side_by_side_on_many_ctas():
    import scipy.sparse as sp

    from nangila_spice.gpu import DeviceCsr

    a, b = _one_way_chain(None, 5, gain=5.0, back=1e-8)
    copies = 4000  # 52 000 entries: 25 CTAs
    big = sp.block_diag([sp.csr_matrix(a)] * copies, format="csr")
    x, it, rel, ok = DeviceCsr(big.indptr, big.indices, big.data).solve(np.tile(b, copies), tol=1e-10, max_iter=400)
    assert ok and rel < 1e-10
    rest = np.tile(b, copies) - big @ x
    assert np.linalg.norm(rest) / np.sqrt(copies) <= 1e-10 + 100 * (it + 1) * 2.3e-16 * 5.0 ** 5
