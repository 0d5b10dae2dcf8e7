"""The thread-per-row product fetches ahead from where a CTA's rows would lie if all were of the same length: nothing up to 40 MB of matrix and vectors, the
columns up to 126 MiB, all of it beyond. Rows that lie elsewhere, CTAs without entries, an odd number of rows, vectors that start off a 16-byte line."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [700_001, 1_300_001, 3_300_001])  # 31, 59 and 145 MB and more
@pytest.mark.parametrize("where", ["even", "first", "last"])
@pytest.mark.parametrize("offset", [0, 1])
def test_product(where, n, offset):
    from nangila_spice.gpu import DeviceCsr

    rng = np.random.default_rng(n)
    lengths = np.zeros(n, dtype=np.int64)
    if where == "even":
        lengths[:] = 3
    elif where == "first":
        lengths[:n // 8] = 16
    else:
        lengths[-(n // 8):] = 16
    row_ptr = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    rows = np.repeat(np.arange(n), lengths)
    col = np.clip(rows + rng.integers(-40, 41, rows.size), 0, n - 1).astype(np.int32)
    val = rng.standard_normal(col.size)
    m = DeviceCsr(row_ptr, col, val)
    x = torch.empty(n + 1, dtype=torch.float64, device="cuda")[offset:offset + n]
    y = torch.full((n + 1,), 3.0, dtype=torch.float64, device="cuda")
    host = rng.standard_normal(n)
    x.copy_(torch.from_numpy(host))
    m.matvec_device(x, y[offset:offset + n], torch.cuda.current_stream().cuda_stream)
    got = y.cpu().numpy()
    assert got[n if offset == 0 else 0] == 3.0
    got = got[offset:offset + n]
    products = val * host[col]
    want = np.bincount(rows, products, minlength=n)
    size = np.bincount(rows, np.abs(products), minlength=n)
    assert (np.abs(got - want) <= 2.3e-16 * 2 * (lengths + 1) * size).all()  # one rounding per product and per sum, on either side
