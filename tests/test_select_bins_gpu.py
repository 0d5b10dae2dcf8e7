"""The bin search shared by the selections, through the exact order statistic that is made of three of them: every kind of rank, ties, one
value alone, whatever the alignment of the scratch words."""
import ctypes
import os

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 1, 2, 3])
@pytest.mark.parametrize("n", [1, 255, 1024, 70_001])
@pytest.mark.parametrize("kind", ["normal", "wide", "ties", "equal"])
def test_order_statistic(kind, n, offset):
    lib = ctypes.CDLL(os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nangila", "libnangila_kernels.so"))
    lib.nangila_absmax_hist.argtypes = [ctypes.c_void_p, ctypes.c_int32, ctypes.c_int64, ctypes.c_uint32, ctypes.c_float, ctypes.c_void_p,
                                        ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p]
    gen = torch.Generator(device="cuda").manual_seed(n + offset)
    x = torch.randn(n, device="cuda", generator=gen)
    if kind == "wide":
        x = torch.exp(15 * x)  # 26 decades, all finite
    elif kind == "ties":
        x = torch.round(x)
    elif kind == "equal":
        x = torch.full_like(x, -2.5)
    words = lib.nangila_absmax_scratch_words()
    scratch = torch.full((words + 8,), -1, dtype=torch.int32, device="cuda")
    out = torch.zeros(4, device="cuda")
    ordered = x.abs().sort(descending=True).values
    for k in sorted(k for k in {1, 2, n // 3, n // 2, n - 1, n} if 1 <= k <= n):
        rc = lib.nangila_absmax_hist(x.data_ptr(), 0, n, k, 7.0, scratch[offset:].data_ptr(), out.data_ptr(), None, torch.cuda.current_stream().cuda_stream)
        assert rc == 0
        assert out[1].item() == ordered[k - 1].item() and out[0].item() == ordered[0].item()
    assert (scratch[:offset] == -1).all() and (scratch[offset + words:] == -1).all()
