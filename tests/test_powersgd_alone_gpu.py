"""PowerSGD for a group of one rank, which exchanges nothing: the exchange kernel on the GEMM's factor in place against the general path
through the region (the same group with the factor at an address that the direct path does not take), the GEMM that leaves unwanted columns alone, and
a bucket of several matrices replayed as one graph."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("orth", [True, False])
@pytest.mark.parametrize("r", [1, 3, 4, 6, 8, 13, 16])
@pytest.mark.parametrize("rows", [16, 1000, 66_000])
def test_direct_and_general_path_agree(rows, r, orth):
    from nangila import _cuda as C
    from nangila.parallel.symm import LoopbackArena

    dev = torch.device("cuda", 0)
    gen = torch.Generator(device="cuda").manual_seed(rows + r)
    room = torch.randn(rows * 16 + 1, device=dev, generator=gen)
    total, recv, flag = C.psgd_exchange_layout(rows, r, 1)
    results = []
    for local in (room[1:].clone(), room):
        factor = local[-rows * 16:].view(rows, 16)  # the second one starts four bytes into its storage
        region = LoopbackArena(1, dev).allocate(int(total))
        mean, scratch = (torch.full((rows, 16), 7.0, device=dev) for _ in range(2))
        t = torch.full((16, rows), 7.0, device=dev, dtype=torch.bfloat16)
        status = torch.zeros(8, dtype=torch.int32, device=dev)
        C.psgd_exchange([factor], [mean], [scratch], [t], [status], region.ptrs, recv, flag, rows, r, 0, orth, 1, 2.0, None, False)
        torch.cuda.synchronize()
        assert int(status[0]) == 0
        results.append((mean, t))
    assert room[1:].data_ptr() % 16 != 0
    assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])


@pytest.mark.parametrize("columns", [1, 4, 5, 16])
@pytest.mark.parametrize("m,n", [(16, 64), (512, 4608), (128, 8192)])
def test_columns_that_are_wanted(m, n, columns):
    from nangila import _cuda as C

    gen = torch.Generator(device="cuda").manual_seed(m + n)
    M = torch.randn(m, n, device="cuda", generator=gen).to(torch.bfloat16)
    Bt = torch.randn(16, n, device="cuda", generator=gen).to(torch.bfloat16)
    out = torch.zeros(m, 16, device="cuda")
    status = torch.zeros(8, dtype=torch.int32, device="cuda")
    C.psgd_gemm(M, Bt, False, out, status, 1.0, False, push_rank=columns)
    want = M.double() @ Bt.double().t()
    # products of 8-bit numbers are exact in FP32; n of them are added, in parts that meet in any order
    bound = n * 2.0 ** -24 * (M.double().abs() @ Bt.double().abs().t())
    assert ((out.double() - want).abs() <= bound)[:, :columns].all() and int(status[0]) == 0


def test_graph_of_a_bucket_and_single_launches_agree(monkeypatch):
    from nangila.parallel.powersgd_engine import PowerSGDEngine
    from nangila.parallel.symm import LoopbackArena

    dev = torch.device("cuda", 0)
    shapes = [(16, 512), (256, 2304), (1024, 24), (512, 4608)]

    class Bucket:
        def __init__(self, views):
            self._views = views

        def gradients(self):
            return self._views

    results = []
    for graph in ("1", "0"):
        monkeypatch.setenv("NANGILA_PSGD_GRAPH", graph)
        gen = torch.Generator(device="cuda").manual_seed(2)
        eng = PowerSGDEngine(LoopbackArena(1, dev), dev, rank=4)
        flat = torch.empty(sum(m * n for m, n in shapes), device=dev)
        views, at = [], 0
        for m, n in shapes:
            views.append(flat[at:at + m * n].view(m, n))
            at += m * n
        outs = []
        for _ in range(4):
            for v in views:
                m, n = v.shape
                v.copy_(torch.randn(m, 2, device=dev, generator=gen) @ torch.randn(2, n, device=dev, generator=gen) * 1e-2)
            eng.reduce(0, Bucket(views), flat)
            outs.append(flat.clone())
        eng.check_status()
        results.append(outs)
    for a, b in zip(*results):
        # the parts of a GEMM's K range meet in any order (FP32), and what follows rounds to bf16
        assert ((a - b).norm() / b.norm()).item() < 2e-2
