"""The factor exchange of PowerSGD on its own, where its variants change: ranks up to 4, 8 and 16, factors that stay in
shared memory and taller ones, rank-deficient factors, several emulated ranks. Checked through what it promises: the
mean, an orthonormal basis of the mean's columns, its bf16 transpose, zero columns beyond the rank."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(local, r, orth):
    from nangila import _cuda as C
    from nangila.parallel.symm import LoopbackArena

    world, rows = len(local), local[0].shape[0]
    dev = local[0].device
    total, recv, flag = C.psgd_exchange_layout(rows, r, world)
    region = LoopbackArena(world, dev).allocate(int(total))
    mean = [torch.full((rows, 16), 7.0, device=dev) for _ in range(world)]
    scratch = [torch.full((rows, 16), 7.0, device=dev) for _ in range(world)]
    t = [torch.full((16, rows), 7.0, device=dev, dtype=torch.bfloat16) for _ in range(world)]
    status = [torch.zeros(8, dtype=torch.int32, device=dev) for _ in range(world)]
    C.psgd_exchange(local, mean, scratch, t, status, region.ptrs, recv, flag, rows, r, 0, orth, 1, 2.0, None, False)
    torch.cuda.synchronize()
    assert all(int(s[0]) == 0 for s in status)
    return [m.view(16, rows) for m in mean], t


@pytest.mark.parametrize("world", [1, 3])
@pytest.mark.parametrize("r", [1, 3, 4, 5, 8, 9, 16])
@pytest.mark.parametrize("rows", [16, 200, 4608, 66_000])
@pytest.mark.parametrize("orth", [True, False])
def test_mean_and_orthonormal_basis(world, r, rows, orth):
    gen = torch.Generator(device="cuda").manual_seed(rows + r)
    local = [torch.randn(rows, 16, device="cuda", generator=gen) * torch.logspace(0, -2, 16, device="cuda") for _ in range(world)]
    mean, t = _run(local, r, orth)
    want = torch.stack([x.double() for x in local]).mean(0)[:, :r].t()
    basis = torch.linalg.qr(want.t())[0].t()
    for m, tt in zip(mean, t):
        assert torch.equal(m, mean[0]) and torch.equal(tt, t[0])  # identical bits on every rank
        assert not m[r:].any() and not tt[r:].any()
        q = tt[:r].double()
        if orth:
            got = m[:r].double()
            # two rounds of Cholesky-QR in FP32 on a basis of condition 100: orthonormal to rounding (sums over the rows)
            assert (got @ got.t() - torch.eye(r, device="cuda", dtype=torch.float64)).abs().max() < 1e-5
            assert (got - basis * torch.sign((got * basis).sum(1, keepdim=True))).norm() < 1e-3 * r ** 0.5
            assert (q - got).abs().max() <= 2.0 ** -8 * got.abs().max()  # rounding to bf16
        else:
            assert (m[:r].double() - want).abs().max() <= 4 * 2.0 ** -24 * sum(x.abs().max() for x in local)
            sign = torch.sign((q * basis).sum(1, keepdim=True))
            assert (q - basis * sign).norm() < (2.0 ** -8 + 1e-3) * r ** 0.5


def test_dependent_columns_become_zero():
    rows = 640
    x = torch.randn(rows, 16, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
    x[:, 2] = 2.0 * x[:, 0] - x[:, 1]
    x[:, 3] = 0.0
    (m,), _ = _run([x], 6, True)
    norms = m[:6].norm(dim=1)
    assert norms[[0, 1, 4, 5]].sub(1.0).abs().max() < 1e-5 and norms[3] == 0.0
    # the dependent column's pivot is rounding: either it counted as gone, or what is left of it is orthonormal to the others
    assert norms[2] == 0.0 or (m[2] @ m[[0, 1, 4, 5]].t()).abs().max() < 1e-4
