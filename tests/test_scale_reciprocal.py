"""The packed-bf16 quantizer multiplies by 1 / scale truncated to bf16. Scales that are powers of two (largest magnitude 7 2^k) are where an approximate
reciprocal could fall short of the bf16 number that 1 / scale is: the codes would be off at ties, and the factor by 2^-8."""
import numpy as np
import pytest
import torch


def _bits(x):
    return np.asarray(x, dtype=np.float32).view(np.uint32)


def _live_scales():
    """All bf16 numbers above 1e-30 that a block's scale can be (largest finite magnitude / 7, rounded up)."""
    s = (np.arange(0x7F80, dtype=np.uint32) << 16).view(np.float32)
    return s[(s > 1e-30) & (s <= np.float32(3.4e38) / 6.9)]


def test_truncated_reciprocal_whatever_the_approximation_returns():
    s = _live_scales()
    exact = 1.0 / s.astype(np.float64)
    up = np.nextafter(exact.astype(np.float32), np.float32(np.inf))
    near = np.where(exact.astype(np.float32).astype(np.float64) > exact, exact.astype(np.float32), up)  # the float above, or next above
    below = np.where(near.astype(np.float64) > exact, np.nextafter(near, np.float32(0)), near)           # the largest float not above 1 / s
    assert (below.astype(np.float64) <= exact).all()
    want = _bits(below) >> 16
    ulp = np.spacing(below).astype(np.float64)
    short = 0
    for off in range(-3, 4):  # every float within one ulp of 1 / s
        got = (_bits(below).astype(np.int64) + off).astype(np.uint32)
        allowed = np.abs(got.view(np.float32).astype(np.float64) - exact) <= ulp
        assert (((got + 2) >> 16) == want)[allowed].all()
        short += int((((got >> 16) != want) & allowed).sum())
    assert short > 0  # without the two floats added some of them would fall short
    power = (_bits(s) & 0x7FFFFF) == 0
    assert (want[power] << 16 == _bits(exact[power].astype(np.float32))).all()


def test_scale_of_seven_is_a_power_of_two():
    for e in range(-60, 60):
        assert np.float32(7.0 * 2.0 ** e) * np.float32(0.14285715) == np.float32(2.0 ** e)


def _bf16(x):
    return torch.from_numpy(np.asarray(x, dtype=np.float64)).to(torch.bfloat16).double().numpy()


@pytest.mark.gpu
@pytest.mark.parametrize("error_memory", [False, True])
def test_codes_of_blocks_whose_scale_is_a_power_of_two(error_memory):
    """One rank's reduce-scatter hands out q * scale. Blocks with a largest magnitude of 7 2^k and values at and beside the ties (x.5 steps)."""
    from nangila.parallel.fsdp_collectives import NangilaReduceScatter
    from nangila.parallel.symm import LoopbackArena

    dev = torch.device("cuda", 0)
    exps = list(range(-100, -2))  # (largest magnitude below 2: the packed path)
    n = 8192 * ((64 * len(exps) + 8191) // 8192)
    rng = np.random.RandomState(5)
    steps = np.concatenate([np.arange(-7, 7.01, 0.25), rng.uniform(-7, 7, 64 - 57)])
    x = np.zeros(n)
    for i, e in enumerate(exps):
        block = _bf16(rng.permutation(steps) * 2.0 ** e)
        x[64 * i:64 * i + 64] = block
    g = torch.from_numpy(x).to(torch.bfloat16).to(dev)
    out = torch.empty(n, dtype=torch.bfloat16, device=dev)
    rs = NangilaReduceScatter(arena=LoopbackArena(1, dev), error_feedback=error_memory, stochastic=False)
    rs.reduce([out], [g], 1.0, unit="u")
    rs.check_status()
    got = out.double().cpu().numpy()
    for i, e in enumerate(exps):
        b = slice(64 * i, 64 * i + 64)
        q = np.rint(_bf16(192.0 + x[b] * 2.0 ** -e) - 192.0)  # the multiply-add is rounded once, to even, where bf16 has unit spacing
        q = q if 2.0 ** e > 1e-30 else 0.0 * q  # a block with a scale below that is sent as zeros
        assert np.array_equal(got[b], q * 2.0 ** e), e
        if error_memory:
            assert np.array_equal(rs._units["u"].ef[0].double().cpu().numpy()[b], _bf16(x[b] - q * 2.0 ** e)), e
