"""One element of a gradient that is not finite, or nearly as large as BF16 goes: above 3e38 (BF16 makes 3.004e38 of 3e38) it counts as zero, below it survives, and the rest of its warp's 256 elements, which
leave the packed arithmetic for FP32 with it, stay within the quantizer's bound."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda", 0)


def _step(x):
    """One quantization step per element: the largest magnitude of its 64 over 7, rounded up to bf16."""
    return (x.view(-1, 64).abs().amax(1) / 7.0 * (1 + 2.0 ** -7)).repeat_interleave(64)


@pytest.mark.parametrize("bad", [float("nan"), float("inf"), float("-inf"), 3e38, -3e38, 2.9e38, -2.9e38])
@pytest.mark.parametrize("error_memory", [False, True])
def test_values_around_one_that_is_not_ordinary(bad, error_memory):
    from nangila.parallel.fsdp_collectives import NangilaReduceScatter
    from nangila.parallel.symm import LoopbackArena

    shard, at = 8192, 70
    gen = torch.Generator(device="cuda").manual_seed(3)
    ins = [(torch.randn(2 * shard, device=DEV, generator=gen) * 0.01).to(torch.bfloat16) for _ in range(2)]
    ins[0][at] = bad
    rs = NangilaReduceScatter(arena=LoopbackArena(2, DEV), error_feedback=error_memory, stochastic=False)
    outs = [torch.empty(shard, dtype=torch.bfloat16, device=DEV) for _ in range(2)]
    rs.reduce(outs, ins, 0.5, unit="u")
    rs.check_status()
    x = [i.double() for i in ins]
    kept = bool(x[0][at].abs() <= 3e38)
    if not kept:
        x[0][at] = 0.0
    for r in range(2):
        mine = slice(r * shard, (r + 1) * shard)
        want = 0.5 * (x[0][mine] + x[1][mine])
        steps = 0.5 * (_step(x[0][mine]) + _step(x[1][mine]))
        # half a code; 7 * 2^-7 of one for the truncated reciprocal; scale and partial sums in bf16: 2^-9 of up to seven steps each, and the result's rounding
        bound = steps * (0.5 + 7 * 2.0 ** -7 + 7 * 3 * 2.0 ** -9) + 2.0 ** -9 * want.abs() + 1e-7
        assert ((outs[r].double() - want).abs() <= bound).all()
    if kept:
        assert abs(float(outs[0][at]) / (0.5 * bad) - 1.0) < 0.02  # its block's largest: code seven
        assert (outs[0][64:at].abs() < 0.1).all()
    if error_memory:
        left = rs._units["u"].ef[0].double()
        assert torch.isfinite(left).all()
        if not kept:
            assert (left.abs() <= _step(x[0]) * (0.5 + 7 * 2.0 ** -7 + 2.0 ** -6) + 1e-9).all()
