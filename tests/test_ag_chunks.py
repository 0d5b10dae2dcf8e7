"""How the quantizing all-gather cuts a shard into chunks, and the kernel at the sizes where the cut changes."""
import ctypes
from pathlib import Path

import pytest
import torch


def _rule():
    lib = ctypes.CDLL(str(Path(__file__).resolve().parent.parent / "nangila" / "libnangila_kernels.so"))
    lib.nangila_ag_chunk_elems.argtypes = [ctypes.c_int64, ctypes.c_int32]
    return lib.nangila_ag_chunk_elems


def test_chunk_rule_limits():
    rule = _rule()
    for resident in (0, 1, 74, 148, 592):
        for shard in (8, 2048, 16_376, 16_384, 148 * 4096, 148 * 4096 + 8, 3_145_728, 1 << 30, 1 << 34):
            c = rule(shard, resident)
            assert c % 2048 == 0 and 2048 <= c <= 131072
            if shard >= 4 * 4096:
                assert c >= 4096
            chunks = -(-shard // c)
            # whole waves of quantize tasks, each wave short of one by rounding at most
            waves = -(-shard // (max(resident, 1) * 131072))
            assert chunks <= max(resident, 1) * waves or c <= 4096


@pytest.mark.gpu
@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("shard", [8, 2040, 2056, 16_376, 16_384, 296 * 4096 - 8, 296 * 4096 + 8])
def test_gather_at_the_cuts(shard, dtype, bits):
    from nangila.parallel.fsdp_collectives import NangilaAllGather
    from nangila.parallel.symm import LoopbackArena

    dev = torch.device("cuda", 0)
    gen = torch.Generator(device="cuda").manual_seed(shard)
    ins = [(torch.randn(shard, device=dev, generator=gen) * 0.02).to(dtype) for _ in range(2)]
    outs = [torch.full((2 * shard + 8,), 3.0, dtype=dtype, device=dev) for _ in ins]
    ag = NangilaAllGather(arena=LoopbackArena(2, dev), bits=bits)
    for _ in range(3):  # both sets of slots, and one of them again
        ag.gather([o[:2 * shard] for o in outs], ins)
    ag.check_status()
    x = torch.cat(ins).double()
    top = 2 ** (bits - 1) - 1
    amax = torch.cat([torch.nn.functional.pad(i.double().abs(), (0, -shard % 64)).view(-1, 64).amax(1).repeat_interleave(64)[:shard] for i in ins])
    step = amax / top * (1 + 2.0 ** -7)  # the scale is rounded up to bf16
    for o in outs:
        assert (o[2 * shard:] == 3.0).all()
        # half a step, and the rounding of the result to its type
        eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -22
        assert ((o[:2 * shard].double() - x).abs() <= 0.5 * step * (1 + 1e-5) + eps * x.abs() + eps * step).all()
        assert torch.equal(o, outs[0])
