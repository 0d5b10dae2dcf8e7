"""decompress_gpu queues the decoder of a layer it knows before the host has seen the packet: the result is the one of a decoder that is queued
afterwards, whatever the packet says, at the edges of the tiles, with and without a history."""
import struct

import pytest
import torch

pytestmark = pytest.mark.gpu


def _hook(n, history, dtype=torch.float32):
    import nangila

    hook = nangila.NangilaHook.all_drivers(2, nangila.NangilaConfig(warmup_steps=0, shadow_run_steps=0))
    hook.step()
    gen = torch.Generator(device="cuda").manual_seed(n)
    base = torch.randn(n, device="cuda", generator=gen) * 0.02
    for t in range(2 if history else 0):
        hook.update_gpu(1, base + 1e-3 * t * torch.randn(n, device="cuda", generator=gen))
    grad = (base + 1e-3 * torch.randn(n, device="cuda", generator=gen)).to(dtype)
    return hook, grad, hook.compress_gpu(1, grad, sync_mode=0)


def _after(hook, packet, n, predict, ndim=1):
    """The decoder on its own."""
    from nangila import _cuda as C

    prev, curr = hook.gpu_history(1)
    out = torch.empty(n, device="cuda")
    C.packet_decode(packet[32:], ndim, curr if predict else None, prev if predict else None, float(hook.momentum()), -1.0 if predict else 0.0, out)
    return out


def _sealed(packet):
    from nangila import _cuda as C

    packet = packet.clone()
    packet[12:16] = C.crc32(packet[32:]).view(torch.uint8)[:4]
    return packet


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("history", [False, True])
@pytest.mark.parametrize("n", [1, 7, 64, 2047, 2049, 1184 * 2048 + 5])
def test_result_is_the_decoders(n, history, dtype):
    hook, grad, packet = _hook(n, history, dtype)
    for mode in (0, 1):
        out = hook.decompress_gpu(1, packet, n, sync_mode=mode)
        assert torch.equal(out, _after(hook, packet, n, history))
    # the scale of a block is its largest residual over 7, so no element is off by more than the largest gradient over 14, and rounding
    assert (out - grad.float()).abs().max() <= grad.float().abs().max() * (1 / 14 + 1e-2)
    fresh, _, _ = _hook(n, False)  # a layer that is not known yet
    fresh._gpu["layers"].clear()
    assert torch.equal(fresh.decompress_gpu(1, packet, n), _after(hook, packet, n, False))


def test_packets_that_are_not_what_was_expected():
    n = 5000
    hook, _, packet = _hook(n, True)
    plain = _after(hook, packet, n, False)
    without = packet.clone()
    without[3] |= 0x80  # made without a prediction
    assert torch.equal(hook.decompress_gpu(1, without, n), plain)
    # two dimensions: one word more in front of the gain
    raw = bytes(packet.cpu().numpy())
    two = raw[:32] + raw[32:40] + struct.pack("<III", 2, 50, 100) + raw[48:]
    two = _sealed(torch.frombuffer(bytearray(two), dtype=torch.uint8).cuda())
    assert torch.equal(hook.decompress_gpu(1, two, n), _after(hook, packet, n, True))
    for at, value, message in ((0, 0, "not a nangila packet"), (2, 9, "not a nangila packet"), (8, 0, "layer 0"), (300, 0x5A, "checksum")):
        bad = packet.clone()
        bad[at] = value
        with pytest.raises(RuntimeError, match=message):
            hook.decompress_gpu(1, bad, n)
    for at, message in ((36, "elements"), (35, "block-64")):
        bad = packet.clone()
        bad[at] ^= 0x01
        with pytest.raises(RuntimeError, match=message):
            hook.decompress_gpu(1, _sealed(bad), n)
    with pytest.raises(RuntimeError):
        hook.decompress_gpu(1, packet[:200].clone(), n, sync_mode=0)  # too short for what its header promises
    with pytest.raises(RuntimeError, match="elements"):
        hook.decompress_gpu(1, packet, n - 1)
    assert torch.equal(hook.decompress_gpu(1, packet, n), _after(hook, packet, n, True))  # and the layer is as it was
