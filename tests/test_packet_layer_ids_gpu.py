"""decompress_gpu takes any number that equals the packet's layer, and refuses all others with the same error, whether it knows the layer or not."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

N = 3000


def _hook_and_packet(layer):
    import nangila

    hook = nangila.NangilaHook.all_drivers(2, nangila.NangilaConfig(warmup_steps=0, shadow_run_steps=0))
    hook.step()
    gen = torch.Generator(device="cuda").manual_seed(1)
    grad = torch.randn(N, device="cuda", generator=gen) * 0.02
    for layer_id in (layer, 1):
        hook.update_gpu(layer_id, grad)
        hook.update_gpu(layer_id, grad * 1.01)
    return hook, hook.compress_gpu(1, grad, sync_mode=0)


@pytest.mark.parametrize("same", [1.0, True, np.int32(1), np.float64(1.0)])
def test_equal_ids(same):
    hook, packet = _hook_and_packet(1)
    assert torch.equal(hook.decompress_gpu(same, packet, N), hook.decompress_gpu(1, packet, N))


@pytest.mark.parametrize("other", [0, -1, 1.5, 1 << 32, (1 << 32) + 1, 1 << 70])
def test_other_ids_that_have_a_history(other):
    hook, packet = _hook_and_packet(other)
    with pytest.raises(RuntimeError, match="packet is for layer 1"):
        hook.decompress_gpu(other, packet, N)
