"""The compressed all-reduce of a group of one rank (a kernel of its own) at the sizes where its work is cut: slices of 256
elements, one per warp of the resident grid, and what is left over. Checked through what the format promises, element by
element: value sent + error kept = gradient + error before, codes are whole multiples of the block's scale, and the error
is at most half a step."""
import pytest
import torch

pytestmark = pytest.mark.gpu

GRID = 592 * 8 * 256  # one slice for every warp of 148 SMs x 4 CTAs


def _blocks(x):
    return torch.nn.functional.pad(x, (0, -x.numel() % 64)).view(-1, 64)


@pytest.mark.parametrize("gain", [0.0, 1.0])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("n", [1, 7, 8, 63, 255, 256, 257, 2047, 2049, GRID - 1, GRID, GRID + 8, 3 * GRID + 777])
def test_one_pass_at_the_cuts(n, dtype, gain):
    from nangila.parallel.predres_engine import PredResEngine
    from nangila.parallel.symm import LoopbackArena

    dev = torch.device("cuda", 0)
    gen = torch.Generator(device="cuda").manual_seed(n)
    guard = 64
    eng = PredResEngine(LoopbackArena(1, dev), dev, stochastic=False, use_side_stream=False, adaptive_gain=False)
    eng.fixed_gain = gain
    eng.probe_every = 1 << 30
    base = torch.randn(n, device=dev, generator=gen) * 1e-2
    st = None
    for t in range(4):
        g = (base + torch.randn(n, device=dev, generator=gen) * 1e-3).to(dtype)
        buf = torch.full((n + guard,), 3.0, dtype=dtype, device=dev)
        buf[:n] = g
        before = None
        if t >= 2:  # two exact steps build the history
            before = tuple(v[0].float().clone() for v in (st.ef, st.prev, st.curr))
        st = eng.reduce(0, [buf[:n]], compressed=t >= 2, step=t)
        eng.check_status()
        assert (buf[n:] == 3.0).all()
        if t < 2:
            assert torch.equal(buf[:n], g)
            continue
        ef, prev, curr = before
        sent, kept = buf[:n].float(), st.ef[0].float()
        pred = gain * (curr + 0.9 * (curr - prev))
        x = g.float() + ef - pred
        coded = sent - pred
        # rounding to the types that hold the numbers: of the sum, of the value sent, of the error kept
        eps = 2.0 ** -8 if dtype != torch.float32 else 2.0 ** -21
        slack = eps * (g.float().abs() + ef.abs() + sent.abs() + pred.abs() + kept.abs())
        amax = _blocks(x).abs().amax(1, keepdim=True).expand(-1, 64).reshape(-1)[:n]
        step = amax / 7 * (1 + 2.0 ** -7)                       # the scale is rounded up to bf16
        assert ((coded + kept - x).abs() <= 2 * slack + 1e-30).all()
        assert (kept.abs() <= 0.5 * step * (1 + 2.0 ** -6) + 2 * slack + 1e-30).all()
        if gain:
            assert torch.equal(st.curr[0].float(), buf[:n].to(st.curr[0].dtype).float()) or dtype != torch.float32
            assert ((st.curr[0].float() - sent).abs() <= slack).all()
