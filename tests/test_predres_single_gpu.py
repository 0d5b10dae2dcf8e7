"""The compressed all-reduce of a group of one rank (a kernel of its own) at the sizes where its work is cut: tiles of 2048
elements, CTAs of two tiles without statistics and of one to eight with them, the end of the last whole chunk (from where
packed-bf16 arithmetic gives way to FP32), and fewer CTAs than the bucket needs. Checked through what the format promises, element by
element: value sent + error kept = gradient + error before, codes are whole multiples of the block's scale, and the error
is at most half a step."""
import pytest
import torch

pytestmark = pytest.mark.gpu

TILE = 2048
CHUNK = 4096              # chunk size of buckets up to 592 x 4096 elements; beyond, a multiple of it
GRID = 592 * TILE         # a tile for each of four CTAs on 148 SMs
WAVE = 1600 * TILE        # with statistics a CTA takes one tile more for each of these


def _blocks(x):
    return torch.nn.functional.pad(x, (0, -x.numel() % 64)).view(-1, 64)


def _engine(gain, **kw):
    from nangila.parallel.predres_engine import PredResEngine
    from nangila.parallel.symm import LoopbackArena

    dev = torch.device("cuda", 0)
    eng = PredResEngine(LoopbackArena(1, dev), dev, stochastic=False, use_side_stream=False, adaptive_gain=False, **kw)
    eng.fixed_gain = gain
    eng.probe_every = 1 << 30
    return eng


@pytest.mark.parametrize("gain", [0.0, 1.0])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("n", [1, 7, 8, 63, 255, 256, 257, 2047, 2048, 2049, 4095, 4096, 4097, 3 * CHUNK - 8, 3 * CHUNK + 8, GRID - 1, GRID, GRID + 8,
                               592 * CHUNK + 8, 3 * GRID + 777, 2 * WAVE - 8, 2 * WAVE + 3])
def test_one_pass_at_the_cuts(n, dtype, gain):
    _one_pass(n, dtype, gain)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n", [3 * WAVE + TILE + 5, 8 * WAVE - TILE, 8 * WAVE + TILE + 777])
def test_several_tiles_per_cta(n, dtype):
    _one_pass(n, dtype, 1.0)


def _one_pass(n, dtype, gain):
    dev = torch.device("cuda", 0)
    gen = torch.Generator(device="cuda").manual_seed(n)
    guard = 64
    eng = _engine(gain)
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
        if dtype == torch.float16:
            slack += 2.0 ** -25  # numbers below 2^-14 lie 2^-24 apart there: rounding one is half of that, however small it is
        amax = _blocks(x).abs().amax(1, keepdim=True).expand(-1, 64).reshape(-1)[:n]
        step = amax / 7 * (1 + 2.0 ** -7)                       # the scale is rounded up to bf16
        assert ((coded + kept - x).abs() <= 2 * slack + 1e-30).all()
        assert (kept.abs() <= 0.5 * step * (1 + 2.0 ** -6) + 2 * slack + 1e-30).all()
        if gain:
            assert torch.equal(st.curr[0].float(), buf[:n].to(st.curr[0].dtype).float()) or dtype != torch.float32
            assert ((st.curr[0].float() - sent).abs() <= slack).all()


@pytest.mark.parametrize("gain", [0.0, 1.0])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n", [5 * CHUNK + 1, 40 * CHUNK, 2 * WAVE + 3])
def test_capped_ctas_go_round_again_with_the_same_bits(n, dtype, gain):
    gen = torch.Generator(device="cuda").manual_seed(n)
    grads = [(torch.randn(n, device="cuda", generator=gen) * 1e-2).to(dtype) for _ in range(4)]
    results = []
    for ctas in (0, 3):
        eng = _engine(gain, ctas=ctas)
        for t, g in enumerate(grads):
            buf = g.clone()
            st = eng.reduce(0, [buf], compressed=t >= 2, step=t)
        eng.check_status()
        results.append((buf, st.ef[0], st.prev[0], st.curr[0]))
    assert all(torch.equal(a, b) for a, b in zip(*results))


@pytest.mark.parametrize("ctas", [0, 3])
@pytest.mark.parametrize("gain", [0.0, 1.0])
@pytest.mark.parametrize("n", [777, 5 * CHUNK + 1, 2 * WAVE + 3, 8 * WAVE + TILE + 777])
def test_statistics_match_64_bits(n, gain, ctas):
    """The five sums the gain controller reads: residual, gradient, <gradient + error, prediction>, prediction, error kept."""
    gen = torch.Generator(device="cuda").manual_seed(n)
    eng = _engine(gain, ctas=ctas)
    base = torch.randn(n, device="cuda", generator=gen) * 1e-2
    for t in range(4):
        g = base + torch.randn(n, device="cuda", generator=gen) * 1e-3
        if t == 3:  # (without a gain only a probe keeps them)
            eng.probe_every = st.probe_every = st.next_probe = 1
            ef, prev, curr = (v[0].double() for v in (st.ef, st.prev, st.curr))
            st.stats[0].zero_()
        st = eng.reduce(0, [g.clone()], compressed=t >= 2, step=t)
    eng.check_status()
    x = g.double() + ef
    pred = curr + eng.momentum * (curr - prev)
    terms = [(x - gain * pred) ** 2, g.double() ** 2, x * pred, pred ** 2, st.ef[0].double() ** 2]
    got = st.stats[0][:5].double()
    # FP32 sums: 64 values a thread and round, a tree of eight levels, then one addition per CTA; and a few roundings per term
    adds = (64 if ctas == 0 else -(-n // (3 * 256))) + 8 + min(-(-n // TILE), 3200) + 8
    for k, term in enumerate(terms):
        assert abs(float(got[k] - term.sum())) <= adds * 2.0 ** -24 * float(term.abs().sum()) + 1e-30, k
