"""The calibration kernels where their work is cut: tiles of 1024 elements, odd lengths (the five state vectors of a pair are
then unaligned), gradients at odd addresses, pairs of different sizes in one step, more pairs than one launch carries."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("sizes", [[1], [3, 255], [256, 1023], [1024, 1025], [4099, 7], [16_384 * 40 + 1]])
def test_step_statistics_match_64_bits(sizes, dtype):
    from nangila import _cuda as C

    gen = torch.Generator(device="cuda").manual_seed(sum(sizes))
    steps = 3
    data = [[torch.randn(n + 1, device="cuda", generator=gen).to(dtype)[i % 2:][:n] for n in sizes for i in range(2)] for _ in range(steps)]
    state = [torch.zeros(5 * n, device="cuda") for n in sizes]
    for t, layers in enumerate(data):
        norms = C.sculptor_layer_sumsq(layers)
        want = torch.stack([(x.double() ** 2).sum() for x in layers])
        assert ((norms - want).abs() <= 1e-13 * want * 64).all()  # FP64 sums in another order
        C.sculptor_pair_update(layers[0::2], layers[1::2], state, [t + 1] * len(sizes))
    for p, n in enumerate(sizes):
        x = torch.stack([d[2 * p] for d in data]).double()
        y = torch.stack([d[2 * p + 1] for d in data]).double()
        mx, my = x.mean(0), y.mean(0)
        want = torch.cat([mx, my, ((x - mx) ** 2).sum(0), ((y - my) ** 2).sum(0), ((x - mx) * (y - my)).sum(0)])
        size = torch.cat([x.abs().amax(0), y.abs().amax(0), (x ** 2).amax(0), (y ** 2).amax(0), (x.abs() * y.abs().amax(0)).amax(0)])
        # a handful of FP32 operations per step on numbers of this size
        assert ((state[p].double() - want).abs() <= steps * 16 * 2.0 ** -24 * (size + 1e-30)).all()


def test_more_pairs_than_one_launch_carries():
    from nangila.ops import DeviceSculptor

    n = 777
    ds = DeviceSculptor()
    gen = torch.Generator(device="cuda").manual_seed(5)
    seen = []
    for _ in range(2):
        layers = [torch.randn(n, device="cuda", generator=gen) for _ in range(13)]  # 78 pairs
        seen.append(layers)
        for i, x in enumerate(layers):
            ds.record(i, x)
        ds.end_step()
    assert len(ds._pair_state) == 78
    for (i, j), st in ds._pair_state.items():
        a, b = (seen[0][i] + seen[1][i]) / 2, (seen[0][j] + seen[1][j]) / 2
        assert torch.allclose(st[:n], a, atol=1e-5) and torch.allclose(st[n:2 * n], b, atol=1e-5)
