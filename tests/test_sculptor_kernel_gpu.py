"""The calibration kernels where their work is cut: tiles of 1024 elements, odd lengths (the five state vectors of a pair are
then unaligned), gradients at odd addresses, pairs of different sizes in one step, more pairs than one launch carries."""
import ctypes
import os

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


@pytest.mark.parametrize("max_numel", [1, 1024, 5000, 70_001, 1 << 30])
def test_descriptors_in_device_memory_whatever_the_grid_is_sized_for(max_numel):
    """The C entries take descriptors in device memory and a size for the grid, which may be less than a pair's."""
    lib = ctypes.CDLL(os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nangila", "libnangila_kernels.so"))

    class Pair(ctypes.Structure):
        _fields_ = [("i", ctypes.c_void_p), ("j", ctypes.c_void_p), ("state", ctypes.c_void_p), ("numel", ctypes.c_int64),
                    ("dtype", ctypes.c_int32), ("count", ctypes.c_int32)]

    class Layer(ctypes.Structure):
        _fields_ = [("data", ctypes.c_void_p), ("numel", ctypes.c_int64), ("dtype", ctypes.c_int32), ("reserved", ctypes.c_int32)]

    lib.nangila_sculptor_pair_update.argtypes = [ctypes.c_void_p, ctypes.c_int32, ctypes.c_int64, ctypes.c_void_p]
    lib.nangila_sculptor_layer_sumsq.argtypes = [ctypes.c_void_p, ctypes.c_int32, ctypes.c_int64, ctypes.c_void_p, ctypes.c_void_p]
    gen = torch.Generator(device="cuda").manual_seed(2)
    sizes = [70_001, 333]
    x = [torch.randn(n, device="cuda", generator=gen) for n in sizes for _ in range(2)]
    state = [torch.zeros(5 * n, device="cuda") for n in sizes]
    to_device = lambda d: torch.frombuffer(bytearray(bytes(d)), dtype=torch.uint8).cuda()  # noqa: E731
    pairs = to_device((Pair * 2)(*[Pair(x[2 * p].data_ptr(), x[2 * p + 1].data_ptr(), state[p].data_ptr(), n, 0, 1) for p, n in enumerate(sizes)]))
    layers = to_device((Layer * 4)(*[Layer(t.data_ptr(), t.numel(), 0, 0) for t in x]))
    out = torch.zeros(4, dtype=torch.float64, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    assert lib.nangila_sculptor_pair_update(pairs.data_ptr(), 2, max_numel, st) == 0
    assert lib.nangila_sculptor_layer_sumsq(layers.data_ptr(), 4, max_numel, out.data_ptr(), st) == 0
    for p, n in enumerate(sizes):
        # the first observation: means are the values, everything else is zero
        assert torch.equal(state[p], torch.cat([x[2 * p], x[2 * p + 1], torch.zeros(3 * n, device="cuda")]))
    want = torch.stack([(t.double() ** 2).sum() for t in x])
    assert ((out - want).abs() <= 1e-12 * want).all()
