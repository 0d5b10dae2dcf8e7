"""NANGILA_FSDP_CTAS: a rank has no more CTAs in any launch of the fully-sharded collectives than the cap says, however many peers there are, and
a cap below the number of peers still reaches all of them."""
import ctypes
from pathlib import Path

import pytest
import torch


def _grid(tiles, groups, cap):
    lib = ctypes.CDLL(str(Path(__file__).resolve().parent.parent / "nangila" / "libnangila_kernels.so"))
    lib.nangila_fsdp_grid.argtypes = [ctypes.c_int64, ctypes.c_int32, ctypes.c_int32, ctypes.POINTER(ctypes.c_uint32), ctypes.POINTER(ctypes.c_uint32)]
    x, y = ctypes.c_uint32(), ctypes.c_uint32()
    capped = lib.nangila_fsdp_grid(tiles, groups, cap, ctypes.byref(x), ctypes.byref(y))
    return x.value, y.value, capped


@pytest.mark.parametrize("groups", [1, 2, 7, 8, 16])
@pytest.mark.parametrize("tiles", [1, 3, 16, 24 * 16, 100_000])
def test_grid(tiles, groups):
    assert _grid(tiles, groups, 0) == (tiles, groups, 0)
    for cap in (1, 3, 4, 24, 32, 148, 592, tiles * groups - 1, tiles * groups, tiles * groups + 1):
        if cap <= 0:
            continue
        x, y, capped = _grid(tiles, groups, cap)
        assert 1 <= x * y <= cap
        assert capped == (0 if cap >= tiles * groups else 1 if cap >= groups else 2) and x <= tiles and y <= groups
        assert capped or (x, y) == (tiles, groups)
        assert x * y > cap // 2 or x == tiles  # most of what is allowed is used


class _Arena:
    world, rank = 8, 1

    def allocate(self, nbytes):
        return type("Region", (), {"ptrs": [0] * self.world, "nbytes": nbytes})()


class _Glue:
    def __init__(self):
        from nangila import _cuda

        self._real, self.caps = _cuda, []

    def __getattr__(self, name):
        return getattr(self._real, name)

    def ag_launch(self, *args):
        self.caps.append(args[-1])

    def rs_launch(self, *args):
        self.caps.append(args[-1])


@pytest.mark.parametrize("cap", [0, 3, 32, 4096])
def test_the_cap_reaches_the_launcher_as_it_is(cap, monkeypatch):
    from nangila.parallel import fsdp_collectives as F

    monkeypatch.setenv("NANGILA_FSDP_CTAS", str(cap))
    monkeypatch.setenv("NANGILA_CHUNK", "131072")  # few chunks
    rs, ag = F.NangilaReduceScatter(arena=_Arena()), F.NangilaAllGather(arena=_Arena())
    rs._glue = ag._glue = glue = _Glue()
    x = torch.zeros(8 * 3 * 131072)
    rs.reduce([torch.zeros(3 * 131072)], [x], 1.0, unit="u")
    ag.gather([x], [torch.zeros(3 * 131072)])
    assert glue.caps == [cap, cap]


@pytest.mark.gpu
@pytest.mark.parametrize("cap", [1, 2, 5, 40])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("shard", [8, 8200, 5 * 8192 - 8])
def test_every_tile_is_reached(shard, dtype, cap):
    """The results are those without a cap, bit for bit."""
    from nangila.parallel import fsdp_collectives as F
    from nangila.parallel.symm import LoopbackArena

    dev, world = torch.device("cuda", 0), 8
    gen = torch.Generator(device="cuda").manual_seed(shard + cap)
    grads = [(torch.randn(world * shard, device=dev, generator=gen) * 0.01).to(dtype) for _ in range(world)]
    results = []
    for ctas in (0, cap):
        rs = F.NangilaReduceScatter(arena=LoopbackArena(world, dev), error_feedback=True)
        ag = F.NangilaAllGather(arena=LoopbackArena(world, dev))
        rs.ctas = ag.ctas = ctas
        shards = [torch.full((shard,), 3.0, dtype=dtype, device=dev) for _ in range(world)]
        full = [torch.full((world * shard,), 3.0, dtype=dtype, device=dev) for _ in range(world)]
        for _ in range(2):
            rs.reduce(shards, grads, 1.0 / world, unit="u")
            ag.gather(full, shards)
        rs.check_status()
        ag.check_status()
        results.append(shards + full + rs._units["u"].ef)
    for a, b in zip(*results):
        assert torch.equal(a, b)
