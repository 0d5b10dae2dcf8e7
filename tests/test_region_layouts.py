"""Peers write slots and flags into one another's exchange regions, so the layout must not depend on how many CTAs one rank's
device happens to hold. Host logic with a stand-in for the kernels; no GPU."""
import pytest
import torch


class _Arena:
    world, rank = 4, 1

    def allocate(self, nbytes):
        return type("Region", (), {"ptrs": [0] * self.world, "nbytes": nbytes})()


class _Glue:
    """The real layout rules, a device that holds `resident` CTAs, and launches that only note the chunk size."""

    def __init__(self, resident):
        from nangila import _cuda

        self._real, self._resident, self.chunks = _cuda, resident, []

    def __getattr__(self, name):
        return getattr(self._real, name)

    def predres_resident_ctas(self):
        return self._resident

    def ag_launch(self, inputs, outputs, status, ptrs, r, f, rank, chunk, *rest):
        self.chunks.append((r, f, chunk))


SIZES = [2048, 131_072, 3_145_728, 50_000_000]


def _chunks(resident):
    from nangila.parallel.fsdp_collectives import NangilaAllGather

    ag = NangilaAllGather(arena=_Arena())
    ag._glue = _Glue(resident)
    for n in SIZES:
        ag.gather([torch.empty(0)], [torch.empty(n, dtype=torch.bfloat16, device="meta")])
    return ag._glue.chunks


@pytest.mark.parametrize("resident", [592, 148, 4])
def test_all_gather_layout_is_the_same_on_every_device(resident):
    assert _chunks(resident) == _chunks(528)
