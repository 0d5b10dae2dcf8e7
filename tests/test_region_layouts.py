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

    def rs_launch(self, inputs, outputs, ef, status, ptrs, r, f, nchunks, rank, chunk, *rest):
        self.chunks.append((r, f, nchunks, chunk))


SIZES = [2048, 131_072, 3_145_728, 50_000_000]


def _chunks(what, resident):
    from nangila.parallel import fsdp_collectives as F
    from nangila.parallel.predres_engine import PredResEngine

    glue = _Glue(resident)
    if what == "bucket":
        eng = PredResEngine(_Arena(), torch.device("meta"), use_side_stream=False)
        eng._glue = glue
        return [(st.layout, st.chunk) for i, n in enumerate(SIZES) for st in [eng.bucket_state(i, [torch.empty(n, dtype=torch.bfloat16, device="meta")])]]
    obj = (F.NangilaAllGather if what == "all_gather" else F.NangilaReduceScatter)(arena=_Arena())
    obj._glue = glue
    for n in SIZES:
        x = [torch.empty(n, dtype=torch.bfloat16, device="meta")]
        if what == "all_gather":
            obj.gather([torch.empty(0)], x)
        else:
            obj.reduce([torch.empty(0)], x, 0.25, unit=n)
    return glue.chunks


@pytest.mark.parametrize("what", ["all_gather", "reduce_scatter", "bucket"])
@pytest.mark.parametrize("resident", [592, 148, 4])
def test_layout_is_the_same_on_every_device(what, resident):
    assert _chunks(what, resident) == _chunks(what, 528)
