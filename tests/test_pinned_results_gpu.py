"""Results that the device writes into pinned host memory: the block is not given back while a write to it may still be on its way, and a call
that is refused has queued nothing."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda", 0)


def _packet(n):
    from nangila import _cuda as C

    return C.packet_compress(torch.randn(n, device=DEV), None, None, None, 0.9, 0.0, bytes(32))


@pytest.mark.parametrize("what", ["out's type", "out on the host", "curr's type", "curr's size", "curr on the host", "curr with gaps", "prev's size", "no prev"])
def test_a_refused_inspection_has_queued_nothing(what):
    from nangila import _cuda as C

    n = 5000
    packet, out, curr, prev = _packet(n), torch.empty(n, device=DEV), torch.zeros(n, device=DEV), torch.zeros(n, device=DEV)
    if what == "out's type":
        out = out.half()
    elif what == "out on the host":
        out = out.cpu()
    elif what == "curr's type":
        curr = curr.double()
    elif what == "curr's size":
        curr = torch.zeros(n - 1, device=DEV)
    elif what == "curr on the host":
        curr = curr.cpu()
    elif what == "curr with gaps":
        curr = torch.zeros(2 * n, device=DEV)[::2]
    elif what == "prev's size":
        prev = torch.zeros(n - 1, device=DEV)
    else:
        prev = None
    torch.cuda.synchronize()
    before = torch.cuda.memory_stats()["allocation.all.allocated"]
    with pytest.raises(RuntimeError):
        C.packet_inspect(packet, True, 0, curr, prev, 0.9, out)
    assert torch.cuda.memory_stats()["allocation.all.allocated"] == before  # not even the checksum's word
    assert torch.cuda.current_stream().query()


def test_sums_that_nobody_asks_for_are_waited_for():
    from nangila import _cuda as C

    layers = [torch.ones(4096, device=DEV), torch.full((100,), 2.0, device=DEV)]
    assert C.PendingSums(layers).result() == [4096.0, 400.0]  # (the first use of a kernel and of pinned memory waits for the device)
    torch.cuda.synchronize()
    torch.cuda._sleep(100_000_000)  # some 50 ms
    pending = C.PendingSums(layers)
    assert not torch.cuda.current_stream().query()
    del pending
    assert torch.cuda.current_stream().query()
