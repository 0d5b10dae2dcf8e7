"""The fully-sharded collectives at the edges of their tiles (2048-element iterations, four to a tile, chunks, shards), under a cap on CTAs,
in place, and when a rank does not come."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda", 0)


def _loopback(world):
    from nangila.parallel.symm import LoopbackArena

    return LoopbackArena(world, DEV)


def _blocks(x):
    return torch.nn.functional.pad(x.double(), (0, -x.numel() % 64)).view(-1, 64)


def _step(x, top):
    """One quantization step per element: the block's largest magnitude / top, rounded up to bf16."""
    n = x.numel()
    return (_blocks(x).abs().amax(1) / top * (1 + 2.0 ** -7)).repeat_interleave(64)[:n]


@pytest.mark.parametrize("ctas", [0, 3])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("shard", [8, 2040, 2056, 8192, 3 * 8192 - 8, 592 * 1024 + 8])
@pytest.mark.parametrize("world,ef", [(1, True), (2, False), (4, True)])
def test_reduce_scatter(world, ef, shard, dtype, ctas):
    from nangila.parallel.fsdp_collectives import NangilaReduceScatter

    gen = torch.Generator(device="cuda").manual_seed(shard + world)
    n = shard * world
    ins = [(torch.randn(n, device=DEV, generator=gen) * 0.01).to(dtype) for _ in range(world)]
    rs = NangilaReduceScatter(_loopback(world), error_feedback=ef, stochastic=False)
    rs.ctas = ctas
    full = [torch.full((shard + 8,), 3.0, dtype=dtype, device=DEV) for _ in range(world)]
    memory = [torch.zeros(n, dtype=torch.float64, device=DEV) for _ in range(world)]
    for _ in range(3):  # both sets of slots, and one of them again
        rs.reduce([f[:shard] for f in full], ins, 1.0 / world, unit="u")
        rs.check_status()
        x = [i.double() + m for i, m in zip(ins, memory)]
        if ef:
            memory = [e.double() for e in rs._units["u"].ef]
        for r in range(world):
            mine = slice(r * shard, (r + 1) * shard)
            steps = sum(_step(v[mine], 7.0) for v in x) / world
            want = sum(v[mine] for v in x) / world
            # a code: half a step, and 7 * 2^-7 of one for the truncated reciprocal; gradient + memory and, in packed bf16, scale and partial
            # sums are rounded to 8 bits: 2^-9 of up to 7 steps each
            eps = 2.0 ** -9 if dtype == torch.bfloat16 else 2.0 ** -11
            bound = steps * (0.5 + 7 * 2.0 ** -7 + 7 * 2.0 ** -9 + 7 * (world + 1) * eps) + eps * want.abs() + 1e-7
            assert ((full[r][:shard].double() - want).abs() <= bound).all()
            assert (full[r][shard:] == 3.0).all()


@pytest.mark.parametrize("bad", [float("nan"), float("inf"), 3e38])
@pytest.mark.parametrize("shard", [8192, 2056])
def test_reduce_scatter_non_finite(shard, bad):
    """A NaN or an infinity counts as zero and leaves all other blocks alone; the largest finite values survive."""
    from nangila.parallel.fsdp_collectives import NangilaReduceScatter

    gen = torch.Generator(device="cuda").manual_seed(3)
    clean = [(torch.randn(2 * shard, device=DEV, generator=gen) * 0.01).to(torch.bfloat16) for _ in range(2)]
    dirty = [c.clone() for c in clean]
    dirty[0][70] = bad
    outs = {}
    for name, ins in (("clean", clean), ("dirty", dirty)):
        rs = NangilaReduceScatter(_loopback(2), stochastic=False)
        outs[name] = [torch.empty(shard, dtype=torch.bfloat16, device=DEV) for _ in range(2)]
        rs.reduce(outs[name], ins, 0.5)
        rs.check_status()
    assert torch.isfinite(outs["dirty"][0].float()).all()
    # the packed and the FP32 arithmetic of the 256 elements of the warp may differ by a code; outside of it nothing changes
    assert torch.equal(outs["dirty"][1], outs["clean"][1]) and torch.equal(outs["dirty"][0][256:], outs["clean"][0][256:])


@pytest.mark.parametrize("ctas", [0, 3])
@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("shard", [8, 2056, 8192, 3 * 8192 - 8])
@pytest.mark.parametrize("world", [1, 3])
def test_all_gather_in_place(world, shard, dtype, bits, ctas):
    """Each rank's shard is its own part of the result buffer, as FSDP passes it."""
    from nangila.parallel.fsdp_collectives import NangilaAllGather

    gen = torch.Generator(device="cuda").manual_seed(shard + bits)
    shards = [(torch.randn(shard, device=DEV, generator=gen) * 0.02).to(dtype) for _ in range(world)]
    shards[0][0] = float("nan")
    apart = [torch.empty(world * shard, dtype=dtype, device=DEV) for _ in range(world)]
    ag = NangilaAllGather(arena=_loopback(world), bits=bits)
    ag.ctas = ctas
    ag.gather(apart, shards)
    outs = [torch.zeros(world * shard, dtype=dtype, device=DEV) for _ in range(world)]
    for r, (o, s) in enumerate(zip(outs, shards)):
        o[r * shard:(r + 1) * shard] = s
    ag.gather(outs, [o[r * shard:(r + 1) * shard] for r, o in enumerate(outs)])
    ag.check_status()
    x = torch.nan_to_num(torch.cat(shards).double(), nan=0.0)
    top = 2 ** (bits - 1) - 1
    step = torch.cat([_step(torch.nan_to_num(s.double(), nan=0.0), top) for s in shards])
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11  # the result's own rounding
    for o, a in zip(outs, apart):
        assert torch.equal(o, outs[0]) and torch.equal(o, a)
        assert ((o.double() - x).abs() <= 0.5 * step * (1 + 1e-5) + eps * (x.abs() + step) + 1e-7).all()


class _OneOfTwo:
    """Arena of a two-rank group in which only rank 0 exists: nobody ever releases rank 1's words."""

    world, rank, provider = 2, 0, "test"

    def __init__(self):
        self._inner = _loopback(2)

    def allocate(self, nbytes):
        return self._inner.allocate(nbytes)


@pytest.mark.parametrize("what", ["reduce_scatter", "all_gather"])
def test_a_rank_that_does_not_come(what):
    from nangila.parallel import fsdp_collectives as F

    x = [torch.randn(8192, device=DEV)]
    if what == "all_gather":
        obj, out = F.NangilaAllGather(arena=_OneOfTwo(), timeout_s=0.2), [torch.full((2 * 8192,), 3.0, device=DEV)]
        obj.gather(out, x)
    else:
        obj, out = F.NangilaReduceScatter(arena=_OneOfTwo(), timeout_s=0.2), [torch.full((4096,), 3.0, device=DEV)]
        obj.reduce(out, x, 0.5)
    with pytest.raises(RuntimeError, match="waiting for rank 1"):
        obj.check_status()
    assert (out[0][-4096:] == 3.0).all()  # nothing was made of data that did not come
    assert torch.ones(4, device=DEV).sum().item() == 4.0
    assert int(obj._status[0][0].item()) == 0  # cleared by the check


@pytest.mark.parametrize("what", ["reduce_scatter", "all_gather"])
def test_a_rank_that_has_failed_before_is_missed(what):
    """A status that nobody has looked at: the rank sends nothing more, and the others find out instead of taking what lies in its slots."""
    from nangila.parallel import fsdp_collectives as F

    x = [torch.randn(8192, device=DEV) for _ in range(2)]
    obj = (F.NangilaAllGather if what == "all_gather" else F.NangilaReduceScatter)(arena=_loopback(2), timeout_s=0.2)
    size = 2 * 8192 if what == "all_gather" else 4096
    outs = [torch.zeros(size, device=DEV) for _ in range(2)]
    call = (lambda: obj.gather(outs, x)) if what == "all_gather" else (lambda: obj.reduce(outs, x, 0.5))
    call()
    obj.check_status()
    obj._status[1][0] = 3
    for o in outs:
        o.fill_(3.0)
    call()
    with pytest.raises(RuntimeError, match="waiting for rank 1"):
        obj.check_status()
    assert (outs[0][-4096:] == 3.0).all()
    obj._status[1].zero_()
    call()
    obj.check_status()
    assert not (outs[0] == 3.0).any()


class _Rank:
    """One rank of a group of two whose regions are shared with the other's object."""

    world, provider = 2, "test"

    def __init__(self, rank, region):
        self.rank, self._region = rank, region

    def allocate(self, nbytes):
        if not self._region:
            self._region.append(_loopback(2).allocate(nbytes))
        return self._region[0]


@pytest.mark.parametrize("what", ["reduce_scatter", "all_gather"])
def test_ranks_of_a_group_meet(what):
    """Rank 1 first (rank 0's word is put there by hand, so that it has nothing to wait for), then rank 0, which finds rank 1's codes and word: the same
    bits as with both ranks in one launch. Three launches of both parities."""
    from nangila.parallel import fsdp_collectives as F

    cls = F.NangilaAllGather if what == "all_gather" else F.NangilaReduceScatter
    shard = 3 * 8192 - 8
    gen = torch.Generator(device="cuda").manual_seed(4)
    region = []
    ranks = [cls(arena=_Rank(r, region), timeout_s=0.5, **({} if what == "all_gather" else {"stochastic": False})) for r in range(2)]
    both = cls(arena=_loopback(2), **({} if what == "all_gather" else {"stochastic": False}))
    size = 2 * shard if what == "all_gather" else shard
    for epoch in (1, 2, 3):
        ins = [(torch.randn(shard if what == "all_gather" else 2 * shard, device=DEV, generator=gen) * 0.02).to(torch.bfloat16) for _ in range(2)]
        want = [torch.empty(size, dtype=torch.bfloat16, device=DEV) for _ in range(2)]
        got = [torch.empty(size, dtype=torch.bfloat16, device=DEV) for _ in range(2)]
        call = (lambda o, w, x: o.gather(w, x)) if what == "all_gather" else (lambda o, w, x: o.reduce(w, x, 0.5))
        call(both, want, ins)
        if epoch == 1:  # the regions exist from the first call on: let rank 1's wait for the word run out once
            call(ranks[1], [got[1]], [ins[1]])
            with pytest.raises(RuntimeError, match="waiting for rank 0"):
                ranks[1].check_status()
        else:
            st = next(iter(ranks[1]._regions.values()))
            at = st["f"] if what == "all_gather" else st["f1"]
            region[0].segment._keepalive[1][at:at + 4].view(torch.int32)[0] = epoch
            call(ranks[1], [got[1]], [ins[1]])
            ranks[1].check_status()
        call(ranks[0], [got[0]], [ins[0]])
        ranks[0].check_status()
        assert torch.equal(got[0], want[0])
