"""Where the ranks of a fully-sharded collective meet depends on how many CTAs read (csrc/comm/meet.cuh): in the kernel that reads up to 296, in a kernel in
between beyond; nowhere for up to 592 (all-gather) or 1184 (reduce-scatter) CTAs of ranks that share a launch. Both sides of each line give the same bits, and miss a rank that stays away."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda", 0)
TILE = 8192


def _loopback(world):
    from nangila.parallel.symm import LoopbackArena

    return LoopbackArena(world, DEV)


class _Rank:
    """One rank of a group of two whose regions are shared with the other's object; on its own, rank 1 never comes."""

    world, provider = 2, "test"

    def __init__(self, rank, region):
        self.rank, self._region = rank, region

    def allocate(self, nbytes):
        if not self._region:
            self._region.append(_loopback(2).allocate(nbytes))
        return self._region[0]


def _object(what, arena, **kw):
    from nangila.parallel import fsdp_collectives as F

    return F.NangilaAllGather(arena=arena, **kw) if what == "all_gather" else F.NangilaReduceScatter(arena=arena, stochastic=False, **kw)


def _call(obj, outs, ins):
    obj.gather(outs, ins) if hasattr(obj, "gather") else obj.reduce(outs, ins, 0.5, unit="u")


def _sizes(what, shard):
    return (shard, 2 * shard) if what == "all_gather" else (2 * shard, shard)


@pytest.mark.parametrize("what", ["reduce_scatter", "all_gather"])
@pytest.mark.parametrize("tiles", [1, 296, 297])
def test_ranks_of_a_group(what, tiles, monkeypatch):
    """Rank 1's wait runs out once (its data lie in rank 0's region from then on); then rank 0 finds word and data, and rank 1 those of rank 0."""
    monkeypatch.setenv("NANGILA_CHUNK", str(TILE))
    gen = torch.Generator(device="cuda").manual_seed(tiles)
    n_in, n_out = _sizes(what, tiles * TILE)
    ins = [(torch.randn(n_in, device=DEV, generator=gen) * 0.02).to(torch.bfloat16) for _ in range(2)]
    want = [torch.empty(n_out, dtype=torch.bfloat16, device=DEV) for _ in range(2)]
    both = _object(what, _loopback(2))
    _call(both, want, ins)
    both.check_status()
    region = []
    ranks = [_object(what, _Rank(r, region), timeout_s=0.3) for r in range(2)]
    got = [torch.full((n_out,), 3.0, dtype=torch.bfloat16, device=DEV) for _ in range(2)]
    _call(ranks[1], [got[1]], [ins[1]])
    with pytest.raises(RuntimeError, match="waiting for rank 0"):
        ranks[1].check_status()
    part = slice(0, tiles * TILE)  # (a gather has written its own shard)
    assert (got[1][part] == 3.0).all()
    _call(ranks[0], [got[0]], [ins[0]])
    ranks[0].check_status()
    assert torch.equal(got[0], want[0])
    next(iter(ranks[1]._regions.values()))["epoch"] = 0  # the same launch again: rank 0's word has come
    _call(ranks[1], [got[1]], [ins[1]])
    ranks[1].check_status()
    assert torch.equal(got[1], want[1])


@pytest.mark.parametrize("what", ["reduce_scatter", "all_gather"])
@pytest.mark.parametrize("tiles", [1, 297, 593])
@pytest.mark.parametrize("emulated", [False, True])
def test_a_rank_that_has_failed(what, tiles, emulated, monkeypatch):
    """Rank 0 has failed and nobody has looked: it stores nothing more, and rank 1 does not take what lies in its slots."""
    monkeypatch.setenv("NANGILA_CHUNK", str(TILE))
    n_in, n_out = _sizes(what, tiles * TILE)
    ins = [torch.randn(n_in, dtype=torch.bfloat16, device=DEV) for _ in range(2)]
    outs = [torch.full((n_out,), 3.0, dtype=torch.bfloat16, device=DEV) for _ in range(2)]
    if emulated:
        obj = _object(what, _loopback(2), timeout_s=0.2)
        _call(obj, outs, ins)
        obj.check_status()
        obj._status[0][0] = 3
        for o in outs:
            o.fill_(3.0)
        _call(obj, outs, ins)
        torch.cuda.synchronize()
        assert int(obj._status[1][0]) != 0 and int(obj._status[1][2]) == 0  # rank 1 has waited for rank 0
        assert (outs[1][:tiles * TILE] == 3.0).all() and (outs[0] == 3.0).all()
        for s in obj._status:
            s.zero_()
    else:
        obj = _object(what, _Rank(0, []), timeout_s=0.2)
        _call(obj, [outs[0]], [ins[0]])  # (makes the status block; nobody else comes)
        with pytest.raises(RuntimeError, match="waiting for rank 1"):
            obj.check_status()
        obj._status[0][0] = 3
        outs[0].fill_(3.0)
        st = next(iter(obj._regions.values()))
        buffers = st["region"].segment._keepalive
        at = st["f"] if what == "all_gather" else st["f1"]
        before = buffers[1][at:at + 8].clone()
        _call(obj, [outs[0]], [ins[0]])
        torch.cuda.synchronize()
        assert (outs[0] == 3.0).all() and torch.equal(buffers[1][at:at + 8], before)  # no data, no word


@pytest.mark.parametrize("what", ["reduce_scatter", "all_gather"])
@pytest.mark.parametrize("tiles", [296, 297, 592, 593])
def test_ranks_that_share_a_launch(what, tiles, monkeypatch):
    """The same bits as in pieces of 100 tiles."""
    monkeypatch.setenv("NANGILA_CHUNK", str(TILE))
    gen = torch.Generator(device="cuda").manual_seed(tiles)
    shard = tiles * TILE
    n_in, n_out = _sizes(what, shard)
    ins = [(torch.randn(n_in, device=DEV, generator=gen) * 0.02).to(torch.bfloat16) for _ in range(2)]
    whole = [torch.empty(n_out, dtype=torch.bfloat16, device=DEV) for _ in range(2)]
    obj = _object(what, _loopback(2))
    for _ in range(2):
        _call(obj, whole, ins)
    for a in range(0, shard, 100 * TILE):
        b = min(shard, a + 100 * TILE)
        part_in = [i.view(-1, shard)[:, a:b].reshape(-1) for i in ins]
        part = [torch.empty(_sizes(what, b - a)[1], dtype=torch.bfloat16, device=DEV) for _ in range(2)]
        _call(obj, part, part_in)
        for w, p in zip(whole, part):
            assert torch.equal(w.view(-1, shard)[:, a:b].reshape(-1), p)
    obj.check_status()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("iterations", [296, 297])
def test_small_shards_are_quantized_by_iterations(iterations, dtype):
    """The same bits as in pieces of ten iterations of 2048 elements."""
    gen = torch.Generator(device="cuda").manual_seed(iterations)
    shard = iterations * 2048 - 8
    ag = _object("all_gather", _loopback(1))
    x = (torch.randn(shard, device=DEV, generator=gen) * 0.02).to(dtype)
    whole = torch.empty_like(x)
    ag.gather([whole], [x])
    for a in range(0, shard, 20480):
        part = torch.empty_like(x[a:a + 20480])
        ag.gather([part], [x[a:a + 20480].clone()])
        assert torch.equal(whole[a:a + 20480], part)
    ag.check_status()
