"""The DGC selection where its path changes: without a previous threshold, on the candidate list, with a threshold that has
grown past the list's range or fallen below it, with ties, at lengths around the groups of eight. One rank and two."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _engine(world, **kw):
    from nangila.parallel.dgc_engine import DGCEngine
    from nangila.parallel.symm import LoopbackArena

    dev = torch.device("cuda", 0)
    return DGCEngine(LoopbackArena(world, dev), dev, **kw)


def _check(eng, grads, us, vs, m):
    """One step against PyTorch: the entries at or above the k-th largest |v| are sent, all of them where several equal it."""
    world = len(grads)
    k = eng.bucket_state(0, grads).k
    want = torch.zeros_like(grads[0], dtype=torch.float32)
    size = torch.zeros_like(want)
    counts = []
    m32 = float(torch.tensor(m, dtype=torch.float32))
    for r, g in enumerate(grads):
        us[r] = (us[r].double() * m32 + g.double()).float()  # a fused multiply-add: one rounding
        vs[r] = vs[r] + us[r]
        sent = vs[r].abs() >= vs[r].abs().topk(k).values[-1]
        counts.append(int(sent.sum()))
        want += torch.where(sent, vs[r], 0.0) / world
        size += torch.where(sent, vs[r], 0.0).abs() / world
        vs[r] = torch.where(sent, 0.0, vs[r])
        us[r] = torch.where(sent, 0.0, us[r])
    eng.reduce(0, grads)
    eng.check_status()
    st = eng.buckets[0]
    for r in range(world):
        assert int(st.out_count[r][0]) == counts[r]
        assert torch.equal(st.v[r], vs[r]) and torch.equal(st.u[r], us[r])
        # the ranks' values are added one by one in the bucket's type: every addition rounds a number no larger than the sum of
        # their magnitudes (which is what counts where they cancel) by at most the type's unit roundoff (bf16: 8 significant bits)
        eps = world * (2.0 ** -8 if grads[r].dtype == torch.bfloat16 else 2.0 ** -24)
        assert ((grads[r].float() - want).abs() <= eps * size + 1e-30).all()
    return int(st.scratch[0][2048 + 2048 + 512 + 2])


@pytest.mark.parametrize("world", [1, 2])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n", [1000, 1007, 8192 + 8, 296 * 1024 * 8 + 3])
def test_every_path_selects_the_same(world, dtype, n):
    gen = torch.Generator(device="cuda").manual_seed(n)
    eng = _engine(world, sparsity=0.99, momentum=0.9)
    us = [torch.zeros(n, device="cuda") for _ in range(world)]
    vs = [torch.zeros(n, device="cuda") for _ in range(world)]
    # scales of the steps: build up, hold, jump far above the list's range, fall far below it, hold
    paths = []
    for scale in (1.0, 1.0, 0.5, 0.5, 40.0, 1e-4, 1e-4, 1e-4):
        grads = [(torch.randn(n, device="cuda", generator=gen) * scale).to(dtype) for _ in range(world)]
        if dtype == torch.bfloat16 and not paths:
            # the first accumulators would be the gradients themselves, with more ties in 16 bits than the list holds: start from a state
            eng.bucket_state(0, grads)
            for r in range(world):
                us[r] = torch.rand(n, device="cuda", generator=gen) * 0.1
                eng.buckets[0].u[r].copy_(us[r])
        paths.append(_check(eng, [g.clone() for g in grads], us, vs, 0.9))
    assert paths[0] == 0 and 1 in paths[1:] and 0 in paths[1:], paths


def test_ties_at_the_threshold_are_all_sent_or_cut_at_the_capacity():
    eng = _engine(1, sparsity=0.99, momentum=0.0)
    n = 40_000
    for step in range(3):
        g = torch.zeros(n, device="cuda")
        g[step * 1000:step * 1000 + 420] = 2.0  # k = 401 (or 400): 420 equal entries, within the capacity
        eng.reduce(0, g)
        eng.check_status()
        assert int(eng.buckets[0].out_count[0][0]) == 420
        assert int((g == 2.0).sum()) == 420 and not eng.buckets[0].v[0].any()


def test_a_full_candidate_list_stops_the_collection():
    """Gradients that jump put nearly every entry above the previous threshold. The list has no room for them, so what is reserved must
    stay near its size (every warp may add its 256 entries once or twice after it is full) instead of counting them all."""
    n = 16_777_216
    gen = torch.Generator(device="cuda").manual_seed(3)
    eng = _engine(1, sparsity=0.999)
    us, vs = [torch.zeros(n, device="cuda")], [torch.zeros(n, device="cuda")]
    paths = [_check(eng, [torch.randn(n, device="cuda", generator=gen) * scale], us, vs, 0.9) for scale in (1e-3, 1.0)]
    assert paths == [0, 0]
    st = eng.buckets[0]
    reserved = int(st.scratch[0][2048 + 2048 + 512 + 7])
    capacity = (st.scratch[0].numel() - 2048) // 2  # an upper bound: the fixed words come off
    assert 0 < reserved <= capacity + eng._grid(n) * 8 * 256 * 2 < n // 3 * 2
