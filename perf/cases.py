"""What the GPU side of the framework is timed on: one case per public path, over the sizes that training
runs and circuits bring.

Kinds
  bucket   one DDP gradient bucket through the prediction-residual compressor (``PredResEngine.reduce``)
  dgc      one DDP bucket through Deep Gradient Compression (``DGCEngine.reduce``), new gradients every step
  psgd     the matrices of one DDP bucket through PowerSGD (``PowerSGDEngine.reduce``)
  rs       the gradient reduce-scatter of one FSDP unit (``NangilaReduceScatter.reduce``)
  ag       the parameter all-gather of one FSDP unit (``NangilaAllGather.gather``)
  packet   one layer over the wire: ``compress_gpu``, ``decompress_gpu`` with its checksum, ``update_gpu``
  ce       the loss of a language model's head, forward and backward (``fused_cross_entropy``)
  sculptor one calibration step: every layer recorded, every pair's statistics advanced (``DeviceSculptor``)
  spmv     ``y = A x`` of a circuit matrix with device vectors (``DeviceCsr.matvec_device``)
  solve    a circuit matrix solved for one right-hand side (``DeviceCsr.solve``)

The group kinds (rs, ag) emulate ``world`` ranks on one device, as the kernel tests do; bucket, dgc and psgd run a
group of one rank.
"""
import math

import numpy as np
import torch

DTYPES = {"fp32": torch.float32, "bf16": torch.bfloat16, "fp16": torch.float16}
SIZE = {"fp32": 4, "bf16": 2, "fp16": 2}
DGC_WARM = 8      # DGC steps before the measured one: the unsent mass has built up
SPARSITY = 0.999
CG_STEPS = 4000


def listed():
    return [
        # a 100 MB bf16 bucket of a training run whose gradients have nothing to predict: nearly all calls of such a run
        {"name": "bucket_lean_bf16", "kind": "bucket", "n": 52_428_800, "dtype": "bf16", "gain": 0.0},
        # a 25 MB fp32 bucket (DDP's default size) with the momentum prediction on, ragged length
        {"name": "bucket_predicted_fp32", "kind": "bucket", "n": 6_553_605, "dtype": "fp32", "gain": 1.0},
        # a 25 MB bf16 bucket of a BERT-large step at 99.9 % sparsity
        {"name": "dgc_bf16", "kind": "dgc", "n": 13_107_200, "dtype": "bf16"},
        # the convolutions of a ResNet-50 bucket (last stage), rank 4
        {"name": "powersgd_resnet_bf16", "kind": "psgd", "shapes": "512x4608,2048x512,512x2048,2048x1024", "rank": 4, "dtype": "bf16"},
        # gradients of one transformer block (12 x 1024 x 1024 parameters) on four ranks
        {"name": "fsdp_reduce_scatter_bf16", "kind": "rs", "n": 12_582_912, "world": 4, "dtype": "bf16", "ef": False},
        # parameters of the same block, INT8
        {"name": "fsdp_all_gather_int8", "kind": "ag", "n": 3_145_728, "world": 4, "dtype": "bf16", "bits": 8},
        # a bias or norm layer sent as a packet: the cost of the calls themselves
        {"name": "packet_small_fp32", "kind": "packet", "n": 10_007, "dtype": "fp32"},
        # the token embedding of GPT-2 small (50304 x 768 bf16) sent as a packet
        {"name": "packet_embedding_bf16", "kind": "packet", "n": 38_633_472, "dtype": "bf16"},
        # the loss of a GPT-2 small step, 8 x 1024 tokens
        {"name": "loss_gpt2", "kind": "ce", "rows": 8192, "classes": 50257, "stride": 50304},
        # calibration over eight 768 x 768 projections: 28 pairs
        {"name": "sculptor_step_bf16", "kind": "sculptor", "layers": 8, "n": 589_824, "dtype": "bf16"},
        # an RC ladder of a million nodes, the simulator's device benchmark
        {"name": "spmv_ladder", "kind": "spmv", "pattern": "ladder", "n": 1_000_000},
        # the operating point of a 256 x 256 resistor mesh
        {"name": "solve_mesh", "kind": "solve", "pattern": "mesh", "n": 65_536},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["bucket", "dgc", "psgd", "rs", "ag", "packet", "ce", "sculptor", "spmv", "solve"])
    dtype = rng.choice(["fp32", "bf16", "bf16", "fp16"])
    if kind == "bucket":
        return {"kind": kind, "n": _log(rng, 65_536, 52_428_800 * 2 // SIZE[dtype]), "dtype": dtype, "gain": rng.choice([0.0, 1.0])}
    if kind == "dgc":
        return {"kind": kind, "n": _log(rng, 65_536, 33_000_000), "dtype": dtype}
    if kind == "psgd":
        shapes, left = [], 8_000_000
        for _ in range(rng.randint(1, 6)):
            m, n = 8 * _log(rng, 8, 512), 8 * _log(rng, 8, 1024)
            if m * n <= left:
                shapes.append("%dx%d" % (m, n))
                left -= m * n
        return {"kind": kind, "shapes": ",".join(shapes or ["768x2304"]), "rank": rng.choice([1, 2, 4, 8]), "dtype": dtype}
    if kind == "rs":
        world = rng.choice([2, 4, 8])
        return {"kind": kind, "n": 8 * world * _log(rng, 1024, 50_331_648 // (8 * world * world)), "world": world, "dtype": dtype,
                "ef": rng.random() < 0.5}
    if kind == "ag":
        world = rng.choice([2, 4, 8])
        return {"kind": kind, "n": 8 * _log(rng, 1024, 50_331_648 // (8 * world * world)), "world": world, "dtype": dtype,
                "bits": rng.choice([4, 8, 8])}
    if kind == "packet":
        return {"kind": kind, "n": _log(rng, 1000, 38_633_472 * 2 // SIZE[dtype]), "dtype": dtype}
    if kind == "ce":
        classes = _log(rng, 1000, 50_257)
        stride = (classes + 127) // 128 * 128
        return {"kind": kind, "rows": _log(rng, 64, 8192), "classes": classes, "stride": stride}
    if kind == "sculptor":
        layers = rng.randint(2, 8)
        pairs = layers * (layers - 1) // 2
        return {"kind": kind, "layers": layers, "n": _log(rng, 1000, 16_000_000 // pairs), "dtype": dtype}
    if kind == "spmv":
        return {"kind": kind, "pattern": rng.choice(["ladder", "mesh"]), "n": _log(rng, 10_000, 4_000_000)}
    return {"kind": "solve", "pattern": "mesh", "n": _log(rng, 2_500, 400_000)}


# ---- inputs ----------------------------------------------------------------------------------------------------


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _grads(n, dtype, seed, count):
    """``count`` successive gradients of one bucket: a common part, step noise, and a scale that differs from parameter to
    parameter as it does from layer to layer (it is constant over runs of 4096 elements)."""
    g = _gen(seed)
    blocks = (n + 4095) // 4096
    scale = torch.exp(0.7 * torch.randn(blocks, device="cuda", generator=g)).repeat_interleave(4096)[:n] * 1e-3
    base = torch.randn(n, device="cuda", generator=g)
    return [((0.8 * base + 0.6 * torch.randn(n, device="cuda", generator=g)) * scale).to(dtype) for _ in range(count)]


def _shapes(case):
    return [tuple(int(v) for v in s.split("x")) for s in case["shapes"].split(",")]


def _matrices(case, seed):
    """Gradient matrices: a few strong directions and noise. The first list is the step before, the second the measured one."""
    g = _gen(seed)
    before, now = [], []
    for m, n in _shapes(case):
        left = torch.randn(m, 6, device="cuda", generator=g) * torch.tensor([2.0, 1.4, 1.0, 0.7, 0.5, 0.35], device="cuda")
        right = torch.randn(6, n, device="cuda", generator=g)
        for out in (before, now):
            out.append(((left @ right + torch.randn(m, n, device="cuda", generator=g)) * 1e-3).to(DTYPES[case["dtype"]]))
    return before, now


def _circuit(case, seed):
    """CSR arrays of a conductance matrix: a ladder (tridiagonal) or a square-ish mesh (five points), every node with a leak."""
    n = case["n"]
    rng = np.random.RandomState(seed % (1 << 31))
    idx = np.arange(n, dtype=np.int64)
    if case["pattern"] == "ladder":
        edges = [(idx[:-1], idx[1:])]
    else:
        side = int(math.isqrt(n))
        right = idx[(idx % side != side - 1) & (idx + 1 < n)]
        edges = [(right, right + 1), (idx[: n - side], idx[side:])]
    rows, cols, vals = [], [], []
    diag = np.full(n, 1e-2)
    for a, b in edges:
        g = np.exp(0.3 * rng.standard_normal(a.size))
        rows += [a, b]
        cols += [b, a]
        vals += [-g, -g]
        diag += np.bincount(a, weights=g, minlength=n) + np.bincount(b, weights=g, minlength=n)
    rows, cols, vals = np.concatenate(rows + [idx]), np.concatenate(cols + [idx]), np.concatenate(vals + [diag])
    order = np.argsort(rows * n + cols, kind="stable")
    row_ptr = np.zeros(n + 1, dtype=np.int64)
    np.cumsum(np.bincount(rows, minlength=n), out=row_ptr[1:])
    return row_ptr.astype(np.int32), cols[order].astype(np.int32), vals[order], rng.standard_normal(n)


class _Bucket:
    """What DDP hands a communication hook, as far as the PowerSGD engine looks at it."""

    def __init__(self, grads):
        self._grads = grads

    def gradients(self):
        return self._grads


# ---- prepare / run ---------------------------------------------------------------------------------------------


def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed)


def run(state):
    return globals()["_run_" + state["kind"]](state)


def _prepare_bucket(case, seed):
    from nangila.parallel.predres_engine import PredResEngine
    from nangila.parallel.symm import LoopbackArena

    dev = torch.device("cuda", 0)
    g = _grads(case["n"], DTYPES[case["dtype"]], seed, 3)
    # round to nearest with error feedback, as the DDP hook sets it up
    eng = PredResEngine(LoopbackArena(1, dev), dev, stochastic=False, use_side_stream=False, adaptive_gain=False)
    eng.fixed_gain = case["gain"]
    eng.probe_every = 64  # what the spacing of the probes grows to while they find nothing
    for t in (0, 1):  # two exact steps build the history
        eng.reduce(0, [g[t]], compressed=False, step=t)
    return {"kind": "bucket", "eng": eng, "bucket": g[2], "step": 2}


def _run_bucket(s):
    # in place; called again on its own result it sees a stationary gradient (what was not sent is in the error memory)
    st = s["eng"].reduce(0, [s["bucket"]], compressed=True, step=s["step"])
    s["step"] += 1
    return {"bucket": s["bucket"], "error": st.ef[0], "history": st.curr[0] if st.pred_gain > 0 else None}


def _prepare_dgc(case, seed):
    from nangila.parallel.dgc_engine import DGCEngine
    from nangila.parallel.symm import LoopbackArena

    dev = torch.device("cuda", 0)
    source = _grads(case["n"], DTYPES[case["dtype"]], seed, 4)
    eng = DGCEngine(LoopbackArena(1, dev), dev, sparsity=SPARSITY)
    bucket = torch.empty_like(source[0])
    for t in range(DGC_WARM):
        bucket.copy_(source[t % 4])
        eng.reduce(0, bucket)
    return {"kind": "dgc", "eng": eng, "bucket": bucket, "source": source, "step": DGC_WARM}


def _run_dgc(s):
    s["bucket"].copy_(s["source"][s["step"] % 4])  # backward fills the bucket
    s["step"] += 1
    s["eng"].reduce(0, s["bucket"])
    st = s["eng"].buckets[0]
    return {"bucket": s["bucket"], "velocity": st.u[0], "unsent": st.v[0]}


def _prepare_psgd(case, seed):
    from nangila.parallel.powersgd_engine import PowerSGDEngine
    from nangila.parallel.symm import LoopbackArena

    dev = torch.device("cuda", 0)
    before, now = _matrices(case, seed)
    eng = PowerSGDEngine(LoopbackArena(1, dev), dev, rank=case["rank"])
    flat = torch.cat([g.reshape(-1) for g in before])
    views, at = [], 0
    for m, n in _shapes(case):
        views.append(flat[at:at + m * n].view(m, n))
        at += m * n
    bucket = _Bucket(views)
    eng.reduce(0, bucket, flat)
    for v, g in zip(views, now):
        v.copy_(g)
    return {"kind": "psgd", "eng": eng, "bucket": bucket, "flat": flat}


def _run_psgd(s):
    # in place; called again on its own result it sees the same sum of gradient and error memory
    s["eng"].reduce(0, s["bucket"], s["flat"])
    states = [s["eng"].states[(0, i)] for i in range(len(s["bucket"].gradients()))]
    return {"bucket": s["flat"], "error": [st.ef[0] for st in states]}


def _prepare_rs(case, seed):
    from nangila.parallel.fsdp_collectives import NangilaReduceScatter
    from nangila.parallel.symm import LoopbackArena

    dev = torch.device("cuda", 0)
    ins = _grads(case["n"], DTYPES[case["dtype"]], seed, case["world"])
    outs = [torch.empty(case["n"] // case["world"], dtype=ins[0].dtype, device=dev) for _ in ins]
    rs = NangilaReduceScatter(arena=LoopbackArena(case["world"], dev), error_feedback=case["ef"])
    rs.reduce([o.clone() for o in outs], ins, 1.0 / case["world"], unit="other")  # the exchange region exists from the first unit on
    return {"kind": "rs", "rs": rs, "ins": ins, "outs": outs, "scale": 1.0 / case["world"]}


def _run_rs(s):
    s["rs"].reduce(s["outs"], s["ins"], s["scale"], unit="block")
    return s["outs"]


def _prepare_ag(case, seed):
    from nangila.parallel.fsdp_collectives import NangilaAllGather
    from nangila.parallel.symm import LoopbackArena

    dev = torch.device("cuda", 0)
    ins = [p * 20 for p in _grads(case["n"], DTYPES[case["dtype"]], seed, case["world"])]
    outs = [torch.empty(case["n"] * case["world"], dtype=ins[0].dtype, device=dev) for _ in ins]
    ag = NangilaAllGather(arena=LoopbackArena(case["world"], dev), bits=case["bits"])
    ag.gather([o.clone() for o in outs], ins)
    return {"kind": "ag", "ag": ag, "ins": ins, "outs": outs}


def _run_ag(s):
    s["ag"].gather(s["outs"], s["ins"])
    return s["outs"]


def _prepare_packet(case, seed):
    import nangila

    hook = nangila.NangilaHook.all_drivers(1, nangila.NangilaConfig(warmup_steps=0, shadow_run_steps=0))
    hook.step()
    g = _grads(case["n"], DTYPES[case["dtype"]], seed, 3)
    hook.update_gpu(0, g[0], sync_mode=0)
    hook.update_gpu(0, g[1], sync_mode=0)
    return {"kind": "packet", "hook": hook, "grad": g[2], "n": case["n"]}


def _run_packet(s):
    hook, n = s["hook"], s["n"]
    packet = hook.compress_gpu(0, s["grad"])
    out = hook.decompress_gpu(0, packet, n)  # verifies the checksum
    hook.update_gpu(0, out)
    scales = 52 + 4 * ((n + 63) // 64)
    return {"gain": packet[48:52].view(torch.float32), "scales": packet[52:scales].view(torch.float32), "codes": packet[scales:], "out": out}


def _prepare_ce(case, seed):
    g = _gen(seed)
    rows, v, stride = case["rows"], case["classes"], case["stride"]
    logits = torch.empty(rows, stride, dtype=torch.bfloat16, device="cuda")
    for r in range(0, rows, 1024):
        logits[r:r + 1024] = 2.0 * torch.randn(min(1024, rows - r), stride, device="cuda", generator=g)
    targets = torch.randint(0, v, (rows,), device="cuda", generator=g)
    return {"kind": "ce", "logits": logits.requires_grad_(True), "targets": targets, "classes": v}


def _run_ce(s):
    from nangila.ops.fused_ce import fused_cross_entropy

    loss = fused_cross_entropy(s["logits"], s["targets"], s["classes"])
    (grad,) = torch.autograd.grad(loss, s["logits"])
    return {"loss": loss.detach(), "grad": grad}


def _sculptor_steps(case, seed):
    """Gradients of all layers at three successive steps; neighbours share a part, as the layers of a model do."""
    g = _gen(seed)
    n, dtype = case["n"], DTYPES[case["dtype"]]
    steps = []
    for _ in range(3):
        common = torch.randn(n, device="cuda", generator=g)
        steps.append([((0.9 * common + 0.5 * torch.randn(n, device="cuda", generator=g)) * (0.5 + 0.1 * i)).to(dtype) for i in range(case["layers"])])
    return steps


def _prepare_sculptor(case, seed):
    from nangila.ops import DeviceSculptor

    ds = DeviceSculptor()
    steps = _sculptor_steps(case, seed)
    for grads in steps[:2]:
        for i, g in enumerate(grads):
            ds.record(i, g)
        ds.end_step()
    return {"kind": "sculptor", "ds": ds, "grads": steps[2]}


def _run_sculptor(s):
    for i, g in enumerate(s["grads"]):
        s["ds"].record(i, g)
    s["ds"].end_step()
    return [s["ds"]._pair_state[k] for k in sorted(s["ds"]._pair_state)]


def _prepare_spmv(case, seed):
    from nangila_spice.gpu import DeviceCsr

    row_ptr, col, val, x = _circuit(case, seed)
    return {"kind": "spmv", "m": DeviceCsr(row_ptr, col, val), "x": torch.from_numpy(x).cuda(), "y": torch.empty(case["n"], dtype=torch.float64, device="cuda")}


def _run_spmv(s):
    s["m"].matvec_device(s["x"], s["y"], torch.cuda.current_stream().cuda_stream)
    return s["y"]


def _prepare_solve(case, seed):
    from nangila_spice.gpu import DeviceCsr

    row_ptr, col, val, b = _circuit(case, seed)
    m = DeviceCsr(row_ptr, col, val)
    m.solve(np.ones(case["n"]))  # the simulator solves the same matrix again and again
    return {"kind": "solve", "m": m, "b": b}


def _run_solve(s):
    x, _, _, converged = s["m"].solve(s["b"], tol=1e-10)
    if not converged:
        raise RuntimeError("the solver did not converge")
    return x


# ---- what a pass cannot do without -----------------------------------------------------------------------------


def _pattern_nnz(case):
    n = case["n"]
    if case["pattern"] == "ladder":
        return 3 * n - 2
    side = int(math.isqrt(n))
    return n + 2 * (n - side) + 2 * (n - 1 - (n - 1) // side)  # diagonal, vertical neighbours, horizontal ones


def work(case):
    kind = case["kind"]
    if kind == "bucket":
        n, s = case["n"], SIZE[case["dtype"]]
        state = 4 if case["dtype"] == "fp32" else 2
        # gradient and error memory in and out; with a prediction the two-step history in and the new one out
        return {"bytes": n * (2 * s + 2 * state + (3 * state if case["gain"] > 0 else 0)), "flops": 0}
    if kind == "dgc":
        return {"bytes": case["n"] * (2 * SIZE[case["dtype"]] + 16), "flops": 0}
    if kind == "psgd":
        el = sum(m * n for m, n in _shapes(case))
        return {"bytes": el * (2 * SIZE[case["dtype"]] + 4), "flops": 6 * el * case["rank"]}
    if kind == "rs":
        n, w, s = case["n"], case["world"], SIZE[case["dtype"]]
        return {"bytes": w * n * (s + (4 if case["ef"] else 0)) + n * s, "flops": 0}
    if kind == "ag":
        n, w, s = case["n"], case["world"], SIZE[case["dtype"]]
        return {"bytes": w * n * s + w * w * n * s, "flops": 0}
    if kind == "packet":
        # encode: gradient, history, error memory in, error memory and packet out; decode: packet and history in, values out;
        # update: values in, history out
        n = case["n"]
        return {"bytes": n * (SIZE[case["dtype"]] + 16 + 12 + 8) + 2 * (52 + n // 2 + n // 16), "flops": 0}
    if kind == "ce":
        return {"bytes": case["rows"] * 2 * (case["classes"] + case["stride"]), "flops": 0}
    if kind == "sculptor":
        pairs = case["layers"] * (case["layers"] - 1) // 2
        return {"bytes": case["n"] * (case["layers"] * SIZE[case["dtype"]] + pairs * 40), "flops": 0}
    n, nnz = case["n"], _pattern_nnz(case)
    # (solve: the matrix and the two vectors once; the iterations, whose number depends on the matrix, come on top)
    return {"bytes": 12 * nnz + 4 * (n + 1) + 16 * n, "flops": 2 * nnz}


def tolerance(case):
    kind, dtype = case["kind"], case.get("dtype")
    if kind in ("bucket", "rs"):
        # the same codes but for ties: a code that falls on the other side of one is off by a whole step
        return {"rel": 1e-3 if dtype == "fp32" else 1e-2, "max": 0.9}
    if kind == "dgc":
        return {"rel": 1e-2, "max": 0.9}
    if kind == "psgd":
        return {"rel": 1e-2, "max": 0.2}
    if kind == "ag":
        return {"rel": 2e-3, "max": 0.2}
    if kind == "packet":
        # the gain is a sum in no fixed order, so a code may fall on the other side of a tie
        return {"rel": 1e-3, "max": 0.9, "differ": 2e-5}
    if kind == "ce":
        return {"rel": 1e-3, "max": 0.05}
    if kind == "sculptor":
        return {"rel": 1e-6, "max": 1e-4}
    if kind == "spmv":
        return {"rel": 1e-15, "max": 1e-13}
    return {"rel": 2e-8, "max": 2e-6}  # the solver stops at a residual of 1e-10


# ---- the same in plain 64-bit arithmetic -----------------------------------------------------------------------


def exact(case, seed):
    f = globals().get("_exact_" + case["kind"])
    return f(case, seed) if f else None


def _blocks64(x):
    n = x.numel()
    return torch.nn.functional.pad(x, (0, -n % 64)).view(-1, 64)


def _bf16_up(s):
    """The smallest bf16 number at or above s (s >= 0)."""
    bits = (s.to(torch.float32).view(torch.int32) + 0xFFFF) >> 16
    return (bits << 16).view(torch.float32).double()


def _quantized(x, bits, round_up_bf16):
    """q * scale of the block format: one scale per 64 elements, rounded to nearest."""
    top = (1 << (bits - 1)) - 1
    b = _blocks64(x)
    s = b.abs().amax(1, keepdim=True) / top
    if round_up_bf16:
        s = _bf16_up(s)
    q = torch.floor(torch.where(s > 1e-30, b / torch.where(s > 1e-30, s, torch.ones_like(s)), torch.zeros_like(b)) + 0.5)
    q = q.clamp(-top - 1, top)
    return (q * s).view(-1)[:x.numel()], q, s


def _exact_bucket(case, seed):
    g = [t.double() for t in _grads(case["n"], DTYPES[case["dtype"]], seed, 3)]
    state = torch.float32 if case["dtype"] == "fp32" else torch.bfloat16
    prev, curr = g[0].to(state).double(), g[1].to(state).double()
    ghat = case["gain"] * (curr + 0.9 * (curr - prev))
    x = g[2] - ghat
    sent = _quantized(x, 4, True)[0]
    out = sent + ghat
    # in 16 bits the sum of gradient and error memory and the code's own arithmetic are rounded, so that codes near a tie
    # differ; what is left over after them has no exact value
    return {"bucket": out, "error": x - sent if case["dtype"] == "fp32" else None, "history": out if case["gain"] > 0 else None}


def _exact_dgc(case, seed):
    source = _grads(case["n"], DTYPES[case["dtype"]], seed, 4)
    n = case["n"]
    k = min(max(1, math.ceil(float(np.float32(n) * (np.float32(1.0) - np.float32(SPARSITY))))), n)
    u = torch.zeros(n, dtype=torch.float64, device="cuda")
    v = torch.zeros_like(u)
    for t in range(DGC_WARM + 1):
        u = float(np.float32(0.9)) * u + source[t % 4].double()
        v = v + u
        tau = v.abs().topk(k).values[-1]
        sent = (v.abs() >= tau) & (v != 0)  # entries equal to the threshold are all sent (16-bit gradients have many)
        out = torch.where(sent, v, torch.zeros_like(v))
        v = torch.where(sent, torch.zeros_like(v), v)
        u = torch.where(sent, torch.zeros_like(u), u)
    return {"bucket": out, "velocity": u, "unsent": v}


def _orthonormal(p):
    p = p.clone()
    for c in range(p.shape[1]):
        for j in range(c):
            p[:, c] -= (p[:, c] @ p[:, j]) * p[:, j]
        nrm = p[:, c].norm()
        p[:, c] = p[:, c] / nrm if nrm > 1e-10 else 0.0
    return p


def _exact_psgd(case, seed):
    outs, errors = [], []
    for before, now in zip(*_matrices(case, seed)):
        m, n = before.shape
        r = min(case["rank"], m, n)
        i = torch.arange(n, device="cuda", dtype=torch.float64)[:, None] + torch.arange(r, device="cuda", dtype=torch.float64)[None, :]
        q = _orthonormal((i % 100) / 100.0)
        ef = torch.zeros(m, n, dtype=torch.float64, device="cuda")
        for g in (before, now):
            mat = g.double() + ef
            p = _orthonormal(mat @ q)
            qn = mat.t() @ p
            out = p @ qn.t()
            ef = mat - out
            q = _orthonormal(qn)
        outs.append(out.reshape(-1))
        errors.append(ef)
    return {"bucket": torch.cat(outs), "error": errors}


def _exact_rs(case, seed):
    if not case["ef"]:
        return None  # rounds with a random number per element
    ins = _grads(case["n"], DTYPES[case["dtype"]], seed, case["world"])
    w, shard = case["world"], case["n"] // case["world"]
    total = torch.zeros(case["n"], dtype=torch.float64, device="cuda")
    for g in ins:
        for r in range(w):  # blocks of 64 begin at every shard
            total[r * shard:(r + 1) * shard] += _quantized(g[r * shard:(r + 1) * shard].double(), 4, True)[0]
    return [total[r * shard:(r + 1) * shard] / w for r in range(w)]


def _exact_ag(case, seed):
    full = torch.cat([_quantized((p * 20).double(), case["bits"], True)[0] for p in _grads(case["n"], DTYPES[case["dtype"]], seed, case["world"])])
    return [full for _ in range(case["world"])]


def _exact_packet(case, seed):
    g = [t.double() for t in _grads(case["n"], DTYPES[case["dtype"]], seed, 3)]
    mu = float(np.float32(0.9))
    ghat = g[1] + mu * (g[1] - g[0])
    kappa = min(max(float(g[2] @ ghat) / float(ghat @ ghat), 0.0), 1.0)
    x = g[2] - kappa * ghat
    sent, _, s = _quantized(x, 4, False)
    return {"gain": torch.tensor([kappa], dtype=torch.float64), "scales": s.view(-1), "codes": None, "out": sent + kappa * ghat}


def _exact_ce(case, seed):
    s = _prepare_ce(case, seed)
    logits, rows, v = s["logits"].detach(), case["rows"], case["classes"]
    grad = torch.zeros(rows, case["stride"], dtype=torch.float64, device="cuda")
    loss = torch.zeros((), dtype=torch.float64, device="cuda")
    for r in range(0, rows, 1024):
        x = logits[r:r + 1024, :v].double()
        t = s["targets"][r:r + 1024, None]
        logp = torch.log_softmax(x, 1)
        loss -= logp.gather(1, t).sum()
        p = logp.exp_()
        p.scatter_add_(1, t, torch.full_like(t, -1, dtype=torch.float64))
        grad[r:r + 1024, :v] = p / rows
    return {"loss": loss / rows, "grad": grad}


def _exact_sculptor(case, seed):
    steps = [[g.double() for g in grads] for grads in _sculptor_steps(case, seed)]
    outs = []
    for i in range(case["layers"]):
        for j in range(i + 1, case["layers"]):
            x, y = torch.stack([s[i] for s in steps]), torch.stack([s[j] for s in steps])
            mx, my = x.mean(0), y.mean(0)
            outs.append(torch.cat([mx, my, ((x - mx) ** 2).sum(0), ((y - my) ** 2).sum(0), ((x - mx) * (y - my)).sum(0)]))
    return outs


def _csr(case, seed):
    row_ptr, col, val, b = _circuit(case, seed)
    n = case["n"]
    a = torch.sparse_csr_tensor(torch.from_numpy(row_ptr.astype(np.int64)).cuda(), torch.from_numpy(col.astype(np.int64)).cuda(),
                                torch.from_numpy(val).cuda(), size=(n, n))
    rows = np.repeat(np.arange(n), np.diff(row_ptr))
    return a, torch.from_numpy(val[rows == col]).cuda(), torch.from_numpy(b).cuda()


def _exact_spmv(case, seed):
    a, _, x = _csr(case, seed)
    return a @ x


def _exact_solve(case, seed):
    a, diag, b = _csr(case, seed)  # symmetric and positive definite: conjugate gradients with the diagonal
    x = torch.zeros_like(b)
    r = b.clone()
    z = r / diag
    p = z.clone()
    rz = r @ z
    for step in range(CG_STEPS):
        ap = a @ p
        alpha = rz / (p @ ap)
        x += alpha * p
        r -= alpha * ap
        if step % 16 == 0 and float(r.norm()) < 1e-14 * float(b.norm()):
            break
        z = r / diag
        new = r @ z
        p = z + (new / rz) * p
        rz = new
    return x.cpu()
