#!/usr/bin/env python
"""FP64 CSR SpMV benchmark of the circuit simulator's device kernels.

The workload is the one of the reference's GPU benchmark (a tridiagonal matrix, the pattern of an RC
ladder; 1 M rows, 200 products: ``nangila-spice/nangila-node/src/bin/bench_gpu.rs``) plus a size that
does not fit in L2, and a band of nine diagonals, whose rows are too long for the thread-per-row kernel that ladders
take: its slices are staged by bulk copies, in blocks of 2048 or (``NANGILA_SPMV_TILE=1024``) 1024 entries.
The library baseline is the same product through ``torch.sparse_csr_tensor`` (cuSPARSE).
Vectors stay on the device in both arms; timing is by CUDA events after warm-up. The products of a run repeat on the same
data: where ``fits_l2`` is true they come from L2.

    python bench/spmv_bench.py [--rows 1000000 16000000] [--iters 200] [--out FILE]
"""
import argparse
import json
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))

from nangila.utils.benchmarking import ClockSampler  # noqa: E402
from nangila_spice.gpu import DeviceCsr, tridiagonal  # noqa: E402


def peaks():
    path = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "MEASURED_PEAKS.json")
    try:
        return float(json.load(open(path))["hbm_gbs"]), "measured"
    except Exception:
        return 6650.0, "fallback"


def timed(fn, iters: int) -> float:
    for _ in range(5):
        fn()
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    for _ in range(iters):
        fn()
    e1.record()
    torch.cuda.synchronize()
    return e0.elapsed_time(e1) / iters


def banded(n: int, half: int):
    """CSR arrays of a band of 2 half + 1 diagonals, diagonally dominant."""
    first, last = np.maximum(np.arange(n) - half, 0), np.minimum(np.arange(n) + half, n - 1)
    lens = last - first + 1
    row_ptr = np.concatenate([[0], np.cumsum(lens)])
    rows = np.repeat(np.arange(n), lens)
    col = first[rows] + np.arange(row_ptr[-1]) - row_ptr[rows]
    return row_ptr.astype(np.int32), col.astype(np.int32), np.where(col == rows, 2.0 * half + 1.0, -1.0)


def main() -> int:
    ap = argparse.ArgumentParser()
    ap.add_argument("--rows", type=int, nargs="+", default=[1_000_000, 16_000_000])
    ap.add_argument("--iters", type=int, default=200)
    ap.add_argument("--out", default=None)
    args = ap.parse_args()
    torch.cuda.set_device(0)
    hbm, src = peaks()
    stream = torch.cuda.current_stream().cuda_stream
    results = []
    for n, half in [(n, half) for n in args.rows for half in (1, 4)]:
        row_ptr, col, val = tridiagonal(n) if half == 1 else banded(n, half)
        nnz = int(val.size)
        m = DeviceCsr(row_ptr, col, val)
        x = torch.randn(n, dtype=torch.float64, device="cuda")
        y = torch.empty_like(x)
        sampler = ClockSampler(0).start()
        ours = timed(lambda: m.matvec_device(x, y, stream), args.iters)
        clocks = sampler.stop()
        m.check_status()
        variants = {}
        y2 = torch.empty_like(x)
        if half > 1:  # ladders do not look at the tile size
            os.environ["NANGILA_SPMV_TILE"] = "1024"
            small = DeviceCsr(row_ptr, col, val)
            os.environ.pop("NANGILA_SPMV_TILE")
            variants["tile_1024_variant_ms"] = timed(lambda: small.matvec_device(x, y2, stream), args.iters)
            assert torch.allclose(y, y2, rtol=1e-13, atol=1e-12)
            small.close()
        mp = DeviceCsr(row_ptr, col, val, plain_loads=True)
        variants["plain_load_variant_ms"] = timed(lambda: mp.matvec_device(x, y2, stream), args.iters)
        assert torch.allclose(y, y2, rtol=1e-13, atol=1e-12)
        mp.close()
        A = torch.sparse_csr_tensor(torch.from_numpy(row_ptr.astype(np.int64)).cuda().to(torch.int32), torch.from_numpy(col).cuda(),
                                    torch.from_numpy(val).cuda(), size=(n, n))
        ref_y = A @ x
        err = (ref_y - y).abs().max().item()
        lib = timed(lambda: torch.mv(A, x), args.iters)
        # algorithmic traffic: values + column indices + row pointers + x read once + y written once
        bytes_moved = nnz * 12 + (n + 1) * 4 + n * 16
        rec = {"kernel": "spmv_short_rows_kernel" if half == 1 else "spmv_row_blocks_bulk_kernel", "diagonals": 2 * half + 1, "rows": n, "nnz": nnz,
               "ms": ours, **variants, "gbs": bytes_moved / ours / 1e6,
               f"frac_of_{src}_hbm": bytes_moved / ours / 1e6 / hbm, "cusparse_ms": lib, "speedup_vs_cusparse": lib / ours,
               "max_abs_diff_vs_cusparse": err, "working_set_mb": bytes_moved / 1e6, "fits_l2": bytes_moved < 126e6, "clocks": clocks}
        print(json.dumps(rec), flush=True)
        results.append(rec)
        m.close()
        del A, x, y, y2
    if args.out:
        with open(args.out, "w") as f:
            json.dump(results, f, indent=1)
    return 0


if __name__ == "__main__":
    sys.exit(main())
