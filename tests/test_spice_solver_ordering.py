"""The device solver against a stand-in for the CUDA runtime that is as asynchronous as the real one may be: a host-to-device copy
or a memset on the legacy stream is outstanding until somebody waits for that stream, and a kernel on a stream that does
not wait for the legacy one by itself must not be launched before. No GPU."""
import shutil
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent

RUNTIME = r"""
#include <stdlib.h>
#include <string.h>
#include <stddef.h>
typedef void* stream;
static int outstanding, launches;
static int is_legacy(stream s) { return s == NULL || s == (stream)1; }
int cudaGetDevice(int* d) { *d = 0; return 0; }
int cudaDeviceGetAttribute(int* v, int attr, int dev) { (void)dev; *v = attr == 16 ? 148 : 232448; return 0; }
int cudaFuncSetAttribute(const void* f, int a, int v) { (void)f; (void)a; (void)v; return 0; }
int cudaMalloc(void** p, size_t n) { *p = calloc(n ? n : 1, 1); return *p ? 0 : 2; }
int cudaFree(void* p) { free(p); return 0; }
int cudaMemcpy(void* d, const void* s, size_t n, int kind) { memcpy(d, s, n); if (kind == 1) outstanding = 1; else outstanding = 0; return 0; }
int cudaMemset(void* d, int v, size_t n) { memset(d, v, n); outstanding = 1; return 0; }
int cudaMemcpyAsync(void* d, const void* s, size_t n, int kind, stream st) { (void)kind; memcpy(d, s, n); if (is_legacy(st)) outstanding = 1; return 0; }
int cudaMemsetAsync(void* d, int v, size_t n, stream st) { memset(d, v, n); if (is_legacy(st)) outstanding = 1; return 0; }
int cudaStreamCreateWithFlags(stream* s, unsigned f) { *s = f & 1u ? (stream)0x1000 : (stream)0x2000; return 0; }
int cudaStreamDestroy(stream s) { (void)s; return 0; }
int cudaStreamSynchronize(stream s) { if (is_legacy(s) || s == (stream)0x2000) outstanding = 0; return 0; }
int cudaDeviceSynchronize(void) { outstanding = 0; return 0; }
int cudaGetLastError(void) { return 0; }
typedef struct { unsigned x, y, z; } dim;
int cudaLaunchCooperativeKernel(const void* f, dim g, dim b, void** a, size_t m, stream s) {
  (void)f; (void)g; (void)b; (void)a; (void)m;
  ++launches;
  return outstanding && s == (stream)0x1000 ? 999 : 0;
}
int solver_launches(void) { return launches; }
"""

DRIVER = r"""
import ctypes, sys
import numpy as np
sys.path.insert(0, sys.argv[2])
from nangila_spice.gpu import kernels_library, tridiagonal
lib = kernels_library()
count = ctypes.CDLL(sys.argv[1]).solver_launches
n = 5000
row_ptr, col, val = tridiagonal(n, 2.5)
b, x = np.ones(n), np.empty(n)
ctx = lib.nangila_spmv_create()
def solve():
    return lib.nangila_spmv_bicgstab(ctx, b.ctypes.data, x.ctypes.data, 1e-10, 10, None, None)
codes = []
for _ in range(2):  # a matrix, new values for it, another matrix
    assert lib.nangila_spmv_load(ctx, n, val.size, row_ptr.ctypes.data, col.ctypes.data, val.ctypes.data) == 0
    codes.append(solve())
    assert lib.nangila_spmv_update_values(ctx, val.ctypes.data) == 0
    codes += [solve(), solve()]
assert count() == 6, count()
print(codes)
assert all(c in (0, -1) for c in codes), codes
"""


@pytest.mark.skipif(shutil.which("gcc") is None, reason="needs a C compiler")
def test_uploads_have_landed_before_the_solver_kernel_is_queued(tmp_path):
    (tmp_path / "runtime.c").write_text(RUNTIME)
    so = tmp_path / "runtime.so"
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-o", str(so), str(tmp_path / "runtime.c")], check=True)
    proc = subprocess.run([sys.executable, "-c", DRIVER, str(so), str(ROOT)], capture_output=True, text=True, timeout=120,
                          env={"LD_PRELOAD": str(so), "PATH": "/usr/bin:/bin"})
    assert proc.returncode == 0, proc.stdout + proc.stderr
