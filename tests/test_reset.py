"""The primitives after the primary context was torn down and made again (what
a device reset does): a kernel's limits are attributes of its context."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = r"""
import ctypes, sys
from libnegf_b200 import native
cu = ctypes.CDLL("libcuda.so.1")
def ok(rc):
    assert rc == 0, rc
ok(cu.cuInit(0))
L = native.load()
n, batch = 96, 2
one, zero = (ctypes.c_double * 2)(1, 0), (ctypes.c_double * 2)(0, 0)
def run():
    ctx = ctypes.c_void_p()
    ok(cu.cuDevicePrimaryCtxRetain(ctypes.byref(ctx), 0))
    ok(cu.cuCtxSetCurrent(ctx))
    def mem(nbytes):
        p = ctypes.c_uint64()
        ok(cu.cuMemAlloc_v2(ctypes.byref(p), ctypes.c_size_t(nbytes)))
        return p.value
    N = batch * n * n
    host = (ctypes.c_double * (2 * N))()
    for b in range(batch):
        for i in range(n):
            host[2 * (b * n * n + i * n + i)] = 2.0 + b + i
    a, x, y = mem(16 * N), mem(16 * N), mem(16 * N)
    ok(cu.cuMemcpyHtoD_v2(ctypes.c_uint64(a), host, ctypes.c_size_t(16 * N)))
    D = lambda p: ctypes.cast(p, ctypes.POINTER(ctypes.c_double))
    I = lambda p: ctypes.cast(p, ctypes.POINTER(ctypes.c_int32))
    w = mem(max(L.negf_b200_zinv_work_bytes(batch, n), L.negf_b200_decimation_work_bytes(batch, n),
                L.negf_b200_zgemm_i8_work_bytes(batch, n, n, n, 8)))
    info = mem(64)
    V = ctypes.c_void_p
    rcs = [L.negf_b200_zinv_batched(batch, n, D(a), D(x), I(info), V(w), None),
           L.negf_b200_zgemm_batched(batch, n, n, n, one, D(a), 2 * n * n, D(x), 2 * n * n, zero, D(y), 2 * n * n, 0,
                                     None)]
    out = (ctypes.c_double * (2 * N))()
    ok(cu.cuMemcpyDtoH_v2(out, ctypes.c_uint64(y), ctypes.c_size_t(16 * N)))
    good = all(abs(out[2 * (b * n * n + i * n + i)] - 1.0) < 1e-12 for b in range(batch) for i in range(n))
    rcs.append(L.negf_b200_zgemm_batched_i8(batch, n, n, n, one, D(a), 2 * n * n, D(x), 2 * n * n, zero, D(y),
                                            2 * n * n, 8, V(w), None, None))
    rcs.append(L.negf_b200_decimation_batched(batch, n, D(a), D(x), D(x), D(y), I(info), 1e-9, 50, V(w), None))
    ok(cu.cuCtxSynchronize())
    return rcs, good
for k in range(2):
    rcs, good = run()
    print(k, rcs, good, flush=True)
    assert good and not any(rcs)
    ok(cu.cuDevicePrimaryCtxRelease_v2(0))
    ok(cu.cuDevicePrimaryCtxReset_v2(0))
"""


def test_primitives_run_after_their_context_was_made_again():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
