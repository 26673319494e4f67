"""The C entry points in a second context of the same device, and after the context that they first ran in is gone: the shared
memory limit of a kernel belongs to a context.  In a process of its own, with memory from the runtime; each call checks its launches and waits."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = r"""
import ctypes as C, sys
from openkimi_b200 import _lib

lib = _lib.load()
rt, cu = C.CDLL("libcudart.so.12"), C.CDLL("libcuda.so.1")

def call(what):
    p = _lib.KdaParams(B=1, T=64, H=1, dk=128, dv=128, N=1, NT=1, dtype=_lib.DTYPE_BF16, scale=1.0, guard_span=232.0)
    fwd, bwd, held = C.c_size_t(), C.c_size_t(), []
    assert lib.kda_workspace_bytes(C.byref(p), C.byref(fwd), C.byref(bwd)) == 0
    def mem(n):
        x = C.c_void_p()
        assert rt.cudaMalloc(C.byref(x), C.c_size_t(n)) == 0 and rt.cudaMemset(x, 0, C.c_size_t(n)) == 0
        held.append(x)
        return x.value
    for n in ("q", "k", "v", "g", "beta", "o", "grad_o", "grad_q", "grad_k", "grad_v", "grad_g", "grad_beta", "status"):
        setattr(p, n, mem(64 * 128 * 2))
    p.workspace, p.workspace_bytes, p.bwd_scratch, p.bwd_scratch_bytes = mem(fwd.value), fwd.value, mem(bwd.value), bwd.value
    for fn in (lib.kda_fwd, lib.kda_bwd):
        rc = fn(C.byref(p), None)
        assert rc == 0, (what, fn.__name__, rc, lib.kda_last_cuda_error())
        assert rt.cudaDeviceSynchronize() == 0
    for x in held:
        assert rt.cudaFree(x) == 0

assert rt.cudaFree(None) == 0
call("first context")
call("first context again")
other = C.c_void_p()
assert cu.cuCtxCreate_v2(C.byref(other), 0, 0) == 0
call("second context")
assert cu.cuCtxDestroy_v2(other) == 0
call("first context after the second")
assert rt.cudaDeviceReset() == 0
call("after a reset")
print("done")
"""


def test_every_context_gets_its_shared_memory_limits():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "done" in r.stdout, r.stderr[-2000:]
