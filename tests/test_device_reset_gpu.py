"""Assembly after the device's primary context has been reset and created anew
in the same process and thread (include/pq3d.h allows it between calls of the
allocation-free entry): the launch attributes and addresses of the first context
are not taken for the second's.  In a process of its own, through the C ABI and
the driver API, with nothing in flight at the reset."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CHILD = """
import ctypes as C
import numpy as np
from pyquake3d_gb300 import _lib, mesh
cu = C.CDLL("libcuda.so.1")
def ok(rc, what):
    assert rc == 0, (what, rc)
ok(cu.cuInit(0), "init")
ctx = C.c_void_p()
def up():
    ok(cu.cuDevicePrimaryCtxRetain(C.byref(ctx), 0), "retain")
    ok(cu.cuCtxSetCurrent(ctx), "current")
def dev(nbytes, host=None):
    p = C.c_uint64()
    ok(cu.cuMemAlloc_v2(C.byref(p), C.c_size_t(nbytes)), "alloc")
    if host is not None:
        ok(cu.cuMemcpyHtoD_v2(p, C.c_void_p(host.ctypes.data), C.c_size_t(nbytes)), "in")
    return p.value
L = _lib.load()
mu = 32038120320.0
nodes, tris = mesh.rough_fault(16.0, 8.0, 16, 10, seed=5, ratio=5e-3)
nodes = np.ascontiguousarray(nodes - [0.0, 0.0, nodes[:, 2].max() + 500.0])
tris = np.ascontiguousarray(tris, dtype=np.int64)
N = len(tris)
def run():
    up()
    n, t, k, w = dev(nodes.nbytes, nodes), dev(tris.nbytes, tris), dev(48 * N * N), dev(L.pq3d_gf_workspace_bytes(N))
    out = []
    for half in (None, 0, 1):
        if half is None:
            rc = L.pq3d_assemble_dense_noalloc(n, t, N, 0, N, mu, mu, 0, k, None, None)
        else:
            rc = L.pq3d_assemble_dense(n, t, N, 0, N, mu, mu, half, k, None, w, L.pq3d_gf_workspace_bytes(N), None)
        assert rc == 0, L.pq3d_last_error()
        K = np.full((3 * N, 2 * N), np.nan)
        ok(cu.cuCtxSynchronize(), "wait")
        ok(cu.cuMemcpyDtoH_v2(C.c_void_p(K.ctypes.data), C.c_uint64(k), C.c_size_t(K.nbytes)), "out")
        out.append(K)
    return out
first = run()
ok(cu.cuDevicePrimaryCtxReset_v2(0), "reset")
second = run()
for a, b in zip(first, second):
    assert np.isfinite(a).all() and np.array_equal(a, b)
print("same")
"""


def test_assembly_after_a_device_reset(cuda):
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=REPO, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "same", r.stdout + r.stderr
