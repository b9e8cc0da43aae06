"""Factorisations after the device's context was destroyed and made anew (cudaDeviceReset): with a workspace of the caller's,
and tnc_svd_noalloc, whose scratch array has another address then.  In a process of its own, without PyTorch."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = r"""
import ctypes as C, sys
import numpy as np
lib = C.CDLL(sys.argv[1])
rt = C.CDLL("libcudart.so.13")
vp, i64 = C.c_void_p, C.c_int64
noalloc = sys.argv[2] == "noalloc"
lib.tnc_svd_noalloc.argtypes = [C.c_int, i64, i64, vp, i64, vp, vp, vp, C.c_int, C.c_double, vp, vp]
lib.tnc_svd.argtypes = [C.c_int, i64, i64, vp, i64, vp, vp, vp, C.c_int, C.c_double, vp, C.c_size_t, vp, vp]
lib.tnc_svd_workspace_size.argtypes = [C.c_int, i64, i64, C.POINTER(C.c_size_t)]
rt.cudaMalloc.argtypes = [C.POINTER(vp), C.c_size_t]
rt.cudaMemcpy.argtypes = [vp, vp, C.c_size_t, C.c_int]

def alloc(n):
    p = vp()
    assert rt.cudaMalloc(C.byref(p), n) == 0
    return p

def once(code, dt):
    rng = np.random.default_rng(code)
    a = rng.standard_normal((96, 96))
    if np.issubdtype(dt, np.complexfloating):
        a = a + 1j * rng.standard_normal((96, 96))
    a = np.ascontiguousarray(a.astype(dt))
    A, U, S, V, info = (alloc(n) for n in (a.nbytes, a.nbytes, 96 * 8, a.nbytes, 16))
    assert rt.cudaMemcpy(A, a.ctypes.data_as(vp), a.nbytes, 1) == 0
    if noalloc:
        st = lib.tnc_svd_noalloc(code, 96, 96, A, 96, U, S, V, 0, 0.0, info, None)
    else:
        b = C.c_size_t()
        assert lib.tnc_svd_workspace_size(code, 96, 96, C.byref(b)) == 0
        st = lib.tnc_svd(code, 96, 96, A, 96, U, S, V, 0, 0.0, alloc(b.value), b.value, info, None)
    assert st == 0, ("status", code, st)
    assert rt.cudaDeviceSynchronize() == 0
    s, h = np.empty(96, np.finfo(dt).dtype), np.empty(4, np.int32)
    assert rt.cudaMemcpy(s.ctypes.data_as(vp), S, s.nbytes, 2) == 0
    assert rt.cudaMemcpy(h.ctypes.data_as(vp), info, 16, 2) == 0
    ref = np.linalg.svd(a, compute_uv=False)
    assert h[0] == 0 and np.max(np.abs(s - ref)) <= 800 * np.finfo(dt).eps * ref[0], (code, h)

types = [(0, np.float32), (1, np.float64), (2, np.complex64), (3, np.complex128)]
for _ in range(3):
    for code, dt in types:
        once(code, dt)
    assert rt.cudaDeviceSynchronize() == 0
    assert rt.cudaDeviceReset() == 0
print("same results after a reset")
"""


@pytest.mark.parametrize("kind", ["workspace", "noalloc"])
def test_svd_after_reset(gpu, kind):
    from tncontract_gb300 import _build
    r = subprocess.run([sys.executable, "-c", CHILD, _build.LIBPATH, kind], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "same results" in r.stdout, r.stdout + r.stderr
