"""A device whose context is destroyed and created again (cudaDeviceReset): what
the library keeps per context -- scratch pools, kernels' shared-memory limits --
is made again, so that calls work as in a new process.  In a child process: the
reset ends everything else that the process has on the GPU."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r'''
import ctypes as C, sys
import numpy as np
import torch  # loads the CUDA runtime whose calls are used below
sys.path.insert(0, "distributed-ranges_b200")
from drb import _capi as capi
import drb
rt = C.CDLL("libcudart.so.12")
vp = C.c_void_p

def dev(a):
    p = vp()
    assert rt.cudaMalloc(C.byref(p), C.c_size_t(max(a.nbytes, 16))) == 0
    assert rt.cudaMemcpy(p, a.ctypes.data_as(vp), C.c_size_t(a.nbytes), 1) == 0
    return p

def host(p, like):
    a = np.empty_like(like)
    assert rt.cudaMemcpy(a.ctypes.data_as(vp), p, C.c_size_t(a.nbytes), 2) == 0
    return a

def dense(m, n, k):
    g = np.random.default_rng(1)
    A, x = g.standard_normal((m, n)).astype(np.float32), g.standard_normal((k, n)).astype(np.float32)
    y = dev(np.zeros((k, m), np.float32))
    capi.check(capi.lib.drb_dense_gemv(m, n, dev(A), n, dev(x), y, k, 0, capi.DRB_F32, None))
    err = np.abs(host(y, np.zeros((k, m), np.float32)) - x @ A.T).max()
    assert err < (n + 8) * 2.0 ** -24 * (np.abs(x) @ np.abs(A.T)).max(), err

def dot(n):
    a = np.random.default_rng(2).standard_normal(n)
    out = dev(np.zeros(1))
    d = dev(a)
    capi.check(capi.lib.drb_dot(n, d, d, capi.DRB_F64, out, None))
    assert abs(host(out, np.zeros(1))[0] - a @ a) < 1e-12 * n

def cg(g):
    rp, ci, v = drb.gen.laplacian2d_csr(g)
    m = g * g
    h = vp()
    capi.check(capi.lib.drb_csr_create(C.byref(h), m, m, len(v), rp.ctypes.data_as(vp),
                                       ci.ctypes.data_as(vp), v.ctypes.data_as(vp), capi.DRB_I32,
                                       capi.DRB_F64, capi.DRB_F64, 1, 0, 0, None))
    x = dev(np.zeros(m))
    info = capi.CgInfo()
    capi.check(capi.lib.drb_csr_cg(h, dev(np.ones(m)), x, 2000, C.c_double(1e-8), C.byref(info),
                                   None))
    assert info.converged
    capi.check(capi.lib.drb_csr_destroy(h))

def all_of_them():
    dense(300, 1000, 1), dense(5, 400_000, 1), dense(5003, 301, 3), dense(2000, 1000, 20)
    dot(100_000), cg(64)

all_of_them()
assert rt.cudaDeviceReset() == 0
all_of_them()
print("both contexts done")
'''


def test_calls_after_a_device_reset():
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, capture_output=True, text=True,
                       timeout=240)
    assert r.returncode == 0 and "both contexts done" in r.stdout, r.stdout + r.stderr
