"""cudaDeviceReset between two contexts, in a process of its own: it takes the
page-locked memory that results of the reductions are stored to with it, and the
kernels' attributes, so a context created afterwards must have its own."""
from __future__ import annotations

import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

PROGRAM = r"""
import ctypes as C, glob, os
import numpy as np
from cfdarcov2_b200 import capi
from cfdarcov2_b200.capi import call

def total(value, close):
    h, m, d, out = C.c_void_p(), C.c_void_p(), C.c_void_p(), C.c_double()
    call("cfdb_ctx_create", 0, C.byref(h))
    call("cfdb_mesh_create_structured", h, 10, 10, 10, 1.0, 1.0, 1.0, C.byref(m), ctx=h)
    f = np.full(1000, value, np.float64)
    call("cfdb_alloc", h, f.nbytes, C.byref(d), ctx=h)
    call("cfdb_upload", h, d, f.ctypes.data_as(C.c_void_p), f.nbytes, ctx=h)
    call("cfdb_total_fp64", h, m, capi.F64, d, C.byref(out), ctx=h)
    if close:
        capi.lib().cfdb_mesh_destroy(m)
        capi.lib().cfdb_ctx_destroy(h)
    return out.value

def heat(shape, steps):
    h, m, fb = C.c_void_p(), C.c_void_p(), C.c_int()
    call("cfdb_ctx_create", 0, C.byref(h))
    call("cfdb_mesh_create_structured", h, *shape, 0.01, 0.01, 0.01, C.byref(m), ctx=h)
    f = np.random.default_rng(1).uniform(-1, 1, shape).astype(np.float32)
    bufs = [C.c_void_p(), C.c_void_p()]
    for b in bufs:
        call("cfdb_alloc", h, f.nbytes, C.byref(b), ctx=h)
        call("cfdb_upload", h, b, f.ctypes.data_as(C.c_void_p), f.nbytes, ctx=h)
    call("cfdb_heat_run", h, m, capi.F32, capi.FUSED, *bufs, 0.01, 1e-4, steps, 1, C.byref(fb), ctx=h)
    call("cfdb_download", h, f.ctypes.data_as(C.c_void_p), bufs[fb.value], f.nbytes, ctx=h)
    capi.lib().cfdb_mesh_destroy(m)
    capi.lib().cfdb_ctx_destroy(h)
    return f

runs = [((64, 64, 64), 6), ((96, 24, 24), 40), ((128, 64, 64), 8), ((128, 64, 64), 9)]
before = [heat(*r) for r in runs]
assert total(2.0, True) == 2000.0
import torch
lib = glob.glob(os.path.join(os.path.dirname(torch.__file__), "..", "nvidia", "cuda_runtime", "lib", "libcudart.so*"))
cudart = C.CDLL(lib[0] if lib else "libcudart.so.12")
assert cudart.cudaSetDevice(0) == 0 and cudart.cudaDeviceReset() == 0
got = [total(3.0, True), total(4.0, False), total(5.0, True)]
assert got == [3000.0, 4000.0, 5000.0], got
for r, b in zip(runs, before):
    assert np.array_equal(heat(*r), b), r
print("ok")
"""


def test_contexts_around_a_device_reset():
    r = subprocess.run([sys.executable, "-c", PROGRAM], cwd=ROOT, env={**os.environ, "PYTHONPATH": ROOT},
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "ok" in r.stdout, r.stdout + r.stderr
