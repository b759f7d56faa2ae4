"""Calls that take their scratch memory from the library's kept pool, before and after the host
program resets its device (which ends the context and the pool with it).  In a process of its own."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
import ctypes as C, sys
import numpy as np
sys.path.insert(0, sys.argv[1])
from myfluidsimulation_b200 import geometry as G, lib, vtk, workloads as W
lib()
rt = C.CDLL("libcudart.so.12")      # the one the library is linked to

def masks():
    mesh = G.mesh_from_triangles(W.icosphere(2).astype(np.float32))
    return [G.voxelize_mesh_to_mask(mesh, G.VoxelParams(40, 30, 20, 0.7, (0.5, 0.5, 0.5), r, 0.5)) for r in (1, 2)]

def text():
    n = 1000
    v = np.linspace(-1, 1, n).astype(np.float32)
    cap = lib().lbm_vtk_text_bound(vtk.VTK_SCALAR, C.c_int64(n))
    d, t = C.c_void_p(), C.c_void_p()
    assert rt.cudaMalloc(C.byref(d), C.c_size_t(4 * n)) == 0 and rt.cudaMalloc(C.byref(t), C.c_size_t(cap)) == 0
    assert rt.cudaMemcpy(d, v.ctypes.data_as(C.c_void_p), C.c_size_t(4 * n), 1) == 0
    m = C.c_int64()
    assert lib().lbm_vtk_format(vtk.VTK_SCALAR, d, None, None, C.c_int64(n), t, C.c_int64(cap), C.byref(m), None) == 0
    out = np.zeros(m.value, np.uint8)
    assert rt.cudaMemcpy(out.ctypes.data_as(C.c_void_p), t, C.c_size_t(m.value), 2) == 0
    return out.tobytes()

a, b = masks(), text()
assert rt.cudaDeviceReset() == 0
c, d = masks(), text()
assert all(np.array_equal(x, y) for x, y in zip(a, c)) and a[0].any() and b == d and len(b) > 2000
assert rt.cudaDeviceReset() == 0
assert text() == b and np.array_equal(masks()[1], a[1])
print("same")
"""


def test_scratch_pool_after_a_device_reset(gpu):
    r = subprocess.run([sys.executable, "-c", PROGRAM, ROOT], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "same", r.stdout + r.stderr
