"""Kernel attributes (the shared-memory limits) belong to a context on a device: what one process raised for its
first context says nothing about another one. Run in a process of its own: flat meshes and a batch whose rings
need more than the default limit, in the primary context and then in a second one."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

SCRIPT = """
import ctypes as C, sys
import numpy as np
sys.path.insert(0, {root!r})
import volumesurfacediscretemeshoptimization_b200 as V

def fan(n):
    a = 2 * np.pi * np.arange(n) / n
    xyz = np.stack([np.cos(a), np.sin(a), 0 * a], 1)
    j = np.arange(n)
    return (np.concatenate([[[0.3, 0.1, 0]], xyz]).astype(np.float32), np.stack([0 * j, 1 + j, 1 + (j + 1) % n], 1).astype(np.int32))

def run():
    out = []
    for valence in (12, 16, 60):
        xyz, el = fan(valence)
        b = V.BatchDMO([(0, xyz, el)])
        b.iterate(2)
        out.append(b.positions())
        b.close()
        m = V.DMOMeshTri(xyz, el)
        o = V.DMOTriFlatClass(m, n_iter=2, grid_n=4)
        o.iterate(2)
        out.append(m.positions())
        o.close()
        m.close()
    return out

first = run()
cu = C.CDLL("libcuda.so.1")
dev, ctx = C.c_int(), C.c_void_p()
assert cu.cuInit(0) == 0 and cu.cuDeviceGet(C.byref(dev), 0) == 0
assert cu.cuCtxCreate_v2(C.byref(ctx), 0, dev) == 0
second = run()
assert all(np.array_equal(a, b) for a, b in zip(first, second))
assert not np.array_equal(first[0][0], fan(12)[0][0])
print("same")
"""


def test_flat_kernels_in_a_second_context(vsdmo):
    import os
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", SCRIPT.format(root=root)], capture_output=True, text=True, timeout=200)
    assert r.returncode == 0 and "same" in r.stdout, r.stdout + r.stderr
