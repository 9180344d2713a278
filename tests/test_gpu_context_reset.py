"""GPU: trees made after the device's context was reset, and by threads that make their first CUDA call with one.

In a process of its own: builds through every kind of call, a reset of the context
with no tree alive (the caller holds nothing of the library then), and the same
builds again, twice.  The edges have to be the same each time and no launch may be
refused, the first-point block's (which needs a kernel attribute) among them.
"""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CHILD = r"""
import ctypes
import numpy as np
import voronoids_gb300 as V
from voronoids_gb300 import _native

L = _native.load()
rt = ctypes.CDLL("libcudart.so.13")  # the runtime that the library has loaded
rng = np.random.default_rng(3)
pts = {dim: rng.random((3000, dim)) for dim in (2, 3)}


def builds():
    out = []
    for dim, p in pts.items():
        t = V.delaunay(p, seed=1)
        out.append(t.edges())
        assert t.check_delaunay()
        t.insert_point(np.full(dim, 0.4375))
        out.append(t.edges())
        t.close()
        out += V.delaunay_batch([p[:500], p[500:1700]], seed=2)
        uv, m = np.zeros((30000, 2), np.int64), ctypes.c_int64(0)
        rc = L.vd_delaunay(dim, p.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), len(p), 1,
                           uv.ctypes.data_as(ctypes.POINTER(ctypes.c_int64)), len(uv), ctypes.byref(m))
        assert rc == 0, rc
        out.append(uv[:m.value])
    assert rt.cudaGetLastError() == 0
    return out


first = builds()
for _ in range(2):
    assert rt.cudaDeviceReset() == 0
    for a, b in zip(first, builds()):
        assert np.array_equal(a, b)
print("same edges")
"""


def test_builds_after_a_context_reset():
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "same edges" in r.stdout, r.stdout + r.stderr


def test_first_call_of_a_thread(vd, oracle):
    import threading

    from voronoids_gb300 import workloads as W
    p = W.uniform_points(4000, 3, 71)
    want = oracle.Triangulation(p, seed=1).edges()
    good = []

    def build():
        t = vd.delaunay(p, seed=1)
        good.append((t.edges() == want).all())
        t.close()

    for _ in range(3):  # blocks that one thread gives back are another's
        threads = [threading.Thread(target=build) for _ in range(4)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    assert good == [True] * 12
