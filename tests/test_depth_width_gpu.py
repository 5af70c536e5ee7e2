"""A level count that is too low for the depths costs a copy, never a wrong
result or an error: arrays on both sides of the size up to which the packed
depths go straight to pinned memory, returned by the library's own routine with
a wrong count, on a handle that has returned nothing else.  In a process of its
own, because an exception would end the caller."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CODE = """
import ctypes as C, sys
import numpy as np
import graph_analytics_applesilicon_b200 as gb
n, claimed = int(sys.argv[1]), int(sys.argv[2])
g = gb.gen.path(n)
bfs = gb.GpuBfs(g)
bfs.run_many("gpu_do_persistent", np.array([n - 700], np.uint32), device=True)  # depths to n - 700
L = gb.lib()
f = getattr(L, "_ZN2gb16copyDepthsToHostEP6gb_bfsPKjmPjj")
f.argtypes = [C.c_void_p, C.c_void_p, C.c_uint64, C.c_void_p, C.c_uint32]
out = np.zeros(n, np.uint32)
for k in (claimed, n, claimed):
    out[:] = 5
    f(bfs._h, L.gb_bfs_device_dist(bfs._h), n, out.ctypes.data, k)
    assert np.array_equal(out, np.abs(np.arange(n, dtype=np.int64) - (n - 700)).astype(np.uint32)), k
print("ok")
"""


@pytest.mark.parametrize("n,claimed", [(1000, 3), (1000, 14), (3000, 254), (70000, 20), (70000, 300), (1100000, 254)])
def test_too_low_a_count(n, claimed):
    r = subprocess.run([sys.executable, "-c", CODE, str(n), str(claimed)], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stderr[-2000:]
