"""The host thread teams of geometry creation and of the large host copies stay within the caller's
OpenMP setting: in a process with OMP_NUM_THREADS=1 no thread appears."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HEAD = """
import os, sys
sys.path.insert(0, {tests!r})
import conftest
bie = conftest.load_package()
import numpy as np
threads = lambda: len(os.listdir("/proc/self/task"))
itf = bie.single_dielectric_box3d(1.2, 0.8, 0.6, 4, 0.06, 4.0, 1.0)
assert itf.n > 16384
"""

# the sort of the direct sums' node order, called on its own (no device)
SORT = """
import ctypes as C
f = C.CDLL(sys.argv[1]).sort_slots
f.restype = C.c_int64
pts, nrm, w = (np.ascontiguousarray(a) for a in (itf.points, itf.normals, itf.weights))
room = 2 * itf.n
perm, planes = np.empty(room, np.int32), np.empty((room // 128 + 1, 3), np.int32)
before = threads()
assert f(*(C.c_void_p(a.ctypes.data) for a in (pts, nrm, w)), C.c_int64(itf.n), C.c_void_p(perm.ctypes.data),
         C.c_void_p(planes.ctypes.data), C.c_int64(room)) > 0
print("threads", before, threads())
"""

COPY = """
itf.geom(None, 0)
op = bie.lhs_dielectric_box3d(itf)
op @ np.ones((itf.n, 1), order="F")  # the driver's own threads
before = threads()
Y = op @ np.ones((itf.n, 32), order="F")  # 4 MB and more each way
assert itf.n * 32 * 8 > 4 << 20
print("threads", before, threads())
"""


def new_threads(body, *args):
    env = dict(os.environ, OMP_NUM_THREADS="1")
    out = subprocess.run([sys.executable, "-c", HEAD.format(tests=os.path.join(ROOT, "tests")) + body, *args], env=env,
                         check=True, capture_output=True, text=True, timeout=300).stdout
    before, after = map(int, out.split()[-2:])
    return after - before


def test_node_sort(bie, tmp_path):
    import test_sorted_nodes
    csrc = test_sorted_nodes.CSRC
    (tmp_path / "shim.cpp").write_text(test_sorted_nodes.SHIM)
    lib = str(tmp_path / "libsort.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fopenmp", "-I", csrc, str(tmp_path / "shim.cpp"),
                    os.path.join(csrc, "sorted_nodes.cpp"), "-o", lib], check=True)
    assert new_threads(SORT, lib) == 0


@pytest.mark.gpu
def test_host_copies(bie):
    assert new_threads(COPY) == 0
