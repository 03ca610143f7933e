"""The sort of a geometry's nodes into the order of the direct sums (csrc/sorted_nodes.cpp), compiled
on its own and called on the CPU."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "dielectricbie.jl_b200", "csrc")
TILE = 128

SHIM = """
#include <algorithm>
#include "sorted_nodes.h"
extern "C" int64_t sort_slots(const double* pts, const double* nrm, const double* w, int64_t n, int32_t* perm,
                              int32_t* planes, int64_t room) {
    const bie::SortedNodes so = bie::sort_nodes(pts, nrm, w, n);
    if ((int64_t)so.perm.size() > room) return -1;
    std::copy(so.perm.begin(), so.perm.end(), perm);
    for (size_t t = 0; t < so.tiles.size(); ++t) {
        planes[3 * t] = so.tiles[t].axis;
        planes[3 * t + 1] = so.tiles[t].s0;
        planes[3 * t + 2] = so.tiles[t].s1;
    }
    return (int64_t)so.perm.size();
}
"""


@pytest.fixture(scope="module")
def sort(tmp_path_factory):
    d = tmp_path_factory.mktemp("sort")
    (d / "shim.cpp").write_text(SHIM)
    lib = str(d / "libsort.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fopenmp", "-I", CSRC, str(d / "shim.cpp"),
                    os.path.join(CSRC, "sorted_nodes.cpp"), "-o", lib], check=True)
    f = C.CDLL(lib).sort_slots
    f.restype = C.c_int64

    def call(pts, nrm):
        pts, nrm = np.ascontiguousarray(pts), np.ascontiguousarray(nrm)
        n = len(pts)
        w, room = np.ones(n), 2 * n + TILE
        perm, planes = np.empty(room, np.int32), np.empty((room // TILE + 1, 3), np.int32)
        ns = f(*(C.c_void_p(a.ctypes.data) for a in (pts, nrm, w)), C.c_int64(n), C.c_void_p(perm.ctypes.data),
               C.c_void_p(planes.ctypes.data), C.c_int64(room))
        assert ns > 0 and ns % TILE == 0
        return perm[:ns], planes[:ns // TILE]

    return call


def bisected(pts, idx):
    """Whether idx is bisected across the longest side at whole tiles, numbers before not-a-numbers."""
    if len(idx) <= TILE:
        return bool(np.all(np.diff(idx) > 0))
    p = pts[idx]
    with np.errstate(invalid="ignore"):
        lo = np.where(np.isnan(p), np.inf, p).min(0)
        hi = np.where(np.isnan(p), -np.inf, p).max(0)
        ext = hi - lo
    ax = 0
    for c in (1, 2):
        if ext[c] > ext[ax]:
            ax = c
    half = -(-len(idx) // TILE) // 2 * TILE
    key = [(np.isnan(v), 0.0 if np.isnan(v) else v, i) for v, i in zip(p[:, ax], idx)]
    return max(key[:half]) < min(key[half:]) and bisected(pts, idx[:half]) and bisected(pts, idx[half:])


@pytest.mark.parametrize("special", [(), (np.nan,), (np.inf, -np.inf), (np.nan, np.inf, -np.inf)])
@pytest.mark.parametrize("n", [1, 127, 129, 1000, 20000])
def test_order_with_coordinates_that_are_no_numbers(sort, n, special):
    rng = np.random.default_rng(n + len(special))
    pts = rng.uniform(-1.0, 1.0, (n, 3))
    pts[rng.integers(0, n, n // 4), 2] = 0.25  # ties
    for v in special:
        pts[rng.integers(0, n, max(1, n // 10)), rng.integers(0, 3, max(1, n // 10))] = v
    nrm = np.full((n, 3), 1 / np.sqrt(3.0))  # no coordinate planes: one group
    perm, planes = sort(pts, nrm)
    assert np.all(planes[:, 0] == 3)
    assert np.array_equal(np.sort(perm[:n]), np.arange(n)) and np.all(perm[n:] == -1)
    assert bisected(pts, perm[:n])
