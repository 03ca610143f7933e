"""The correction apply in tiles of 32 and 64 columns: the rule (csrc/combine_tile.h) on the CPU, and both
tiles against the sparse matrix of the same blocks, at panels of 4 to 64 nodes.

Tolerance: sums of at most 2,000 terms in FP64, 2,000 * 2^-53 = 2e-13 of their magnitudes (the
correction's and, for the difference that is taken, the full product's): 1e-12."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dielectricbie.jl_b200", "csrc")
NO_CORRECTIONS = 1


@pytest.fixture(scope="module")
def tile(tmp_path_factory):
    d = tmp_path_factory.mktemp("tile")
    (d / "shim.cpp").write_text('#include "combine_tile.h"\n'
                                'extern "C" int tile(int nb, int k, int p, int s) { return bie::combine_tile(nb, k, p, s); }')
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I", CSRC, str(d / "shim.cpp"), "-o",
                    str(d / "libtile.so")], check=True)
    return C.CDLL(str(d / "libtile.so")).tile


@pytest.mark.parametrize("nb", [4, 9, 25, 36, 49, 64])
@pytest.mark.parametrize("panels", [96, 728, 1776, 3000])
def test_rule(tile, nb, panels):
    for k in range(1, 300):
        ct = tile(nb, k, panels, 148)
        if k < 64:
            assert ct == 32
        elif k == 64:
            assert ct == (64 if panels >= 1776 else 32)
        elif (k - 1) % 64 >= 32:  # the last 64-column tile is more than half full
            assert ct == 64
        else:  # three tiles of 32 or two of 64: 64 only where they do not cost warps in flight
            assert ct == (64 if nb in (25, 36, 49) else 32), k


@pytest.mark.gpu
@pytest.mark.parametrize("box", [(1.0, 0.9, 0.7, 2, 0.04, 4.0, 1.0), (1.0, 0.9, 0.7, 3, 0.2, 4.0, 1.0),
                                 (1.0, 0.9, 0.7, 5, 0.25, 4.0, 1.0), (0.7, 0.6, 0.5, 7, 0.25, 4.0, 1.0),
                                 (0.7, 0.6, 0.5, 8, 0.25, 4.0, 1.0)])
def test_corrections_match_the_sparse_matrix(bie, rng, monkeypatch, box):
    monkeypatch.setenv("BIE_NO_AUTOTUNE", "1")
    itf = bie.single_dielectric_box3d(*box)
    assert box[3] > 2 or itf.npanels >= 12 * 148  # 64 columns in one tile
    op = bie.lhs_dielectric_box3d_fmm3d_corrected(itf, 1e-12, 1e-9, 8)
    Cm = op.near.to_scipy()
    X = rng.standard_normal((itf.n, 129))
    CX, S = Cm @ X, abs(Cm) @ np.abs(X)
    for k in (33, 63, 64, 65, 80, 96, 97, 128, 129):
        Xk = np.asfortranarray(X[:, :k])
        Y = op.mul(Xk, precision="bf16x3")
        got = Y - op.mul(Xk, precision="bf16x3", flags=NO_CORRECTIONS)
        assert np.all(np.abs(got - CX[:, :k]) < 1e-12 * (S[:, :k] + np.abs(Y))), k
