"""Large pageable host arrays (staged through pinned pieces of 512 KB from 2 MB on) against the same call
on pinned arrays, which the driver copies directly: every width around the pieces' edges, bit for bit."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [102, 103, 104, 128, 129, 153, 154, 231, 256, 257])
def test_pageable_equals_pinned(bie, rng, monkeypatch, k):
    monkeypatch.setenv("BIE_NO_AUTOTUNE", "1")
    import torch
    from dielectricbie_jl_b200 import _abi
    itf = bie.single_dielectric_box3d(1.2, 0.8, 0.6, 4, 0.2, 4.0, 1.0)  # 2,560 nodes: 20,480 bytes a column
    op = bie.lhs_dielectric_box3d(itf)
    X = np.asfortranarray(rng.standard_normal((itf.n, k)))
    Y = op @ X
    xp = torch.from_numpy(np.ascontiguousarray(X.T)).pin_memory()
    yp = torch.empty_like(xp).pin_memory()
    assert xp.is_pinned() and yp.is_pinned()
    ptr = lambda t: C.cast(t.data_ptr(), C.POINTER(C.c_double))
    _abi.check(_abi.lib().bie_matvec(op.geom._h, ptr(xp), ptr(yp), k, 0, 0))
    assert np.array_equal(Y, yp.numpy().T)
    # and with a base that is no multiple of a piece or a page
    room = np.zeros(X.size + 3)
    odd = room[3:].reshape(k, itf.n).T
    odd[:] = X
    assert np.array_equal(op @ odd, Y)
