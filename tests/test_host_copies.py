"""Host arrays large enough for the staged copies (2 MB), at sizes around their pieces (512 KB dealt to
four threads), from several threads at once and next to pinned arrays: every byte arrives, so the
results equal those of the same call on narrower blocks and on pinned memory bit for bit."""
import ctypes as C
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_staged_copies_of_odd_sizes_and_threads(bie, rng, monkeypatch):
    monkeypatch.setenv("BIE_NO_AUTOTUNE", "1")
    import torch
    from dielectricbie_jl_b200 import _abi
    itf = bie.single_dielectric_box3d(1.2, 0.8, 0.6, 4, 0.2, 4.0, 1.0)  # 2,560 nodes: 20,480 bytes a column
    rows = lambda X: bie.laplace3d_pottrg(itf, np.array([[2.0, 0.0, 0.0], [0.0, 3.0, 0.1]])) @ X
    X = np.asfortranarray(rng.standard_normal((itf.n, 420)))
    # 103 columns are just above 2 MB, 128 a whole number of pieces, 420 many rounds of every thread
    for k in (102, 103, 128, 129, 231, 420):
        assert np.array_equal(rows(np.asfortranarray(X[:, :k])), rows(np.asfortranarray(X[:, :k]))), k
        F = bie.rhs_dielectric_box3d(itf, [bie.PointSource(tuple(0.2 * rng.uniform(-1, 1, 3)), 1.0)] * k, 4.0)
        assert np.array_equal(F, np.repeat(F[:, :1], k, axis=1)), k
    op = bie.lhs_dielectric_box3d(itf)
    Y = op @ X
    xp = torch.from_numpy(np.ascontiguousarray(X.T)).pin_memory()
    yp = torch.empty_like(xp).pin_memory()
    ptr = lambda t: C.cast(t.data_ptr(), C.POINTER(C.c_double))
    _abi.check(_abi.lib().bie_matvec(op.geom._h, ptr(xp), ptr(yp), 420, 0, 0))
    assert np.array_equal(Y, yp.numpy().T)
    # several threads, each with a geometry of its own
    got = [None] * 6
    itfs = [bie.single_dielectric_box3d(1.2, 0.8, 0.6, 4, 0.2, 4.0, 1.0) for _ in got]

    def work(i):
        o = bie.lhs_dielectric_box3d(itfs[i])
        got[i] = [o @ X for _ in range(3)][-1]

    ts = [threading.Thread(target=work, args=(i,)) for i in range(len(got))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for g in got:
        assert np.array_equal(g, Y)
