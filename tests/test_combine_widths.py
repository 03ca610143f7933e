"""The correction apply at the widths and panel counts where its forms change, against the sparse
matrix of the same blocks: 16-node panels (1 to 128 columns), 36-node panels few and many.

Tolerance: sums of at most 2,000 terms in FP64, 2,000 * 2^-53 = 2e-13 of their magnitudes (the
correction's and, for the difference that is taken, the full product's): 1e-12."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NO_CORRECTIONS = 1


@pytest.mark.parametrize("box, panels, widths", [
    ((1.0, 0.9, 0.7, 4, 0.25, 4.0, 1.0), 128, (1, 7, 8, 9, 16, 17, 24, 25, 64, 128)),
    ((0.7, 0.6, 0.5, 6, 0.2, 4.0, 1.0), 96, (1, 8, 9, 16, 17, 24, 25, 64, 65, 128)),
    ((1.1, 0.9, 0.6, 6, 0.12, 4.0, 1.0), 640, (1, 8, 16, 17, 19, 24, 25)),
    ((1.3, 0.9, 0.7, 6, 0.1, 3.0, 1.0), 904, (1, 15, 16, 17, 24)),
])
@pytest.mark.parametrize("precision", ["fp64", "bf16x3"])
def test_corrections_match_the_sparse_matrix(bie, rng, monkeypatch, box, panels, widths, precision):
    # one split of the direct sum in both products, so that their difference is the corrections alone
    monkeypatch.setenv("BIE_NO_AUTOTUNE", "1")
    itf = bie.single_dielectric_box3d(*box)
    assert itf.npanels == panels
    op = bie.lhs_dielectric_box3d_fmm3d_corrected(itf, 1e-12, 1e-9, 8)
    C = op.near.to_scipy()
    X = rng.standard_normal((itf.n, max(widths)))
    CX, S = C @ X, abs(C) @ np.abs(X)
    for k in widths:
        Xk = np.asfortranarray(X[:, :k])
        Y = op.mul(Xk, precision=precision)
        got = Y - op.mul(Xk, precision=precision, flags=NO_CORRECTIONS)
        assert np.all(np.abs(got - CX[:, :k]) < 1e-12 * (S[:, :k] + np.abs(Y))), k
