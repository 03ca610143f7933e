"""A surface with all nodes in one plane of the sorted order, so that no target has a source left: exact
zeros in every precision and width, whatever the workspace held before."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NO_DIAGONAL = 2


@pytest.mark.parametrize("panels", [(4, 4), (5, 4), (9, 7)])  # 256 nodes: the smallest plane; padded ones
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_one_plane_sums_to_zero(bie, rng, panels, axis):
    x, w = bie.gausslegendre(4)
    nrm = np.roll([1.0, 0.0, 0.0], axis)
    at = lambda i, j: np.roll([0.25, i / 8, j / 8], axis)
    flat = [bie.rect_panel3d_discretize(at(i, j), at(i + 1, j), at(i + 1, j + 1), at(i, j + 1), x, w,
                                        nrm if (i + j) % 2 else -nrm)
            for i in range(panels[0]) for j in range(panels[1])]
    itf = bie.DielectricInterface(flat, 4.0, 1.0)
    assert itf.n == 16 * panels[0] * panels[1] >= 256
    op = bie.lhs_dielectric_box3d(itf)
    X = rng.standard_normal((itf.n, 130))
    fill = bie.laplace3d_pottrg(itf, rng.uniform(2.0, 3.0, (4000, 3)))
    for precision, widths in (("fp64", (1, 3, 8, 16, 33, 65)), ("fp32", (1, 2, 8)),
                              ("bf16x3", (8, 17, 64, 130)), ("bf16x6", (8, 33, 70, 130))):
        for k in widths:
            assert np.all((fill @ np.asfortranarray(X))[0] != 0.0)  # the same geometry's partial sums
            Xk = np.asfortranarray(X[:, :k])
            assert np.all(op.mul(Xk, precision=precision, flags=NO_DIAGONAL) == 0.0), (precision, k)
            got = op.mul(Xk, precision=precision)
            assert np.allclose(got, itf.diag[:, None] * Xk, rtol=1e-15, atol=0.0), (precision, k)
