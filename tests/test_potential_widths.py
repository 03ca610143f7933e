"""Single-layer potentials around the edges of their kernels (8, 16, 32 and 64 columns a pass, 32 to 128
targets a tile, source counts that are no multiple of a tile), against the dense sum in numpy.

Tolerance: sums of at most 2,560 positive-kernel terms in FP64, 2,560 * 2^-53 = 3e-13 of their
magnitudes at worst: 1e-12."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("box", [(1.2, 0.8, 0.6, 4, 0.2, 4.0, 1.0), (0.7, 0.6, 0.5, 3, 0.3, 4.0, 1.0)])
@pytest.mark.parametrize("targets", [1, 63, 64, 129, 1000])
def test_potentials_match_the_dense_sum(bie, rng, box, targets):
    itf = bie.single_dielectric_box3d(*box)
    T = rng.uniform(-1.0, 1.0, (targets, 3)) + np.array([1.5, 0.0, 0.0])
    K = itf.weights / (4 * np.pi * np.linalg.norm(T[:, None, :] - itf.points[None], axis=2))
    S = rng.standard_normal((itf.n, 130))
    op = bie.laplace3d_pottrg(itf, T)
    for k in (1, 3, 7, 8, 9, 16, 17, 33, 64, 65, 130):
        phi = op @ np.asfortranarray(S[:, :k])
        assert np.all(np.abs(phi - K @ S[:, :k]) <= 1e-12 * (K @ np.abs(S[:, :k]))), k
