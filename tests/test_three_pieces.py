"""The split-BF16 sum in three pieces at the shapes of its kernel instances (16 and 32 columns folded a thread,
16 and 32 sources a thread, more than one pass): closer to the FP64 sum than in two pieces. Without
the third piece, or without one of the six products, it would be as far off as two pieces are, whose
terms carry 16 to 17 bits; four fifths of that error is the limit, as FP32 coordinates bound both."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("box", [(0.5, 0.5, 0.5, 4, 0.2, 4.0, 1.0), (1.2, 0.8, 0.6, 4, 0.1, 4.0, 1.0)])
def test_three_pieces_beat_two(bie, rng, box):
    itf = bie.single_dielectric_box3d(*box)
    op = bie.lhs_dielectric_box3d(itf)
    X = rng.standard_normal((itf.n, 140))
    for k in (16, 32, 33, 48, 64, 70, 96, 128, 140):
        Xk = np.asfortranarray(X[:, :k])
        Y = op.mul(Xk, flags=2)  # without the diagonal
        e3, e2 = (np.linalg.norm(op.mul(Xk, precision=p, flags=2) - Y) for p in ("bf16x6", "bf16x3"))
        assert e3 < 0.8 * e2, (k, e3 / e2)
