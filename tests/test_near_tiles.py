"""FP32 sums of pairs closer than a tile of the direct sums is wide: two faces at a right angle, their
panels halved again and again towards the common edge, so that the nearest nodes of the two faces
are thousands of times closer than the tiles' sides. Coordinates rounded to FP32 relative to a tile
leave such pairs no more than a few correct digits. And the edges of ordinary boxes.

Tolerances, row by row against s_i = sum_j w_j |X_j| / (4 pi r_ij^2): a kernel value whose
differences carry an FP32 rounding each is off by three times the relative error of 1 / r, 2^-22.9 (the
hardware's reciprocal square root) + 1.5 * 2^-24, so 2^-20.9; 64 additions of a tile lose half of
2^-24 each, 2^-19.1; 2^-18.7 together. On the norm, independent errors: half the kernel value's
2^-20.9, 3.6e-7."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def wedge(bie, levels, turned):
    """Faces z = 0 and y = 0 (turned: about an oblique axis, no coordinate planes), 8 panels along the edge."""
    x, w = bie.gausslegendre(4)
    T = np.eye(3)
    if turned:
        a, b = 0.7, 0.4
        T = (np.array([[np.cos(a), -np.sin(a), 0], [np.sin(a), np.cos(a), 0], [0, 0, 1]])
             @ np.array([[1, 0, 0], [0, np.cos(b), -np.sin(b)], [0, np.sin(b), np.cos(b)]]))
    panels = []
    ends = [0.0] + [2.0 ** -k for k in range(levels, -1, -1)]
    for lo, hi in zip(ends[:-1], ends[1:]):
        for i in range(8):
            l, r = i / 8, (i + 1) / 8
            for c, n in (([[l, lo, 0], [r, lo, 0], [r, hi, 0], [l, hi, 0]], [0, 0, 1.0]),
                         ([[l, 0, lo], [l, 0, hi], [r, 0, hi], [r, 0, lo]], [0, 1.0, 0])):
                panels.append(bie.rect_panel3d_discretize(*(np.array(c, dtype=float) @ T.T), x, w, T @ np.array(n)))
    return bie.DielectricInterface(panels, 4.0, 1.0)


def dense_apply(itf, X):
    """The sum and s."""
    Y, S = np.empty_like(X), np.empty_like(X)
    for lo in range(0, itf.n, 256):
        rows = slice(lo, lo + 256)
        d = itf.points[rows, None, :] - itf.points[None]
        r2 = (d * d).sum(-1)
        w = np.broadcast_to(itf.weights / (4 * np.pi), r2.shape).copy()
        own = np.arange(lo, min(itf.n, lo + 256))
        r2[own - lo, own], w[own - lo, own] = 1.0, 0.0
        Y[rows] = (np.einsum("ia,ija->ij", itf.normals[rows], d) / (r2 * np.sqrt(r2)) * w) @ X
        S[rows] = (w / r2) @ np.abs(X)
    return Y, S


@pytest.mark.parametrize("turned", [False, True])
def test_pairs_much_closer_than_a_tile(bie, rng, turned):
    itf = wedge(bie, 14, turned)
    op = bie.lhs_dielectric_box3d(itf)
    X = rng.standard_normal((itf.n, 4))
    Y, S = dense_apply(itf, X)
    for k in (1, 2, 3, 4):
        got = op.mul(np.asfortranarray(X[:, :k]), precision="fp32", flags=2)  # without the diagonal
        worst = np.max(np.abs(got - Y[:, :k]) / S[:, :k])
        assert worst < 2.0 ** -18.7, (k, worst)


@pytest.mark.parametrize("box", [(1.0, 0.9, 0.7, 4, 0.25, 4.0), (1.1, 0.9, 0.6, 6, 0.12, 4.0)])
def test_edges_of_a_box_in_fp32(bie, rng, box):
    itf = bie.single_dielectric_box3d(*box, 1.0)
    op = bie.lhs_dielectric_box3d(itf)
    X = rng.standard_normal((itf.n, 2))
    Y, _ = dense_apply(itf, X)
    got = op.mul(np.asfortranarray(X), precision="fp32", flags=2)
    assert np.linalg.norm(got - Y) / np.linalg.norm(Y) < 3.6e-7


def sheets(bie, gap):
    """Two parallel unit squares with the same panels, normals towards each other."""
    x, w = bie.gausslegendre(4)
    at = lambda i, j, z: np.array([i / 8, j / 8, z])
    return bie.DielectricInterface([bie.rect_panel3d_discretize(at(i, j, z), at(i + 1, j, z), at(i + 1, j + 1, z),
                                                                at(i, j + 1, z), x, w, (0.0, 0.0, n))
                                    for z, n in ((0.0, 1.0), (gap, -1.0)) for i in range(8) for j in range(8)], 4.0, 1.0)


@pytest.mark.parametrize("precision", ["fp32", "bf16x3", "bf16x6"])
@pytest.mark.parametrize("bits", [30, 45, 50])
def test_facing_nodes_almost_in_one_plane(bie, rng, bits, precision):
    """Facing nodes 2^-bits apart: their term is the sum. r^2 + 1e-24 costs a relative 1.5e-24 / 4^-30, 2^-19,
    at 2^-30; closer than the FP32 range holds, every result is still a number."""
    itf = sheets(bie, 2.0 ** -bits)
    op = bie.lhs_dielectric_box3d(itf)
    X = rng.uniform(0.5, 1.5, (itf.n, 8))
    for k in (1, 2, 3, 4, 8):
        got = op.mul(np.asfortranarray(X[:, :k]), precision=precision, flags=2)  # without the diagonal
        assert np.all(np.isfinite(got)), k
        if bits == 30:
            other = np.roll(np.arange(itf.n), itf.n // 2)
            want = -(itf.weights[:, None] * X[:, :k])[other] * 4.0 ** bits / (4 * np.pi)
            assert np.max(np.abs(got / want - 1)) < (2.0 ** -15.8 if precision == "bf16x3" else 2.0 ** -16.9), k
