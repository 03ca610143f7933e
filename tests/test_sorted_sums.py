"""The direct sums' sorted node order (planes together, padded tiles) on surfaces that exercise
its branches, against the dense sum in numpy: planes of exactly the smallest size that is kept
together (256 nodes), smaller ones, coplanar faces with opposite normals, tilted faces (no planes),
both in one interface, a single panel, and lengths far from 1. Widths around every kernel's edges.

Tolerances, row by row against s_i = sum_j |G_ij| |X_j|: FP64 2^-43 (as the parity tests' 1e-13 on
the norm); the reduced precisions 2^-13: split-BF16 and FP32 terms are good to 2^-16, and rounding
coordinates to FP32 adds up to 3 * 2^-24 * (tile size / distance), 2^-14 at a ratio of 340."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rotated(bie, itf, keep=0):
    """The interface turned about an oblique axis, all panels but the first `keep`."""
    a, b = 0.7, 0.4
    R = (np.array([[np.cos(a), -np.sin(a), 0], [np.sin(a), np.cos(a), 0], [0, 0, 1]])
         @ np.array([[1, 0, 0], [0, np.cos(b), -np.sin(b)], [0, np.sin(b), np.cos(b)]]))
    x, w = bie.gausslegendre(itf.n_quad)
    panels = []
    for p in range(itf.npanels):
        T, shift = (np.eye(3), np.zeros(3)) if p < keep else (R, np.array([3.0, 0.0, 0.0]) if keep else np.zeros(3))
        c = itf.corners[p] @ T.T + shift
        panels.append(bie.rect_panel3d_discretize(*c, x, w, T @ itf.panel_normals[p], bool(itf.is_edge[p])))
    return bie.DielectricInterface(panels, itf.eps_in, itf.eps_out)


def surface(bie, name):
    box = bie.single_dielectric_box3d
    if name == "planes_of_256":
        return box(0.5, 0.5, 0.5, 4, 0.2, 4.0, 1.0)
    if name == "uneven_planes":
        return box(1.2, 0.8, 0.6, 4, 0.2, 4.0, 1.0)
    if name == "touching":
        return bie.multi_dielectric_box3d(4, 0.25, [((0, 0, 0), 1.0, 1.0, 1.0), ((1.0, 0, 0), 1.0, 1.0, 1.0)],
                                          [2.0, 4.0], 1.0)
    if name == "tilted":
        return rotated(bie, box(0.7, 0.6, 0.5, 4, 0.3, 4.0, 1.0))
    if name == "mixed":
        itf = box(0.8, 0.7, 0.6, 4, 0.2, 4.0, 1.0)
        return rotated(bie, itf, keep=itf.npanels // 2)
    if name == "one_panel":
        x, w = bie.gausslegendre(4)
        c = np.array([[0, 0, 0], [1, 0, 0], [1, 1, 0], [0, 1, 0]], dtype=float)
        c = np.stack([c, c + [0.2, 0.3, 0.5]])
        return bie.DielectricInterface([bie.rect_panel3d_discretize(*q, x, w, (0, 0, 1.0)) for q in c], 4.0, 1.0)
    if name == "nanometres":
        return box(1.2e-9, 0.8e-9, 0.6e-9, 4, 0.2e-9, 4.0, 1.0)
    raise ValueError(name)


def dense(itf):
    d = itf.points[:, None, :] - itf.points[None, :, :]
    r2 = (d * d).sum(-1)
    np.fill_diagonal(r2, 1.0)
    G = np.einsum("ia,ija->ij", itf.normals, d) / (r2 * np.sqrt(r2)) * itf.weights / (4 * np.pi)
    np.fill_diagonal(G, 0.0)
    return G


@pytest.mark.parametrize("name", ["planes_of_256", "uneven_planes", "touching", "tilted", "mixed", "one_panel",
                                  "nanometres"])
def test_direct_sums_match_the_dense_sum(bie, rng, name):
    itf = surface(bie, name)
    op = bie.lhs_dielectric_box3d(itf)
    G = dense(itf)
    X = rng.standard_normal((itf.n, 70))
    Y, S = G @ X, np.abs(G) @ np.abs(X)
    todo = [("fp64", k, -43) for k in (1, 2, 3, 4, 5, 6, 7, 8, 9, 17, 33, 64, 65, 70)]
    todo += [("fp32", k, -13) for k in (1, 2, 3, 4, 8)]
    todo += [("bf16x3", k, -13) for k in (3, 16, 17, 48, 64, 70)] + [("bf16x6", k, -13) for k in (5, 33, 64, 70)]
    for precision, k, bits in todo:
        got = op.mul(np.asfortranarray(X[:, :k]), precision=precision, flags=2)  # without the diagonal
        worst = np.max(np.abs(got - Y[:, :k]) / S[:, :k])
        assert worst < 2.0 ** bits, (precision, k, worst)
