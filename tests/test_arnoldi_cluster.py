"""Per-column GMRES around the sizes where its orthogonalisation step runs in one cluster (at most
8,192 values and 8 columns), against numpy's solve of the dense matrix: below, at and past both limits,
fewer nodes than the cluster has threads, restarts, FP64 (two Gram-Schmidt passes) and refined (one).

Tolerance: FP64 solves stop at a residual of 1e-13, and the matrices' condition numbers are below 100:
1e-11. Refined solves stop at 1e-10: 1e-8."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def dense(itf):
    d = itf.points[:, None, :] - itf.points[None, :, :]
    r2 = (d * d).sum(-1)
    np.fill_diagonal(r2, 1.0)
    A = np.einsum("ia,ija->ij", itf.normals, d) / (r2 * np.sqrt(r2)) * itf.weights / (4 * np.pi)
    np.fill_diagonal(A, itf.diag)
    return A


@pytest.mark.parametrize("box, widths", [
    ((1.0, 0.9, 0.7, 4, 0.25, 4.0, 1.0), (1, 4, 5, 8, 9)),    # 2,048 nodes: 4 columns at the limit
    ((0.5, 0.5, 0.5, 4, 0.3, 4.0, 1.0), (3, 5, 6, 8, 9)),
    ((0.5, 0.4, 0.3, 2, 1.0, 2.0, 1.0), (1, 8, 9)),           # fewer nodes than threads
])
def test_small_column_solves_match_the_dense_solve(bie, rng, box, widths):
    itf = bie.single_dielectric_box3d(*box)
    op = bie.lhs_dielectric_box3d(itf)
    A = dense(itf)
    assert np.linalg.cond(A) < 100
    F = rng.standard_normal((itf.n, max(widths)))
    X = np.linalg.solve(A, F)
    for k in widths:
        for restart in (200, 7):
            for _ in range(2):  # the second solve replays captured iterations
                S, st = bie.gpu_solve(op, F[:, :k], rtol=1e-13, restart=restart)
            assert st.solved
            assert np.linalg.norm(S - X[:, :k]) < 1e-11 * np.linalg.norm(X[:, :k]), (k, restart)
        S, st = bie.gpu_solve(op, F[:, :k], rtol=1e-10, precision="bf16x3")
        assert st.solved and np.linalg.norm(S - X[:, :k]) < 1e-8 * np.linalg.norm(X[:, :k]), k
