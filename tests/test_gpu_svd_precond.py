"""The SVD of one matrix by way of its QR factorisation, where that can go wrong: sizes next to the one from which it
is taken, blocks of 32 columns and one more, tall matrices, columns out of order by norm, ties, rank-deficient and
zero matrices (V' is completed there, U comes from Q), and values alone.  Tolerances 2 sqrt(m n) 1e-13 of the
largest singular value, as for the other Jacobi kernels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def matrix(m, n, kind):
    rng = np.random.default_rng(1000 * m + n)
    if kind == "zero":
        return np.zeros((m, n))
    if kind == "ties":
        return rng.choice([-1.0, 1.0], size=(m, n))
    A = rng.standard_normal((m, n)) * 10.0 ** (-8.0 * rng.permutation(n) / n)  # norms in no order
    if kind == "deficient":
        A[:, ::3] = 0.0
        A[:, 1] = A[:, 2]
    return A


@pytest.mark.parametrize("kind", ["mixed", "ties", "deficient", "zero"])
@pytest.mark.parametrize("m,n", [(24, 24), (25, 25), (26, 25), (32, 32), (33, 33), (40, 25), (200, 30), (64, 64),
                                 (100, 65), (400, 96), (200, 192)])
def test_vectors_and_values(m, n, kind):
    import tensornetworks_b200 as T
    A = matrix(m, n, kind)
    for B in (A, A.T):
        U, s, Vt = T.CudaSVDSolver().SolveAll(B)
        s0 = np.linalg.svd(B, compute_uv=False)
        tol = 2 * np.sqrt(m * n) * 1e-13
        assert np.abs(s - s0).max() <= tol * s0[0]
        assert np.abs(U.T @ U - np.eye(n)).max() < tol
        assert np.abs(Vt @ Vt.T - np.eye(n)).max() < tol
        assert np.abs((U * s) @ Vt - B).max() <= tol * s0[0]
