"""The cluster Jacobi SVD at the edges of its ranges: the four columns of a warp, the
warps of a CTA, the CTAs of a cluster, the row slots of a lane, and the sizes next to the
one-CTA kernel; full-rank, graded and rank-deficient matrices.  Tolerances: 2 sqrt(m n)
1e-13 of the largest singular value, as for the one-CTA kernel."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def T():
    import tensornetworks_b200 as T
    return T


def matrix(m, n, kind, seed):
    rng = np.random.default_rng(seed)
    A = rng.standard_normal((m, n))
    if kind == "graded":
        A = A * 10.0 ** (-8.0 * np.arange(n) / n)
    if kind == "deficient":
        A[:, n // 2:] = 0.0
        A[:, 0] = A[:, min(1, n - 1)]
    return A


@pytest.mark.parametrize("kind", ["full", "graded", "deficient"])
@pytest.mark.parametrize("m,n", [(1, 1), (2, 2), (3, 3), (4, 4), (5, 5), (32, 8), (33, 9), (64, 16), (65, 17), (64, 33),
                                 (96, 64), (65, 65), (128, 128), (129, 128), (129, 129), (250, 97), (256, 256),
                                 (480, 31), (481, 33)])
def test_vectors(T, m, n, kind):
    A = matrix(m, n, kind, 1000 * m + n)
    for B in (A, A.T):
        U, s, Vt = T.CudaSVDSolver().SolveAll(B)
        s0 = np.linalg.svd(B, compute_uv=False)
        tol = 2 * np.sqrt(m * n) * 1e-13
        assert np.abs(s - s0).max() <= tol * s0[0]
        assert np.abs(U.T @ U - np.eye(n)).max() < tol
        assert np.abs(Vt @ Vt.T - np.eye(n)).max() < tol
        assert np.abs((U * s) @ Vt - B).max() <= tol * s0[0]  # a zero matrix included


@pytest.mark.parametrize("m,n", [(7, 6), (257, 130), (300, 257), (512, 260), (513, 40), (520, 515)])
def test_values(T, m, n):
    import torch
    A = matrix(m, n, "graded", m + n)
    ctx = T.default_context()
    dA = torch.from_numpy(np.ascontiguousarray(A.T)).cuda()
    s = torch.empty(n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    T._capi.check(ctx._lib.tn_svd_values(ctx.handle, m, n, C.c_void_p(dA.data_ptr()), m, C.c_void_p(s.data_ptr())),
                  "tn_svd_values")
    s0 = np.linalg.svd(A, compute_uv=False)
    assert np.abs(s.cpu().numpy() - s0).max() <= 2 * np.sqrt(m * n) * 1e-13 * s0[0]
