"""SVD and QR at the ends of the floating-point range, where squares of the entries underflow or overflow: whole
matrices of tiny and huge entries, harmless tiny columns beside ordinary ones (with zero columns after them), and
equal columns, whose remainders shrink by a rounding error a step.  Sizes next to those from which the SVD factors
first, one and several warps and CTAs of its kernel, and batches (the values of a chain's bonds).  SVD tolerances:
2 sqrt(m n) 1e-13 of the largest singular value, as for the Jacobi kernels elsewhere; QR: the bounds of
test_gpu_qr_cluster.py, 4 eps (k + 16) of orthogonality and of the matrix."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


def tiny_columns(m, n):
    """Ordinary columns, one of norm 1e-157, a smaller one, and zero ones after it."""
    A = np.random.default_rng(m + 100 * n).standard_normal((m, n))
    A[:, 5] *= 1e-157 / np.linalg.norm(A[:, 5])
    A[:, 6] = 0.0
    A[:, 8] = 0.0
    A[:, 9] *= 1e-160
    return A


def equal_columns(m, n, seed):
    rng = np.random.default_rng(seed)
    V = rng.standard_normal((m, 2))
    return V[:, rng.integers(0, 1 + seed % 2, n)]


def check_svd(T, B):
    U, s, Vt = T.CudaSVDSolver().SolveAll(B)
    top = np.abs(B).max()  # LAPACK and the products below on a matrix of ordinary size
    e = 2.0 ** np.round(np.log2(top)) if top > 0 else 1.0
    s0 = np.linalg.svd(B / e, compute_uv=False)
    k = len(s0)
    tol = 2 * np.sqrt(B.shape[0] * B.shape[1]) * 1e-13
    assert np.abs(s / e - s0).max() <= tol * s0[0]
    assert np.abs(U.T @ U - np.eye(k)).max() < tol
    assert np.abs(Vt @ Vt.T - np.eye(k)).max() < tol
    assert np.abs((U * (s / e)) @ Vt - B / e).max() <= tol * s0[0]


@pytest.mark.parametrize("scale", [1e-156, 1e-170, 1e-290, 1e-121, 1e121, 1e156, 1e290])
@pytest.mark.parametrize("m,n", [(1, 1), (5, 4), (12, 8), (33, 24), (25, 25), (40, 33), (150, 128), (300, 200)])
def test_svd_of_a_scaled_matrix(m, n, scale):
    import tensornetworks_b200 as T
    A = np.random.default_rng(m).standard_normal((m, n)) * 10.0 ** (-3.0 * np.arange(n) / n)
    check_svd(T, A * scale)
    check_svd(T, A.T * scale)


@pytest.mark.parametrize("m,n", [(20, 16), (30, 24), (40, 25), (40, 32), (64, 64), (200, 100)])
def test_svd_with_tiny_columns(m, n):
    import tensornetworks_b200 as T
    check_svd(T, tiny_columns(m, n))
    check_svd(T, tiny_columns(m, n).T)


@pytest.mark.parametrize("m,n", [(20, 16), (24, 24), (40, 32), (64, 60)])
def test_svd_of_equal_columns(m, n):
    import tensornetworks_b200 as T
    for seed in range(40):
        check_svd(T, equal_columns(m, n, seed))


@pytest.mark.parametrize("scale", [1e-156, 1e-290, 1e156])
@pytest.mark.parametrize("m,n", [(7, 6), (64, 40), (600, 20)])
def test_singular_values_alone(m, n, scale):
    import torch
    import tensornetworks_b200 as T
    ctx = T.default_context()
    A = np.random.default_rng(n).standard_normal((m, n))
    dA = torch.from_numpy(np.ascontiguousarray((A * scale).T)).cuda()
    s = torch.empty(n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    T._capi.check(ctx._lib.tn_svd_values(ctx.handle, m, n, C.c_void_p(dA.data_ptr()), m, C.c_void_p(s.data_ptr())),
                  "tn_svd_values")
    s0 = np.linalg.svd(A, compute_uv=False)
    assert np.abs(s.cpu().numpy() / scale - s0).max() <= 2 * np.sqrt(m * n) * 1e-13 * s0[0]


def qr(A):
    """tn_qr of A on a context of its own."""
    import torch
    import tensornetworks_b200 as T
    ctx = T.Context(0)
    m, n = A.shape
    k = min(m, n)
    a = torch.from_numpy(np.ascontiguousarray(A.T)).cuda()
    q = torch.empty((k, m), dtype=torch.float64, device="cuda")
    r = torch.empty((n, k), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    T._capi.check(ctx._lib.tn_qr(ctx.handle, m, n, C.c_void_p(a.data_ptr()), m, C.c_void_p(q.data_ptr()), m,
                                 C.c_void_p(r.data_ptr()), k), "tn_qr")
    return q.cpu().numpy().T, r.cpu().numpy().T


def check_qr(A, e=1.0):
    Q, R = qr(A)
    k = min(A.shape)
    unit = 4 * EPS * (k + 16)
    assert np.abs(Q.T @ Q - np.eye(k)).max() <= unit
    assert np.linalg.norm(Q @ (R / e) - A / e) <= unit * np.linalg.norm(A / e)
    assert np.array_equal(np.tril(R[:, :k], -1), np.zeros((k, k)))


@pytest.mark.parametrize("m,n", [(20, 16), (40, 32), (64, 64), (300, 96), (512, 100), (700, 80), (1300, 40), (1600, 40)])
def test_qr_with_tiny_columns(m, n):
    check_qr(tiny_columns(m, n))
    for x in (1e-150, 1e-154, 1e-158):  # at and below the square root of the smallest normal number
        A = tiny_columns(m, n)
        A[:, 3] *= x / np.linalg.norm(A[:, 3])
        check_qr(A)


@pytest.mark.parametrize("m,n", [(20, 16), (40, 33), (300, 96), (512, 100), (700, 80), (1300, 40), (1600, 40)])
def test_qr_of_a_tiny_matrix(m, n):
    A = np.random.default_rng(m).standard_normal((m, n))
    check_qr(A * 2.0 ** -512, 2.0 ** -512)
    check_qr(A * 2.0 ** -505, 2.0 ** -505)


@pytest.mark.parametrize("seed", range(8))
def test_qr_of_equal_columns(seed):
    check_qr(equal_columns(40, 32, seed))
    check_qr(equal_columns(600, 96, seed))
