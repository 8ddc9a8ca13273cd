"""The cluster Householder QR (one launch; columns in blocks of 32, rows dealt to
the CTAs of a cluster) at the edges of its tiles: single rows and columns, one
more and one less than a block, every cluster size and row count per lane, wide
and square matrices, leading dimensions above the row count, outputs in the
input's memory (which take the path with a copy), and rank-deficient input; QR,
LQ, RQ and QL against LAPACK's factors."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


@pytest.fixture(scope="module")
def env():
    import torch
    import tensornetworks_b200 as T
    from tensornetworks_b200 import _capi
    return torch, _capi.load(), T.Context(0)


def call(env, kind, A, pad=0, inplace=False):
    """(first factor, second factor) of tn_<kind>; column-major device buffers with `pad` extra rows."""
    torch, lib, ctx = env
    m, n = A.shape
    k = min(m, n)

    def dev(r, c, M=None):
        t = torch.full((c, r + pad), 7.0, dtype=torch.float64, device="cuda")
        if M is not None:
            t[:, :r] = torch.from_numpy(np.ascontiguousarray(M.T)).cuda()
        return t
    a = dev(m, n, A)
    f1 = a if inplace else dev(m, k)
    f2 = dev(k, n)
    rc = getattr(lib, "tn_" + kind)(ctx.handle, m, n, C.c_void_p(a.data_ptr()), m + pad, C.c_void_p(f1.data_ptr()),
                                    m + pad, C.c_void_p(f2.data_ptr()), k + pad)
    assert rc == 0
    F1, F2 = f1.cpu().numpy().T, f2.cpu().numpy().T
    if pad:  # nothing beyond the rows is written
        assert (F1[m:, :k] == 7.0).all() and (F2[k:] == 7.0).all()
    if not inplace:
        assert np.array_equal(a.cpu().numpy().T[:m], A)
    return F1[:m, :k], F2[:k]


def bounds(A):
    """Householder QR in k steps: backward error and loss of orthogonality of a few eps per step; R moves by
    at most about (1 + sqrt 2) cond times the (Frobenius) backward error of each side."""
    k = min(A.shape)
    unit = 4 * EPS * (k + 16)
    s = np.linalg.svd(A[:, :k], compute_uv=False)
    na = np.linalg.norm(A)
    return unit, unit * na, 5 * unit * na * (na / s[-1] if s[-1] > 0 else np.inf)


def check(A, Q, R, signs=True):
    uo, ua, ur = bounds(A)
    k = min(A.shape)
    assert np.abs(Q.T @ Q - np.eye(k)).max() <= uo
    assert np.linalg.norm(Q @ R - A) <= ua
    assert np.array_equal(np.tril(R[:, :k], -1), np.zeros((k, k)))
    if signs:
        assert np.linalg.norm(R - np.linalg.qr(A, mode="r")) <= ur


SIZES = [(1, 1), (1, 40), (40, 1), (2, 3), (31, 31), (32, 32), (33, 32), (33, 33), (64, 65), (65, 31), (128, 128),
         (128, 300), (129, 96), (160, 40), (192, 193), (256, 70), (257, 64), (384, 100), (512, 512), (512, 600),
         (513, 33), (768, 96), (1000, 130), (1025, 65), (1280, 97), (1536, 512), (1537, 40)]


@pytest.mark.parametrize("m,n", SIZES)
def test_qr_at_tile_edges(env, m, n):
    rng = np.random.default_rng(1000 * m + n)
    A = rng.uniform(-1, 1, size=(m, n))
    Q, R = call(env, "qr", A, pad=m % 3)
    check(A, Q, R)


@pytest.mark.parametrize("m,n", [(5, 7), (33, 40), (40, 33), (130, 200), (300, 90), (70, 600)])
def test_other_orders(env, m, n):
    rng = np.random.default_rng(m + 1000 * n)
    A = rng.uniform(-1, 1, size=(m, n))
    L, Q = call(env, "lq", A, pad=1)
    check(A.T.copy(), Q.T, L.T)
    R, Q = call(env, "rq", A)                     # P A^T P = (P Q^T P)(P R^T P)
    check(A.T[::-1, ::-1].copy(), Q.T[::-1, ::-1], R.T[::-1, ::-1])
    Q, L = call(env, "ql", A, pad=2)              # P A P = (P Q P)(P L P)
    check(A[::-1, ::-1].copy(), Q[::-1, ::-1], L[::-1, ::-1])


def test_output_in_the_input(env):
    A = np.random.default_rng(3).uniform(-1, 1, size=(200, 100))
    Q, R = call(env, "qr", A, inplace=True)
    check(A, Q, R)


@pytest.mark.parametrize("m,n", [(96, 80), (200, 128), (600, 64)])
def test_rank_deficient(env, m, n):
    rng = np.random.default_rng(m)
    A = rng.uniform(-1, 1, size=(m, 5)) @ rng.uniform(-1, 1, size=(5, n))
    A[:, 3] = 0.0
    A[:, 40] = A[:, 2]
    Q, R = call(env, "qr", A)
    check(A, Q, R, signs=False)
    Z = np.zeros((m, n))
    Q, R = call(env, "qr", Z)
    check(Z, Q, R, signs=False)
    assert np.array_equal(Q, np.eye(m, n))
