"""The QR of a sweep's gauge moves, reached by tn_qr with the cluster QR switched off (TN_NO_CLUSTER_QR, read when a
context is created): that it is another kernel than the cluster one, its bounded waits, and its ways of forming Q at
the gauge shapes of a bulk D = 256 site.  Bounds as in test_gpu_kernels.py and test_gpu_qr_waits.py."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def context(monkeypatch, **env):
    import tensornetworks_b200 as T
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    return T, T.Context(0)


def raw_qr(ctx, A):
    import torch
    m, n = A.shape
    k = min(m, n)
    a = torch.from_numpy(np.ascontiguousarray(A.T)).cuda()
    q = torch.empty((k, m), dtype=torch.float64, device="cuda")
    r = torch.empty((n, k), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    rc = ctx._lib.tn_qr(ctx.handle, m, n, C.c_void_p(a.data_ptr()), m, C.c_void_p(q.data_ptr()), m,
                        C.c_void_p(r.data_ptr()), k)
    return rc, q.cpu().numpy().T, r.cpu().numpy().T


@pytest.mark.parametrize("forward", ["1", "0"])
def test_gauge_shapes(monkeypatch, oracle, forward):
    T, cluster = context(monkeypatch)
    _, gauge = context(monkeypatch, TN_NO_CLUSTER_QR="1", TN_QR_FORWARD_Q=forward)
    rng = np.random.default_rng(77)
    for m, n in [(512, 256), (512, 512), (256, 512), (480, 200), (65, 33)]:
        A = rng.uniform(-1, 1, size=(m, n))
        k = min(m, n)
        rc, Q, R = raw_qr(gauge, A)
        assert rc == 0
        assert np.abs(Q.T @ Q - np.eye(k)).max() < 1e-13
        assert np.abs(Q @ R - A).max() < 1e-12
        np.testing.assert_allclose(R, oracle.qr(A)[1], atol=1e-11)
        if m >= 256:  # sums in another order: not the cluster kernel's bits
            assert not np.array_equal(R, raw_qr(cluster, A)[2])
        A[:, n // 2 + 3:] = 0.0  # a grown bond
        rc, Q, R = raw_qr(gauge, A)
        assert rc == 0
        assert np.abs(Q.T @ Q - np.eye(k)).max() < 1e-13
        assert np.abs(Q @ R - A).max() < 1e-12


@pytest.mark.parametrize("off", ["0", "1"])
def test_expired_wait(monkeypatch, off):
    import torch
    T, ctx = context(monkeypatch, TN_NO_CLUSTER_QR=off, TN_QR_SPIN_LIMIT="1")
    A = np.random.default_rng(5).uniform(-1, 1, size=(512, 256))
    rc, _, _ = raw_qr(ctx, A)
    assert rc == 4 and "bounded wait" in T._capi.last_error()  # TN_CUDA_ERROR
    B = A[:9, :4].copy()  # the SVD of four columns waits for nothing
    b, sv = torch.from_numpy(np.ascontiguousarray(B.T)).cuda(), torch.empty(4, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    assert ctx._lib.tn_svd_values(ctx.handle, 9, 4, C.c_void_p(b.data_ptr()), 9, C.c_void_p(sv.data_ptr())) == 0
    assert np.abs(sv.cpu().numpy() - np.linalg.svd(B, compute_uv=False)).max() < 1e-12
