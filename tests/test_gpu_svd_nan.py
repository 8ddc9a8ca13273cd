"""A matrix with a NaN or an infinity in it does not come back as one with clean singular values: every value is NaN
(an infinity may show as such), whatever its place, with and without vectors, by the cluster kernel, by way of the QR
and by the one-CTA kernel; the dense eigensolver's values likewise."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("m,n", [(1, 1), (3, 3), (9, 2), (40, 24), (24, 60), (64, 25), (150, 128), (600, 10)])
def test_svd(m, n, bad):
    import torch
    import tensornetworks_b200 as T
    ctx = T.default_context()
    rng = np.random.default_rng(m * n)
    k = min(m, n)
    for place in [(0, 0), (m - 1, n - 1), (m // 2, n // 3)]:
        A = rng.standard_normal((m, n))
        A[place] = bad
        a = torch.from_numpy(np.ascontiguousarray(A.T)).cuda()
        for vectors in (False, True):
            s = torch.zeros(k, dtype=torch.float64, device="cuda")
            u, v = (torch.zeros(r, dtype=torch.float64, device="cuda") for r in (m * k, n * k))
            torch.cuda.synchronize()
            p = lambda t: C.c_void_p(t.data_ptr())
            if vectors:
                rc = ctx._lib.tn_svd(ctx.handle, m, n, p(a), m, p(u), m, p(s), p(v), k)
            else:
                rc = ctx._lib.tn_svd_values(ctx.handle, m, n, p(a), m, p(s))
            assert rc == 0
            got = s.cpu().numpy()
            assert not np.isfinite(got[0])
            if np.isnan(bad):
                assert np.isnan(got).all()


@pytest.mark.parametrize("N", [1, 5, 30, 70])
def test_eigenvalues(N):
    import torch
    import tensornetworks_b200 as T
    ctx = T.default_context()
    A = np.random.default_rng(N).standard_normal((N, N))
    A = A + A.T
    A[N // 2, N // 3] = A[N // 3, N // 2] = np.nan
    a, u = torch.from_numpy(A).cuda(), torch.zeros((N, N), dtype=torch.float64, device="cuda")
    w = np.zeros(N)
    torch.cuda.synchronize()
    rc = ctx._lib.tn_eigensolve_dense(ctx.handle, N, C.c_void_p(a.data_ptr()), N, N, 1e-12, C.c_void_p(w.ctypes.data),
                                      C.c_void_p(u.data_ptr()), N)
    assert rc != 0 or np.isnan(w).all()
