"""The waits between warps and CTAs inside the SVD, cluster QR and site-solve kernels are bounded: with the limit at
no poll at all (TN_WAIT_POLLS, read when a context is created) the first one expires, the kernel ends, the call
reports it, and the same context goes on with work that has no such waits.  No GPU fault is involved."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_kernels import envs

pytestmark = pytest.mark.gpu

CUDA_ERROR = 4


@pytest.fixture
def impatient(monkeypatch):
    """(T, a context whose waits do not wait)."""
    import tensornetworks_b200 as T
    monkeypatch.setenv("TN_WAIT_POLLS", "0")
    return T, T.Context(0)


def svd(T, ctx, A):
    import torch
    m, n = A.shape
    a = torch.from_numpy(np.ascontiguousarray(A.T)).cuda()
    s = torch.empty(n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    rc = ctx._lib.tn_svd_values(ctx.handle, m, n, C.c_void_p(a.data_ptr()), m, C.c_void_p(s.data_ptr()))
    return rc, s.cpu().numpy()


def works(T, ctx):
    """Four columns are one warp's: nothing to wait for."""
    A = np.random.default_rng(1).standard_normal((9, 4))
    rc, s = svd(T, ctx, A)
    assert rc == 0
    s0 = np.linalg.svd(A, compute_uv=False)
    assert np.abs(s - s0).max() <= 1e-12 * s0[0]


# within a CTA, between CTAs, inboxes of one parity, and after an expired factorisation
@pytest.mark.parametrize("factor", ["0", "1"])
@pytest.mark.parametrize("m,n", [(16, 8), (24, 24), (70, 65), (200, 128), (500, 260)])
def test_svd(monkeypatch, m, n, factor):
    import tensornetworks_b200 as T
    monkeypatch.setenv("TN_WAIT_POLLS", "0")
    monkeypatch.setenv("TN_QR_FORWARD_Q", factor)  # 0: no cluster QR, so no factorisation in front
    ctx = T.Context(0)
    A = np.random.default_rng(n).standard_normal((m, n))
    for _ in range(2):
        rc, _ = svd(T, ctx, A)
        assert rc == CUDA_ERROR and "wait" in T._capi.last_error()
        works(T, ctx)


@pytest.mark.parametrize("m,n", [(100, 40), (300, 20), (512, 256), (1000, 64)])
def test_qr(impatient, m, n):
    import torch
    T, ctx = impatient
    a = torch.rand((n, m), dtype=torch.float64, device="cuda")
    q, r = torch.empty_like(a), torch.empty((n, n), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    rc = ctx._lib.tn_qr(ctx.handle, m, n, *(C.c_void_p(p) if i % 2 == 0 else p for i, p in
                                            enumerate((a.data_ptr(), m, q.data_ptr(), m, r.data_ptr(), n))))
    assert rc == CUDA_ERROR and "wait" in T._capi.last_error()
    works(T, ctx)


def test_site_solve(impatient, oracle):
    import torch
    T, ctx = impatient
    d, D = 2, 64  # a grid of CTAs
    W, A, F, G = envs(oracle, d, D, D, 3)
    Dw1, Dw2 = W.shape[:2]
    dF, dG, dx = (torch.from_numpy(np.ascontiguousarray(v).ravel()).cuda() for v in (F, G, oracle.site_flat(A)))
    torch.cuda.synchronize()
    Wc = np.ascontiguousarray(W.ravel())
    th, res, nmv = C.c_double(), C.c_double(), C.c_int()
    opt = T.SolverOptions(krylov=20, max_restarts=30).to_c()
    rc = ctx._lib.tn_eigensolve_heff(ctx.handle, C.byref(opt), d, Dw1, Dw2, D, D, Wc.ctypes.data, dF.data_ptr(),
                                     dG.data_ptr(), dx.data_ptr(), 1e-10, C.byref(th), C.byref(res), C.byref(nmv))
    assert rc == CUDA_ERROR and "wait" in T._capi.last_error()
    works(T, ctx)


def test_sweep(impatient):
    T, ctx = impatient
    H = T.Factory(ctx).Make1D_NN_HeisenbergHamiltonian(8, 1.0, T.RegularLower, 1.0, 1.0, 0.0)
    psi = H.CreateMPS(81, 1e-12, 1e-12)
    psi.InitializeWith(T.Random, seed=3)
    sched = T.IterationSchedule()
    sched.Insert(T.IterationScheduleLine(2, 81, T.Epsilons(1e-12)))
    with pytest.raises(RuntimeError, match="wait"):
        psi.FindVariationalGroundState(H, sched, T.SolverOptions(precision=T.FP64))
    works(T, ctx)
