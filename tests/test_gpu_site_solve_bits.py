"""The one-launch FP64 site solve forms every sum in the order of the Lanczos launch chain: the two give equal Ritz
values, step counts and vectors, bit for bit, at cluster and grid launches, even and odd bonds, spins 1/2 and 1,
bases smaller than the site and site spaces smaller than the basis, one and several restarts.  A sweep's stopping
decisions see the last bit, so whole searches are compared as well.  The unit vector's Rayleigh quotient by the oracle's
matvec is the Ritz value to 1e-10, as in the other solver tests."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_kernels import envs

pytestmark = pytest.mark.gpu


@pytest.fixture
def contexts(monkeypatch):
    """(T, context with the one-launch solve, context with the chain)."""
    import tensornetworks_b200 as T
    one = T.Context(0)
    monkeypatch.setenv("TN_NO_SITE_SOLVE", "1")
    return T, one, T.Context(0)


@pytest.mark.parametrize("krylov,tol", [(20, 1e-10), (7, 1e-10), (30, 1e-6)])
@pytest.mark.parametrize("d,D,site", [(2, 1, 3), (2, 3, 3), (2, 16, 1), (2, 17, 3), (2, 23, 3), (2, 32, 6), (2, 45, 3),
                                      (2, 64, 3), (3, 13, 3), (3, 33, 3), (3, 90, 3), (2, 128, 3), (2, 194, 3)])
def test_site(contexts, oracle, d, D, site, krylov, tol):
    import torch
    T, one, chain = contexts
    W, A, F, G = envs(oracle, d, 1 if site == 1 else D, 1 if site == 6 else D, site)
    Dw1, Dw2 = W.shape[:2]
    D1, D2 = A.shape[1:]
    x0 = oracle.site_flat(A)
    dF, dG = (torch.from_numpy(np.ascontiguousarray(v).ravel()).cuda() for v in (F, G))
    Wc = np.ascontiguousarray(W.ravel())
    opt = T.SolverOptions(krylov=krylov, max_restarts=30).to_c()
    got = []
    for ctx in (one, chain):
        dx = torch.from_numpy(x0.copy()).cuda()
        torch.cuda.synchronize()
        th, res, nmv = C.c_double(), C.c_double(), C.c_int()
        n0 = ctx._lib.tn_launch_count()
        st = ctx._lib.tn_eigensolve_heff(ctx.handle, C.byref(opt), d, Dw1, Dw2, D1, D2, Wc.ctypes.data, dF.data_ptr(),
                                         dG.data_ptr(), dx.data_ptr(), tol, C.byref(th), C.byref(res), C.byref(nmv))
        assert st in (0, 1), T._capi.last_error()
        got.append((st, th.value, res.value, nmv.value, dx.cpu().numpy(), ctx._lib.tn_launch_count() - n0))
    (st, th, res, nmv, x, n1), b = got
    assert (st, th, res, nmv) == b[:4]
    assert np.array_equal(x, b[4])
    assert n1 < b[5]  # two ways indeed
    y = oracle.heff_matvec(W, F, G, x, D1, D2)
    assert abs(np.linalg.norm(x) - 1) < 1e-12
    assert abs(x @ y - th) < 1e-10 * max(1, abs(th))


@pytest.mark.parametrize("S,L,D", [(0.5, 10, 8), (0.5, 12, 33), (1.0, 8, 20)])
def test_search(contexts, S, L, D):
    T, one, chain = contexts
    got = []
    for ctx in (one, chain):
        H = T.Factory(ctx).Make1D_NN_HeisenbergHamiltonian(L, S, T.RegularLower, 1.0, 1.0, 0.1)
        psi = H.CreateMPS(D, 1e-12, 1e-12)
        psi.InitializeWith(T.Random, seed=11)
        sched = T.IterationSchedule()
        eps = T.Epsilons(1e-12)
        eps.itsEigenSolverEpsilon = 1e-10
        sched.Insert(T.IterationScheduleLine(2, D, 1, eps))
        var = psi.FindVariationalGroundState(H, sched, T.SolverOptions(precision=T.FP64))
        got.append((var, psi.GetSiteEnergies(), [psi.GetSite(i) for i in range(1, L + 1)]))
    assert got[0][0] == got[1][0]
    assert np.array_equal(got[0][1], got[1][1])
    assert all(np.array_equal(a, b) for a, b in zip(got[0][2], got[1][2]))
