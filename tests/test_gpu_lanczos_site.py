"""The one-launch site solve against the FP64 oracle at the edges of its ranges: sites smaller
than the Krylov basis, one and several blocks of 512 elements, cluster and grid launches, even
and odd bonds (16- and 8-byte copies), bases that are only 8-byte aligned, MPO boundaries,
spins with more terms, and sizes next to the launch chain's.  Tolerance 1e-10 relative on the
Ritz value and 1e-12 on the vector's norm, as for the launch chain (test_gpu_kernels.py)."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_kernels import envs, dev, host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("d,D,site", [(2, 1, 3), (2, 3, 3), (2, 7, 3), (2, 16, 1), (2, 17, 3), (2, 22, 3), (2, 23, 3), (2, 32, 6),
                                      (2, 45, 3), (2, 64, 3), (3, 13, 3), (3, 33, 3), (3, 90, 3), (2, 128, 3), (2, 194, 3),
                                      (2, 195, 3)])
def test_site_solve(oracle, d, D, site, offset):
    import torch
    import tensornetworks_b200 as T
    ctx = T.default_context()
    W, A, F, G = envs(oracle, d, 1 if site == 1 else D, 1 if site == 6 else D, site)  # the chain ends in bonds of 1
    Dw1, Dw2 = W.shape[:2]
    D1, D2 = A.shape[1:]
    x0 = oracle.site_flat(A)

    def shifted(a):
        t = torch.empty(a.size + offset, dtype=torch.float64, device="cuda")
        t[offset:] = torch.from_numpy(np.ascontiguousarray(a).ravel())
        return t

    dF, dG, dx = shifted(F), shifted(G), shifted(x0)
    torch.cuda.synchronize()
    p = lambda t: C.c_void_p(t.data_ptr() + 8 * offset)
    Wc = np.ascontiguousarray(W.ravel())
    th, res, nmv = C.c_double(), C.c_double(), C.c_int()
    opt = T.SolverOptions(krylov=20, max_restarts=30).to_c()
    st = ctx._lib.tn_eigensolve_heff(ctx.handle, C.byref(opt), d, Dw1, Dw2, D1, D2, Wc.ctypes.data, p(dF), p(dG), p(dx),
                                     1e-10, C.byref(th), C.byref(res), C.byref(nmv))
    assert st in (0, 1), T._capi.last_error()
    tho, _, _, _ = oracle.lanczos_heff(W, F, G, x0, D1, D2, krylov=20, max_restarts=30, tol=1e-10)
    assert abs(th.value - tho) < 1e-10 * max(1, abs(tho))
    x = dx[offset:].cpu().numpy()
    assert abs(np.linalg.norm(x) - 1) < 1e-12
