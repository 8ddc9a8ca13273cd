"""The Lanczos launch chain (sites or bases beyond the one-launch solve) at the edges of the sums its passes keep
in registers: bases of 31 to 63 vectors, so that a pass takes one chunk of 32 sums, exactly one, or two; sites of
less than one block and of more elements than threads.  Against the FP64 oracle's Ritz value, 1e-10 relative (as the
other solver tests; the residual target is 1e-10 and the value's error its square over the gap), unit vector 1e-12."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_kernels import envs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,krylov", [(4, 63), (16, 32), (16, 33), (17, 47), (17, 63), (40, 34), (196, 8), (196, 20),
                                      (200, 33)])
def test_basis_sizes(oracle, D, krylov):
    import torch
    import tensornetworks_b200 as T
    ctx = T.default_context()
    d = 2
    W, A, F, G = envs(oracle, d, D, D, 3)
    Dw1, Dw2 = W.shape[:2]
    x0 = oracle.site_flat(A)
    dF, dG, dx = (torch.from_numpy(np.ascontiguousarray(a).ravel()).cuda() for a in (F, G, x0))
    torch.cuda.synchronize()
    Wc = np.ascontiguousarray(W.ravel())
    th, res, nmv = C.c_double(), C.c_double(), C.c_int()
    opt = T.SolverOptions(krylov=krylov, max_restarts=60).to_c()
    st = ctx._lib.tn_eigensolve_heff(ctx.handle, C.byref(opt), d, Dw1, Dw2, D, D, Wc.ctypes.data, dF.data_ptr(),
                                     dG.data_ptr(), dx.data_ptr(), 1e-10, C.byref(th), C.byref(res), C.byref(nmv))
    assert st in (0, 1), T._capi.last_error()
    tho, _, _, _ = oracle.lanczos_heff(W, F, G, x0, D, D, krylov=20, max_restarts=30, tol=1e-10)
    assert abs(th.value - tho) < 1e-10 * max(1, abs(tho))
    assert abs(np.linalg.norm(dx.cpu().numpy()) - 1) < 1e-12
