"""The exchange of partial tiles between the CTAs of a split-precision GEMM where it can go wrong: more CTAs in a
cluster than K chunks (some send zeros), tiles with rows and columns beyond the matrix, each cluster size in both
GEMMs, two and three pieces (whose landing place lies behind the operand ring and over it).  Against the FP64
oracle with the tolerances of the split-precision matvec (test_gpu_mixed.py)."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_mixed import TOL, dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("split", ["1,1", "2,4", "4,2", "8,8"])
@pytest.mark.parametrize("d,D1,D2", [(2, 16, 16), (3, 144, 80), (2, 80, 272)])
def test_split_edges(oracle, split, d, D1, D2, monkeypatch):
    import torch
    import tensornetworks_b200 as T
    monkeypatch.setenv("TN_CHAIN_SPLITK", split)
    ctx = T.default_context()
    rng = np.random.default_rng(D1 + D2)
    W = oracle.mpo_site(10, (d - 1) / 2, 2, 1.0, 1.0, 0.2, 5)
    F = rng.uniform(-1, 1, size=5 * D1 * D1)
    G = rng.uniform(-1, 1, size=5 * D2 * D2)
    x = rng.uniform(-1, 1, size=d * D1 * D2)
    ref = oracle.heff_matvec(W, F, G, x, D1, D2)
    dF, dG, dx = dev(F), dev(G), dev(x)
    Wc = np.ascontiguousarray(W.ravel())
    for prec in (1, 2):
        h = C.c_void_p()
        T._capi.check(ctx._lib.tn_heff_create(ctx.handle, prec, d, 5, 5, D1, D2, Wc.ctypes.data, dF.data_ptr(),
                                              dG.data_ptr(), C.byref(h)), "create")
        y = dev(np.full(x.size, np.nan))
        T._capi.check(ctx._lib.tn_heff_apply(h, dx.data_ptr(), y.data_ptr()), "apply")
        torch.cuda.synchronize()  # the handle's launches are on the context's stream
        assert np.linalg.norm(y.cpu().numpy() - ref) / np.linalg.norm(ref) <= TOL[prec]
        T._capi.check(ctx._lib.tn_heff_destroy(h), "destroy")
