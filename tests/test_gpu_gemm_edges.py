"""The FP64 GEMM's asynchronous-copy path through the matvec and environment entry points at
the edges of its tiles (32 rows and columns, k-tiles of 16), even and odd leading dimensions
(16- and 8-byte copies) and bases that are only 8-byte aligned, against the FP64 oracle.
Tolerance 1e-12 normwise: sums of at most 5 x 200 products of O(1) values."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("D1,D2", [(1, 1), (1, 7), (8, 3), (15, 16), (16, 17), (31, 33), (32, 32), (33, 64), (65, 47),
                                   (96, 90), (131, 128), (200, 161)])
def test_edges(oracle, D1, D2, offset):
    import torch
    import tensornetworks_b200 as T
    ctx = T.default_context()
    rng = np.random.default_rng(100 * D1 + D2)
    d, Dw = 2, 5
    W = np.ascontiguousarray(oracle.mpo_site(10, 0.5, 2, 1.0, 0.7, 0.3, 5))
    host = [rng.uniform(-1, 1, n) for n in (Dw * D1 * D1, Dw * D2 * D2, d * D1 * D2)]

    def dev(a):
        t = torch.empty(a.size + offset, dtype=torch.float64, device="cuda")
        t[offset:] = torch.from_numpy(a)
        return t

    F, G, x = map(dev, host)
    y = dev(np.zeros(d * D1 * D2))
    Fo, Go = dev(np.zeros(Dw * D2 * D2)), dev(np.zeros(Dw * D1 * D1))
    torch.cuda.synchronize()
    p = lambda t: C.c_void_p(t.data_ptr() + 8 * offset)
    chk = T._capi.check
    chk(ctx._lib.tn_heff_matvec(ctx.handle, T.FP64, d, Dw, Dw, D1, D2, W.ctypes.data, p(F), p(G), p(x), p(y)), "matvec")
    chk(ctx._lib.tn_env_left(ctx.handle, T.FP64, d, Dw, Dw, D1, D2, W.ctypes.data, p(x), p(F), p(Fo)), "left")
    chk(ctx._lib.tn_env_right(ctx.handle, T.FP64, d, Dw, Dw, D1, D2, W.ctypes.data, p(x), p(G), p(Go)), "right")
    ctx.synchronize()
    A = host[2].reshape(d, D2, D1).transpose(0, 2, 1)
    Fh = host[0].reshape(Dw, D1, D1).transpose(0, 2, 1)
    Gh = host[1].reshape(Dw, D2, D2).transpose(0, 2, 1)
    left = np.einsum("vwmn,vnib->wmib", W, Fh[:, None] @ A[None])                             # sum W F A
    right = np.einsum("vwmn,wnaj->vmaj", W, Gh[:, None] @ A.transpose(0, 2, 1)[None])         # sum W G A^T
    ref = [(left @ Gh.transpose(0, 2, 1)[:, None]).sum(0),
           (A.transpose(0, 2, 1)[None] @ left).sum(1),
           (A[None] @ right).sum(1)]
    for got, want in zip((y, Fo, Go), ref):
        g = got[offset:].cpu().numpy().reshape(want.shape[0], want.shape[2], want.shape[1]).transpose(0, 2, 1)
        assert np.linalg.norm(g - want) <= 1e-12 * max(np.linalg.norm(want), 1e-300)
