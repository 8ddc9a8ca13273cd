"""Memory that is held and given back.  Growing a chain's site tensors holds the new ones and little else: with less
free memory than the new tensors take together, but enough beside the old ones given back on the way, the growth
succeeds and keeps the contents.  Large workspaces of the dense solvers and of a chain do not stay behind."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20


def test_growth_within_the_memory_of_the_new_tensors():
    import torch
    import tensornetworks_b200 as T
    ctx = T.Context(0)
    L, D = 64, 512                      # 64 tensors of 4 MB, then of 16 MB: 1024 MB, 768 MB more than before
    H = T.Factory(ctx).Make1D_NN_HeisenbergHamiltonian(L, 0.5, T.RegularLower, 1.0, 1.0, 0.0)
    psi = H.CreateMPS(D, 1e-12, 1e-12)
    rng = np.random.default_rng(2)
    some = {i: rng.standard_normal((2, 1 if i == 1 else D, 1 if i == L else D)) for i in (1, 2, 17, 33, 63, 64)}
    for i, A in some.items():
        psi.SetSite(i, A)
    ctx.synchronize()
    torch.cuda.synchronize()
    fill = torch.cuda.mem_get_info()[0] - 960 * MB
    if fill < 0:
        pytest.skip("another process holds the memory")
    hold = torch.empty(fill, dtype=torch.uint8, device="cuda")
    try:
        assert torch.cuda.mem_get_info()[0] < 1000 * MB
        psi.SetSite(5, np.ones((2, D, 2 * D)))
        for i, A in some.items():
            assert np.array_equal(psi.GetSite(i), A)
        assert (psi.GetSite(5) == 1).all()
    finally:
        del hold
        torch.cuda.empty_cache()


@pytest.mark.parametrize("solve", ["values", "solve", "eigen"])
def test_large_workspaces_of_the_dense_solvers_are_given_back(solve):
    import torch
    import tensornetworks_b200 as T
    ctx = T.Context(0)

    def run(m, n):
        rng = np.random.default_rng(m)
        A = rng.standard_normal((m, n))
        if solve == "eigen":
            A = np.diag(np.arange(1.0, n + 1))
        a = torch.from_numpy(np.ascontiguousarray(A.T)).cuda()
        u, s = torch.empty((n, m), dtype=torch.float64, device="cuda"), torch.empty(n, dtype=torch.float64, device="cuda")
        v = torch.empty((n, n), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        p = lambda t: C.c_void_p(t.data_ptr())
        if solve == "values":
            rc = ctx._lib.tn_svd_values(ctx.handle, m, n, p(a), m, p(s))
        elif solve == "solve":
            rc = ctx._lib.tn_svd_solve(ctx.handle, m, n, p(a), m, 1e-12, n, p(u), m, p(s), p(v), n)
        else:
            w = np.empty(1)
            rc = ctx._lib.tn_eigensolve_dense(ctx.handle, n, p(a), n, 1, 1e-12, C.c_void_p(w.ctypes.data), p(u), m)
            assert abs(w[0] - 1) < 1e-10 * n
        assert rc == 0, T._capi.last_error()

    big = (1600, 1600) if solve == "eigen" else (3000000, 3)  # 82 MB (four matrices) and 72 MB of workspace
    run(3, 3)
    torch.cuda.empty_cache()
    ctx.synchronize()
    before = torch.cuda.mem_get_info()[0]
    run(*big)
    torch.cuda.empty_cache()
    assert before - torch.cuda.mem_get_info()[0] < 32 * MB


def test_large_workspaces_of_a_chain_are_given_back():
    import gc
    import torch
    import tensornetworks_b200 as T
    ctx = T.Context(0)
    H = T.Factory(ctx).Make1D_NN_HeisenbergHamiltonian(4, 0.5, T.RegularLower, 1.0, 1.0, 0.0)
    psi = H.CreateMPS(8, 1e-12, 1e-12)
    psi.GetExpectation(H)
    torch.cuda.empty_cache()
    ctx.synchronize()
    before = torch.cuda.mem_get_info()[0]
    D = 3000  # two environments of 343 MB
    psi = H.CreateMPS(D, 1e-12, 1e-12)
    psi.GetExpectation(H)
    del psi
    gc.collect()
    contraction = 2 * 8 * 2 * 5 * D * D  # the context's own pair of scratch buffers
    assert before - torch.cuda.mem_get_info()[0] < contraction + 64 * MB


def test_work_buffers_do_not_outlive_a_change_of_stream():
    """A chain that has worked on a stream that the context no longer uses frees its buffers (which waits for the
    device) instead of handing them to the next chain, which would use them on another stream."""
    import gc
    import torch
    import tensornetworks_b200 as T
    ctx = T.Context(0)
    H = T.Factory(ctx).Make1D_NN_HeisenbergHamiltonian(4, 0.5, T.RegularLower, 1.0, 1.0, 0.0)
    D = 1000  # two environments of 38 MB
    streams = [torch.cuda.Stream() for _ in range(2)]
    left = []
    for change in (True, False):
        T._capi.check(ctx._lib.tn_ctx_set_stream(ctx.handle, C.c_void_p(streams[0].cuda_stream)), "set_stream")
        psi = H.CreateMPS(D, 1e-12, 1e-12)
        psi.GetExpectation(H)
        if change:
            T._capi.check(ctx._lib.tn_ctx_set_stream(ctx.handle, C.c_void_p(streams[1].cuda_stream)), "set_stream")
        del psi
        gc.collect()
        torch.cuda.synchronize()
        left.append(torch.cuda.mem_get_info()[0])
    T._capi.check(ctx._lib.tn_ctx_set_stream(ctx.handle, None), "set_stream")
    assert left[0] - left[1] > 64 * MB  # kept without a change, not kept with one
