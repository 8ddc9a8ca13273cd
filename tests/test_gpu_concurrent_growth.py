"""Buffers of a chain that grow while other streams of the device are being captured: by a torch graph in the same
thread (no timing involved), and by the split-precision sweeps of other worker threads, which record graphs of their
own.  Growth may wait for its own context's streams only: a device-wide wait fails during a capture and invalidates
it.  Energies as without the capture and as one worker's, 1e-12 per site (tests/test_gpu_scan.py)."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def T():
    import tensornetworks_b200 as T
    return T


@pytest.mark.parametrize("precision", ["FP64", "MIXED"])
def test_growth_beside_a_capture(T, precision):
    import torch
    from tensornetworks_b200 import scan
    inst = scan.make_xxz_scan(1, seed=9, Lmin=12, Lmax=12, Ds=(32,))[0]
    opts = T.SolverOptions(precision=getattr(T, precision))
    ref = scan.solve(T.Context(0), inst, opts, dstart=16)
    ctx = T.Context(0)
    x = torch.zeros(8, device="cuda")
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=torch.cuda.Stream(), capture_error_mode="relaxed"):
        x += 1
        got = scan.solve(ctx, inst, opts, dstart=16)
        x += 1
    g.replay()
    torch.cuda.synchronize()
    assert (x == 2).all()
    assert abs(got["energy_per_site"] - ref["energy_per_site"]) < 1e-12


def test_workers_that_capture_and_grow(T):
    from tensornetworks_b200 import scan
    inst = scan.make_xxz_scan(12, seed=21, Lmin=10, Lmax=18, Ds=(32, 48, 64))
    opts = T.SolverOptions(precision=T.MIXED)
    one, _ = scan.run_scan(inst, workers=1, options=opts)
    many, _ = scan.run_scan(inst, workers=4, options=opts)
    assert len({r.worker for r in many}) > 1
    for a, b in zip(one, many):
        assert abs(a.energy_per_site - b.energy_per_site) < 1e-12, a.instance
