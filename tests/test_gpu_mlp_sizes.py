"""Gradient of the learned correction at the edges of its chunks (32 pairs up to 32 per
SM, 128 above) against the FP64 oracle.  Tolerance: at most ~300 FP32 additions in a row per
component (2e-5 of its absolute sum), 1e-4 of the largest component."""
import numpy as np
import pytest

from oracle import mlp_oracle as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 32, 33, 4095, 4736, 4737, 4865, 37889])
def test_gradient_sizes(n):
    import torch
    import tensornetworks_b200 as T
    rng = np.random.default_rng(n)
    m = T.LearnedCorrection(seed=3)
    p = (0.2 * rng.standard_normal(M.NP)).astype(np.float32)
    m.set_params(p)
    F = rng.standard_normal((n, 4)).astype(np.float32)
    t = rng.standard_normal(n).astype(np.float32)
    g, loss = m.gradient(torch.from_numpy(F).cuda(), torch.from_numpy(t).cuda())
    lref, gref = M.loss_and_grad(p.astype(np.float64), F, t)
    assert abs(loss - lref) <= 1e-5 * max(1.0, lref)
    assert np.abs(g - gref).max() <= 1e-4 * np.abs(gref).max()
