"""Gram-Schmidt kernels at the edges of their row groups, blocks and vector loads,
against the same steps in numpy (FP64, pairwise sums: agreement to 1e-13 of the
orbital's norm before the projections are taken out)."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 255, 256, 513, 1000, 4097, 70002])
@pytest.mark.parametrize("rows", [1, 2, 8, 9, 17, 130])
@pytest.mark.parametrize("shift", [0, 1])
def test_gram_schmidt_step_matches_numpy(dev, native, n, rows, shift):
    rng = np.random.default_rng(n + rows)
    target = rows - 1
    V = rng.standard_normal((rows, n)) / np.sqrt(n)
    U, W = rng.standard_normal(n), rng.uniform(0.5, 1.5, n)
    buf = torch.zeros(rows * n + shift, dtype=torch.float64, device="cuda")   # shift: rows at odd 8-byte places
    Vt = buf[shift:].view(rows, n)
    Vt.copy_(torch.as_tensor(V))
    Ut, Wt = torch.as_tensor(U, device="cuda"), torch.as_tensor(W, device="cuda")
    dev.mgs(Vt, Ut, Wt, target)
    u = U - (V[:target] @ (U * W)) @ V[:target]
    norm = np.sqrt((u * u * W).sum())
    scale = np.abs(U).max() + np.abs(V[:target] @ (U * W)).sum() * (np.abs(V).max() if target else 0.0)
    assert np.abs(Ut.cpu().numpy() * norm - u).max() <= 1e-13 * scale
    assert torch.equal(Vt[target], Ut)
    if target <= 128:
        V2, U2 = torch.as_tensor(V, device="cuda"), torch.as_tensor(U, device="cuda")
        p = lambda t: ctypes.c_void_p(t.data_ptr())
        native.check(native.lib().tagi_mgs_dev_noalloc(p(V2), p(U2), p(Wt), target, n, rows, None))
        assert np.abs(U2.cpu().numpy() * norm - u).max() <= 1e-13 * scale


def test_zero_norm_divides_as_before(dev):
    V = torch.zeros(1, 10, dtype=torch.float64, device="cuda")
    U = torch.tensor([0.0] * 5 + [1.0] * 5, dtype=torch.float64, device="cuda")
    W = torch.zeros(10, dtype=torch.float64, device="cuda")
    out = dev.mgs(V, U, W, 0).cpu()
    assert torch.isnan(out[:5]).all() and torch.isinf(out[5:]).all()
