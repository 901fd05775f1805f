"""Gradient of the proposal network at sample counts around its warp tiles (32
samples), blocks (128) and grid (304 blocks): against the FP64 oracle within
the FP32 accumulation error (2e-3 of the largest gradient, the bound of the
existing check), and bit-identical when repeated."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 31, 32, 33, 127, 129, 38912, 38913, 65536])
def test_gradient_sample_counts(ffi, mlp_oracle, n):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(n)
    X = rng.standard_normal((n, 8)).astype(np.float32)
    Y = (rng.random(n) < 0.4).astype(np.float32)
    p = ffi.Proposal(max_samples=16, seed=5)
    g, loss = p.gradient(X, Y, pos_weight=1.5)
    g2, loss2 = p.gradient(X, Y, pos_weight=1.5)
    want_loss, want = mlp_oracle.loss_and_grad(p.params(), X, Y, 1.5)
    p.close()
    assert np.array_equal(g, g2) and loss == loss2
    assert np.abs(g - want).max() <= 2e-3 * np.abs(want).max()
    assert abs(loss - want_loss) <= 2e-3 * abs(want_loss)
