"""Fused inference at the edges of its 64-column chunks: hidden widths that end
inside a chunk or leave epilogue warps without columns, inputs of more than one
chunk, and tiles that end inside a CTA's pair."""
import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "oracle"))
import mlp_oracle  # noqa: E402


@pytest.mark.gpu
@pytest.mark.parametrize("n,n_in,hidden,layers,n_bins", [
    (1, 8, 16, 1, 1), (257, 65, 80, 2, 31), (300, 130, 112, 5, 127), (40000, 8, 192, 3, 64),
    (500, 17, 240, 2, 128)])
def test_matches_oracle(pp, gpu_ctx, n, n_in, hidden, layers, n_bins):
    torch = pytest.importorskip("torch")
    mlp = pp.surrogate.MLP(n_in=n_in, hidden=hidden, n_layers=layers, n_bins=n_bins,
                           max_batch=256, seed=5)
    rng = np.random.default_rng(n)
    x = rng.normal(size=(n, n_in)).astype(np.float32)
    xd = torch.tensor(x, device="cuda")
    expect = torch.full((n,), -1.0, device="cuda")
    pdf = torch.full((n, n_bins), -1.0, device="cuda")
    mlp.infer(xd.data_ptr(), n, expect.data_ptr(), pdf.data_ptr())
    W, b = mlp.unpack(mlp.params())
    lam, p_ref = mlp_oracle.MLPOracle(W, b, n_in, n_bins).predict(x)
    # the oracle has the kernel's BF16 rounding points: tolerances of the
    # comparison with it in test_mlp.py
    np.testing.assert_allclose(np.log(expect.cpu().numpy()), np.log(lam), atol=1e-2)
    np.testing.assert_allclose(pdf.cpu().numpy(), p_ref, rtol=1e-2, atol=1e-5)
    mlp.close()
