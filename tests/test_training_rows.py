"""Gradients of the training step that takes 64 rows of the batch through all
layers at once, against the oracle at the edges of its tiles: rows per block,
64-column chunks of the layers' inputs, 8-column blocks of the outputs."""
import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "oracle"))
import mlp_oracle  # noqa: E402


@pytest.mark.gpu
@pytest.mark.parametrize("n_in,hidden,layers,n_bins,B", [
    (8, 128, 1, 15, 1),
    (1, 256, 1, 64, 63),
    (8, 128, 2, 63, 64),
    (8, 256, 2, 127, 65),
    (64, 256, 4, 64, 129),
    (17, 128, 5, 1, 500),
    (8, 256, 3, 32, 9800),  # more blocks than SMs
])
def test_gradients_match_oracle(pp, gpu_ctx, n_in, hidden, layers, n_bins, B):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(B)
    x = rng.normal(size=(B, n_in)).astype(np.float32)
    count = rng.poisson(5.0, B).astype(np.float32)
    hist = rng.poisson(0.5, (B, n_bins)).astype(np.float32)
    dev = [torch.tensor(a, device="cuda") for a in (x, count, hist)]
    mlp = pp.surrogate.MLP(n_in=n_in, hidden=hidden, n_layers=layers, n_bins=n_bins,
                           max_batch=B, seed=3)
    W, b = mlp.unpack(mlp.params())
    loss_ref, gW, gb = mlp_oracle.MLPOracle(W, b, n_in, n_bins).loss_grad(x, count, hist)
    for _ in range(2):  # the second call finds the accumulators of the first one zeroed
        loss, g = mlp.loss_grad(*[t.data_ptr() for t in dev], B)
        assert loss == pytest.approx(loss_ref, rel=1e-3)
        gW_dev, gb_dev = mlp.unpack(g)
        for l in range(len(gW)):
            for got, want, name in ((gW_dev[l], gW[l], "W"), (gb_dev[l], gb[l], "b")):
                err = np.linalg.norm(got - want) / max(np.linalg.norm(want), 1e-12)
                assert err < 2e-2, (l, name, err)
    mlp.close()
