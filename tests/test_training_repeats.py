"""Runs over the same batches: up to 256 rows the weight gradients are sums in one order,
so that nearly every parameter agrees between runs of many steps, however they were
issued and whatever ran between them."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("hidden, layers, n_bins, B", [(256, 4, 64, 256), (256, 2, 127, 193),
                                                       (128, 3, 32, 129), (128, 1, 15, 64)])
def test_small_batches_repeat(pp, gpu_ctx, hidden, layers, n_bins, B):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(B)
    n, steps = 2000, 12
    dev = [torch.tensor(a, device="cuda") for a in
           (rng.normal(size=(n, 8)).astype(np.float32), rng.poisson(5.0, n).astype(np.float32),
            rng.poisson(0.5, (n, n_bins)).astype(np.float32))]
    ptrs = [t.data_ptr() for t in dev]
    first, differ = None, 0.0
    for run in range(40):
        net = pp.surrogate.MLP(hidden=hidden, n_layers=layers, n_bins=n_bins, max_batch=B, seed=10)
        for part in ((steps,), (5, steps - 5), (1,) * steps)[run % 3]:
            net.train_steps(*ptrs, n, B, part, 0, steps, 2e-3, 1e-4, 77)
        p = net.params()
        net.close()
        first = p if first is None else first
        differ = max(differ, float(np.mean(np.abs(p - first) > 1e-6)))
    assert differ < 0.01
