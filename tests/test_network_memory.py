"""Device memory of a network: one set of arrays per batch row, whichever way it trains,
and what the ways share is not mixed up."""
import numpy as np
import pytest


def _up16(n):
    return (n + 15) // 16 * 16


@pytest.mark.gpu
@pytest.mark.parametrize("hidden, layers, n_bins", [(128, 1, 15), (256, 2, 127), (256, 4, 64),
                                                    (128, 16, 64)])
def test_bytes_per_batch_row(pp, gpu_ctx, hidden, layers, n_bins):
    torch = pytest.importorskip("torch")
    rows = 1 << 18

    def used(max_batch):
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        net = pp.surrogate.MLP(n_in=8, hidden=hidden, n_layers=layers, n_bins=n_bins,
                               max_batch=max_batch)
        after = torch.cuda.mem_get_info()[0]
        net.close()
        return before - after

    # BF16 inputs, activations and pre-activations (2 L hidden), two gradients of the
    # width of a layer, the outputs in FP32 and their gradients
    row = 2 * (16 + 2 * layers * hidden + 2 * hidden + 3 * _up16(n_bins + 1))
    assert used(rows) - used(64) <= row * rows + (16 << 20)  # (allocations round up)


@pytest.mark.gpu
@pytest.mark.parametrize("hidden, B", [(128, 500), (256, 129)])
def test_forward_between_gradients(pp, gpu_ctx, hidden, B):
    """A forward call uses the memory of a step: the gradients after it are those
    before it, and its outputs those of a network that never trained."""
    torch = pytest.importorskip("torch")
    torch.manual_seed(B)
    x = torch.randn((B, 8), device="cuda")
    count = torch.poisson(torch.full((B,), 5.0, device="cuda"))
    hist = torch.poisson(torch.full((B, 64), 0.5, device="cuda"))
    net = pp.surrogate.MLP(hidden=hidden, n_layers=3, n_bins=64, max_batch=B, seed=3)
    out = [torch.zeros((B, 80), device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    net.forward(x.data_ptr(), B, out[0].data_ptr())
    torch.cuda.synchronize()
    runs = []
    for _ in range(2):
        runs.append(net.loss_grad(x.data_ptr(), count.data_ptr(), hist.data_ptr(), B))
        net.forward(x.data_ptr(), B, out[1].data_ptr())
        torch.cuda.synchronize()
        assert torch.equal(out[0], out[1])
    net.close()
    assert runs[0][0] == pytest.approx(runs[1][0], rel=1e-5)  # (atomic sums)
    np.testing.assert_allclose(runs[0][1], runs[1][1], rtol=0,
                               atol=1e-5 * np.abs(runs[0][1]).max())
