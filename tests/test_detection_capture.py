"""Detection calls recorded by stream capture: a replay takes the targets and models
of the call, which the caller may change or free as soon as it has returned."""
import ctypes

import numpy as np
import pytest


def _targets(pp, n):
    kinds = [lambda p, i: pp.POM.at(p, i), lambda p, i: pp.DOM.at(p, i),
             lambda p, i: pp.make_generic_multipmt_om(p, 0.2159, i),
             lambda p, i: pp.HomogeneousDetector(pp.Spherical(p, 0.3), 0.5, i)]
    rng = np.random.default_rng(n)
    return [kinds[i % 4]([float(v) for v in rng.uniform(-200, 200, 3)], i + 1) for i in range(n)]


@pytest.mark.gpu
# targets and models within one small launch's parameters, in several launches, and
# the kernel of many POM hits
@pytest.mark.parametrize("n_targets, n", [(1, 1000), (400, 5000), (5000, 5000), (400, (1 << 20) + 5)])
def test_replay_after_the_callers_structures_are_gone(pp, gpu_ctx, n_targets, n):
    torch = pytest.importorskip("torch")
    targets = _targets(pp, n_targets)
    rng = np.random.default_rng(3)
    rec = np.zeros(n, dtype=np.dtype(pp._lib.pp_hit_record))
    mi = rng.integers(0, n_targets, n)
    v = rng.normal(size=(n, 3)).astype(np.float32)
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    centre = np.array([t.shape.position for t in targets], np.float32)
    radius = np.array([t.shape.radius for t in targets], np.float32)
    rec["position"] = centre[mi] + radius[mi, None] * v
    rec["direction"] = -v
    rec["wavelength"] = rng.uniform(300.0, 600.0, n)
    rec["module_index"] = mi + 1
    dev = torch.from_numpy(rec.view(np.uint8)).cuda()
    ids = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    qe = torch.full((n,), -1.0, dtype=torch.float32, device="cuda")
    tg = pp.detection.pmt_targets(targets)
    models, keep = pp.detection.detection_models(targets, None, True)
    lib = pp._lib.load()
    stream = torch.cuda.Stream()

    def call():
        rc = lib.pp_make_hits_from_photons_models(
            ctypes.c_void_p(dev.data_ptr()), n, tg, n_targets, ctypes.byref(models), 77,
            ctypes.c_void_p(ids.data_ptr()), ctypes.c_void_p(qe.data_ptr()),
            ctypes.c_void_p(stream.cuda_stream))
        assert rc == 0, pp._lib.last_error()

    torch.cuda.synchronize()
    call()
    stream.synchronize()
    want = ids.cpu().numpy(), qe.cpu().numpy()
    assert (want[0] > 0).any()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        call()
    for a in (tg, *keep):  # overwritten, as memory given back may be
        ctypes.memset(ctypes.addressof(a), 0xff, ctypes.sizeof(a))
    for _ in range(2):
        ids.fill_(-1)
        qe.fill_(-1.0)
        graph.replay()
        torch.cuda.synchronize()
        np.testing.assert_array_equal(ids.cpu().numpy(), want[0])
        np.testing.assert_array_equal(qe.cpu().numpy(), want[1])
