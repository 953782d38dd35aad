"""The bounded detection kernel (many POM hits) against the plain one, PMT by PMT:
a POM model whose QE table ends in a repeated knot is detected alike but keeps
the plain kernel."""
import ctypes

import numpy as np
import pytest

MANY = 1 << 20


def _records(pp, targets, n, seed):
    rng = np.random.default_rng(seed)
    rec = np.zeros(n, dtype=np.dtype(pp._lib.pp_hit_record))
    centre = np.array([t.shape.position for t in targets], np.float32)
    radius = np.array([t.shape.radius for t in targets], np.float32)
    mi = rng.integers(0, len(targets), n)
    v = rng.normal(size=(n, 3)).astype(np.float32)
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    d = pp.pom.pom_pmt_directions().astype(np.float32)
    k = rng.integers(0, 16, n)
    v[::5] = d[k[::5]]            # on a PMT's axis
    v[1::35] = -d[k[1::35]]       # and opposite to it
    v[2::1001] = [0.0, 0.0, 1.0]  # corners and edges of the direction map
    v[3::1001] = [0.0, 0.0, -1.0]
    v[4::1001] = [1.0, 0.0, 0.0]
    v[6::1001] = [0.0, -1.0, 0.0]
    scale = np.ones(n, np.float32)
    scale[7::50] = rng.uniform(0.5, 1.5, len(scale[7::50]))  # off the surface
    rec["position"] = centre[mi] + (radius[mi] * scale)[:, None] * v
    wl = rng.uniform(280.0, 820.0, n)
    wl[8::97] = rng.integers(13, 42, len(wl[8::97])) * 20.0  # on knots
    rec["wavelength"] = wl
    rec["direction"] = -v
    rec["module_index"] = mi + 1
    rec["module_index"][9::1000] = 0
    rec["module_index"][10::1000] = len(targets) + 1
    return rec


@pytest.mark.gpu
@pytest.mark.parametrize("n", [MANY - 1, MANY, MANY + 33, 3 * MANY + 1])
@pytest.mark.parametrize("orientation", [None, [[0.0, -1.0, 0.0], [1.0, 0.0, 0.0], [0.0, 0.0, 1.0]]])
def test_bounded_kernel_takes_the_plain_decisions(pp, gpu_ctx, n, orientation):
    torch = pytest.importorskip("torch")
    targets = [pp.POM.at([10.0 * i, -7.0 * i, 300.0 - 25.0 * i], i + 1) for i in range(24)]
    targets += [pp.DOM.at([0.0, 50.0, 0.0], 25),
                pp.HomogeneousDetector(pp.Spherical([0.0, 0.0, 90.0], 0.3), 0.05, 26)]
    rec = torch.from_numpy(_records(pp, targets, n, n % 7).view(np.uint8)).cuda()
    tg = pp.detection.pmt_targets(targets)
    lib = pp._lib.load()

    def run(lo, hi, models):
        ids = torch.full((hi - lo,), -1, dtype=torch.int32, device="cuda")
        qe = torch.full((hi - lo,), -1.0, dtype=torch.float32, device="cuda")
        rc = lib.pp_make_hits_from_photons_models(
            ctypes.c_void_p(rec[80 * lo:].data_ptr()), hi - lo, tg, len(targets),
            ctypes.byref(models), 77, ctypes.c_void_p(ids.data_ptr()),
            ctypes.c_void_p(qe.data_ptr()), None)
        assert rc == 0, pp._lib.last_error()
        torch.cuda.synchronize()
        return ids.cpu().numpy(), qe.cpu().numpy()

    models, keep = pp.detection.detection_models(targets, orientation, True)
    ids, qe = run(0, n, models)
    assert (ids > 0).mean() > 0.03
    # QE weights do not depend on the row: small calls take the plain kernel
    parts = [run(lo, min(lo + 500_000, n), models)[1] for lo in range(0, n, 500_000)]
    np.testing.assert_array_equal(qe, np.concatenate(parts))
    # decisions do (the row keys the random numbers): the repeated knot
    m = models.pom.contents
    m.qe_wavelength[m.n_qe] = m.qe_wavelength[m.n_qe - 1]
    m.qe[m.n_qe] = m.qe[m.n_qe - 1]
    m.n_qe += 1
    np.testing.assert_array_equal(ids, run(0, n, models)[0])
