"""Mixed module lists at the size of the bounded detection kernel, from a few POM hits to only
POM hits: the decisions and weights of the plain kernel."""
import ctypes

import numpy as np
import pytest

from test_pmt_many import MANY, _records


@pytest.mark.gpu
@pytest.mark.parametrize("poms", [1, 3, 12])
@pytest.mark.parametrize("n", [MANY, MANY + 33])
def test_mixed_lists_take_the_plain_decisions(pp, gpu_ctx, poms, n):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(poms)
    targets = []
    for i in range(12):
        p = [float(c) for c in rng.uniform(-200, 200, 3)]
        if i < poms:
            targets.append(pp.POM.at(p, i + 1))
        elif i % 3 == 0:
            targets.append(pp.DOM.at(p, i + 1))
        elif i % 3 == 1:
            targets.append(pp.make_generic_multipmt_om(p, 0.2159, i + 1))
        else:
            targets.append(pp.HomogeneousDetector(pp.Spherical(p, 0.3), 0.05, i + 1))
    rec = torch.from_numpy(_records(pp, targets, n, poms).view(np.uint8)).cuda()
    tg = pp.detection.pmt_targets(targets)
    models, keep = pp.detection.detection_models(targets, None, True)
    lib = pp._lib.load()

    def run():
        ids = torch.full((n,), -1, dtype=torch.int32, device="cuda")
        qe = torch.full((n,), -1.0, dtype=torch.float32, device="cuda")
        rc = lib.pp_make_hits_from_photons_models(
            ctypes.c_void_p(rec.data_ptr()), n, tg, len(targets), ctypes.byref(models), 77,
            ctypes.c_void_p(ids.data_ptr()), ctypes.c_void_p(qe.data_ptr()), None)
        assert rc == 0, pp._lib.last_error()
        torch.cuda.synchronize()
        return ids.cpu().numpy(), qe.cpu().numpy()

    many = run()
    m = models.pom.contents  # a repeated last knot of the QE table: the plain kernel
    m.qe_wavelength[m.n_qe] = m.qe_wavelength[m.n_qe - 1]
    m.qe[m.n_qe] = m.qe[m.n_qe - 1]
    m.n_qe += 1
    plain = run()
    assert (plain[0] > 0).any()
    np.testing.assert_array_equal(many[0], plain[0])
    inside = plain[1] != 0  # (at the very last wavelength the repeated knot divides 0 by 0)
    np.testing.assert_array_equal(many[1][inside & np.isfinite(plain[1])],
                                  plain[1][inside & np.isfinite(plain[1])])
