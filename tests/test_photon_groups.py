"""Photon ranges that end inside a warp's group of 64 or cross the step where the
photon counter's high word changes: the hits must be those of the same photons
run as separate sources."""
import numpy as np
import pytest

BOUNDARY = 1 << 32


@pytest.mark.gpu
@pytest.mark.parametrize("first, n", [(0, 63), (0, 64), (0, 65), (7, 129), (BOUNDARY - 40, 100),
                                      (BOUNDARY - 1, 64), (BOUNDARY - 64, 64), (BOUNDARY - 97, 5000)])
def test_ranges_equal_their_parts(pp, gpu_ctx, first, n):
    medium = pp.CascadiaMediumProperties(0.95, 0.2, 1.0, 1.0)
    targets = [pp.HomogeneousDetector(pp.Spherical([0.0, 0.0, 10.0], 5.0), 0.1, 1),
               pp.HomogeneousDetector(pp.Spherical([0.0, -12.0, 0.0], 4.0), 0.1, 2)]
    spec = pp.make_monochromatic_spectrum(450.0)

    def run(lo, count):
        src = pp.PointlikeIsotropicEmitter([0.0, 0.0, 0.0], 0.0, count)
        src.first_photon = lo
        return pp.propagate_photons(pp.PhotonPropSetup([src], targets, medium, spec, 3))

    whole = run(first, n)
    assert whole.n_ph_sim == n and whole.nrow > 0
    cuts = sorted({first, first + n // 3, min(max(first, BOUNDARY), first + n), first + n})
    parts = [run(lo, hi - lo) for lo, hi in zip(cuts, cuts[1:]) if hi > lo]
    order = np.argsort(whole["photon_index"])
    for k in ("photon_index", "position", "direction", "wavelength", "time", "dist_travelled",
              "n_steps", "module_id"):
        joined = np.concatenate([p[k] for p in parts])
        index = np.argsort(np.concatenate([p["photon_index"] for p in parts]))
        np.testing.assert_array_equal(whole[k][order], joined[index], err_msg=k)
