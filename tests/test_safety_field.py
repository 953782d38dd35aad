"""The culling kernel against the reference's unculled target loop, hit for hit,
on target layouts where the safety field's box and nodes can go wrong."""
import numpy as np
import pytest


def _layout(name):
    rng = np.random.default_rng(5)
    if name == "one":
        return [[0.0, 0.0, 10.0]]
    if name == "pair_far":       # two spheres at the ends of a long, thin box
        return [[-300.0, 0.0, 0.0], [300.0, 1.0, 2.0]]
    if name == "string":         # one vertical string: two axes a node or two wide
        return [[3.0, -2.0, 7.0 * k] for k in range(30)]
    if name == "plane":          # a horizontal layer: one thin axis
        return [[15.0 * i, 15.0 * j, 30.0] for i in range(9) for j in range(9)]
    if name == "offset":         # far from the origin, where coordinates are coarse
        return [[4000.0 + 20.0 * i, -3000.0 + 20.0 * j, 20.0 * k]
                for i in range(4) for j in range(4) for k in range(4)]
    return (rng.uniform(-40.0, 40.0, (300, 3))).tolist()  # "dense"


@pytest.mark.gpu
@pytest.mark.parametrize("layout", ["one", "pair_far", "string", "plane", "offset", "dense"])
@pytest.mark.parametrize("photons", [1, 33, 200_001])
def test_culled_hits_are_the_unculled_loops(pp, gpu_ctx, layout, photons):
    centres = _layout(layout)
    medium = pp.CascadiaMediumProperties(0.95, 0.2, 1.0, 1.0)
    targets = [pp.HomogeneousDetector(pp.Spherical(c, 0.5), 0.1, i + 1)
               for i, c in enumerate(centres)]
    src = [float(v) for v in np.asarray(centres[len(centres) // 2]) + [4.0, 3.0, -2.0]]
    setup = pp.PhotonPropSetup([pp.PointlikeIsotropicEmitter(src, 0.0, photons)], targets, medium,
                               pp.make_monochromatic_spectrum(450.0), 11)
    ctx = pp.get_context(0)
    got = pp.propagate_photons(setup)
    ctx.set_tuning(target_loop=1)
    try:
        want = pp.propagate_photons(setup)
    finally:
        ctx.set_tuning(target_loop=0)
    assert got.n_ph_sim == want.n_ph_sim == photons
    assert got.nrow == want.nrow and (photons < 1000 or got.nrow > 100)
    a, b = np.argsort(got["photon_index"]), np.argsort(want["photon_index"])
    for k in got:
        np.testing.assert_array_equal(got[k][a], want[k][b], err_msg=k)
