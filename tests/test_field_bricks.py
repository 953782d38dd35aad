"""The safety field's bricks of nodes: spheres that fit a brick's list, more than fit (all
of them passed over again, or the distance from the brick's centre in a large field),
nodes beyond what a byte holds, boxes of few nodes and far from the origin.  Never a
hit less than in the loop over all targets, in either entry point."""
import numpy as np
import pytest

from test_zz_no_alloc import _records_to_columns, _static_call


def _scene(which):
    """(sphere centres, radius, emitter, photons, safety spacing)"""
    rng = np.random.default_rng(5)
    corners = np.array([[-200.0] * 3, [200.0] * 3])

    def cluster(n, half, at):
        return np.concatenate([corners, at + rng.uniform(-half, half, (n, 3))])

    if which == "cluster, all again":
        return cluster(3000, 15.0, np.zeros(3)), 0.2, [0.0, 0.0, -40.0], 20_000, 0.0
    if which == "cluster, large field":
        return cluster(18_500, 20.0, np.array([50.0, 0.0, 0.0])), 0.15, [50.0, 0.0, 30.0], 10_000, 0.0
    if which == "wide spacing":
        return rng.uniform(-100, 100, (2500, 3)), 0.5, [0.0, 0.0, 0.0], 20_000, 60.0
    if which == "one":
        return np.array([[0.0, 0.0, 12.0]]), 3.0, [0.0, 0.0, 0.0], 20_000, 0.0
    if which == "three kilometres apart":
        return np.array([[0.0, 0.0, 10.0], [3000.0, 100.0, 0.0]]), 3.0, [0.0, 0.0, 0.0], 20_000, 0.0
    assert which == "far from the origin"
    at = np.array([30_000.0, -20_000.0, 10_000.0])
    return at + rng.uniform(-60, 60, (2000, 3)), 1.0, list(at), 20_000, 0.0


@pytest.mark.gpu
@pytest.mark.parametrize("which", ["cluster, all again", "cluster, large field", "wide spacing", "one",
                                   "three kilometres apart", "far from the origin"])
def test_same_hits_as_the_unculled_loop(pp, gpu_ctx, which):
    torch = pytest.importorskip("torch")
    centres, r, place, n, spacing = _scene(which)
    targets = [pp.Spherical([float(c) for c in q], r) for q in centres]
    medium = pp.workloads.c1_setup(photons=1, seed=1).medium
    src = pp.PointlikeIsotropicEmitter([float(c) for c in place], 0.0, n)
    setup = pp.PhotonPropSetup([src], targets, medium, pp.make_monochromatic_spectrum(450.0), 5)
    ctx = pp.Context(0)
    runs = []
    for loop in (0, 1):
        ctx.set_tuning(target_loop=loop, safety_cell=spacing)
        setup.upload(ctx)
        rc, hits, _ = ctx.propagate(setup.source_records(), 1, setup.seed, 15, 1.0, n)
        assert rc == 0 and hits > 0  # (something to compare)
        runs.append(ctx.fetch_hits(hits))
    ctx.close()
    raw = torch.empty(n * 80, dtype=torch.uint8, device="cuda")
    rc, ctr = _static_call(pp, setup, raw.data_ptr(), n)
    assert rc == 0, pp._lib.last_error()
    runs.append(_records_to_columns(pp, raw.cpu().numpy(), int(ctr.n_hits)))
    order = [np.argsort(run["photon_index"]) for run in runs]
    for k in runs[0]:
        for run, o in zip(runs[1:], order[1:]):
            np.testing.assert_array_equal(runs[0][k][order[0]], run[k][o], err_msg=k)
