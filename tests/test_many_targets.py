"""Target lists whose tables stay in global memory, with the larger safety field
that goes with them: the same hits as the loop over all targets."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1500, 2500, 9000])
def test_same_hits_as_the_unculled_loop(pp, gpu_ctx, n):
    rng = np.random.default_rng(n)
    targets = [pp.Spherical([float(c) for c in p], float(r))
               for p, r in zip(rng.uniform(-150, 150, (n, 3)), rng.uniform(0.1, 1.5, n))]
    medium = pp.workloads.c1_setup(photons=1, seed=1).medium
    setup = pp.PhotonPropSetup([pp.PointlikeIsotropicEmitter([0.0, 0.0, 0.0], 0.0, 30_000)], targets,
                               medium, pp.make_cherenkov_spectrum((300.0, 800.0), medium), 5)
    ctx = pp.Context(0)
    runs = []
    for loop in (0, 1):
        ctx.set_tuning(target_loop=loop)
        setup.upload(ctx)
        rc, hits, _ = ctx.propagate(setup.source_records(), 1, setup.seed, 15, 1.0, 30_000)
        assert rc == 0 and hits > 0  # (something to compare)
        cols = ctx.fetch_hits(hits)
        order = np.argsort(cols["photon_index"])
        runs.append({k: v[order] for k, v in cols.items()})
    ctx.close()
    for k in runs[0]:
        np.testing.assert_array_equal(runs[0][k], runs[1][k], err_msg=k)
