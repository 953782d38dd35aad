"""Cell sizes of grid and safety field far below what can be held are made coarser until
they can."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("cell, spacing", [(1e-9, 0.0), (0.0, 1e-9), (1e-6, 1e-6), (1e-20, 1e-20)])
def test_same_hits(pp, gpu_ctx, cell, spacing):
    rng = np.random.default_rng(3)
    targets = [pp.Spherical([float(c) for c in q], 1.0) for q in rng.uniform(-250, 250, (300, 3))]
    medium = pp.workloads.c1_setup(photons=1, seed=1).medium
    setup = pp.PhotonPropSetup([pp.PointlikeIsotropicEmitter([0.0, 0.0, 0.0], 0.0, 200_000)],
                               targets, medium, pp.make_monochromatic_spectrum(450.0), 5)
    ctx = pp.Context(0)
    runs = []
    for tuning in (dict(), dict(cell_size=cell, safety_cell=spacing)):
        ctx.set_tuning(**tuning)
        setup.upload(ctx)
        assert np.prod(ctx.grid_info()["dims"], dtype=float) <= 4 * 1024 ** 2
        rc, hits, _ = ctx.propagate(setup.source_records(), 1, setup.seed, 15, 1.0, 200_000)
        assert rc == 0 and hits > 0
        cols = ctx.fetch_hits(hits)
        order = np.argsort(cols["photon_index"])
        runs.append({k: v[order] for k, v in cols.items()})
    ctx.close()
    for k in runs[0]:
        np.testing.assert_array_equal(runs[0][k], runs[1][k], err_msg=k)
