"""The automatic safety field follows the tuning that decides where the tables go, whether
that is set before the targets or after."""
import numpy as np
import pytest

NODES = {True: 48_000, False: 60 * 1500}  # staged tables, tables in global memory


def _spacing(info, nodes):
    """The automatic spacing for `nodes` over the grid's box."""
    box = np.array(info["dims"]) * np.array(info["cell"], float)
    h = np.cbrt(box.prod() / nodes)
    while (np.ceil(box / h) + 1).prod() > nodes:
        h *= 1.02
    return h


@pytest.mark.gpu
@pytest.mark.parametrize("before, after", [(dict(grid_in_global=1), dict(grid_in_global=0)),
                                           (dict(grid_in_global=0), dict(grid_in_global=1)),
                                           (dict(block_threads=64), dict(block_threads=1024))])
def test_order_of_tuning_and_targets(pp, gpu_ctx, before, after):
    rng = np.random.default_rng(3)
    targets = [pp.Spherical([float(c) for c in q], 0.2) for q in rng.uniform(-300, 300, (1500, 3))]
    medium = pp.workloads.c1_setup(photons=1, seed=1).medium
    setup = pp.PhotonPropSetup([pp.PointlikeIsotropicEmitter([0.0, 0.0, 0.0], 0.0, 20_000)], targets,
                               medium, pp.make_monochromatic_spectrum(450.0), 5)
    ctx = pp.Context(0)
    ctx.set_tuning(**before)
    setup.upload(ctx)
    ctx.set_sources(setup.source_records(), 1, 1.0)
    ctx.set_tuning(**after)
    expected = _spacing(ctx.grid_info(), NODES[not after.get("grid_in_global", 0)])
    # autotune tries 1, 0.8 and 0.6 of the field's spacing
    tuned, _ = ctx.autotune(1, 2, 20_000)
    ctx.close()
    ratios = tuned.safety_cell / expected / np.array([1.0, 0.8, 0.6])
    assert np.abs(ratios - 1.0).min() < 5e-3, (tuned.safety_cell, expected)
