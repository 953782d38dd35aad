"""Shaped targets at launch shapes on both sides of the largest CTA they use: the same
hits, whatever the warps of a CTA and the CTAs of an SM."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("lines", [False, True])
def test_same_hits_at_every_launch_shape(pp, gpu_ctx, lines):
    rng = np.random.default_rng(4)
    p = [[float(c) for c in q] for q in rng.uniform(-30, 30, (30, 3))]
    if lines:
        targets = pp.DetectorLines([
            pp.DetectorLine(q[0], q[1], 3.0, [pp.Spherical([q[0], q[1], -20.0 + 5.0 * i], 1.5)
                                              for i in range(8)]) for q in p[:10]])
    else:
        targets = [pp.Circular(q, 3.0) for q in p[:10]]
        targets += [pp.Rectangular(q, 4.0, 2.0) for q in p[10:20]]
        targets += [pp.Spherical(q, 2.0) for q in p[20:]]
    medium = pp.workloads.c1_setup(photons=1, seed=1).medium
    src = pp.PointlikeIsotropicEmitter([0.0, 0.0, 0.0], 0.0, 30_000)
    setup = pp.PhotonPropSetup([src], targets, medium, pp.make_monochromatic_spectrum(450.0), 5)
    ctx = pp.Context(0)
    setup.upload(ctx)
    want = None
    for block in (64, 224, 256, 288, 1024):
        for ctas in (0, 1, 3):
            ctx.set_tuning(block_threads=block, ctas_per_sm=ctas)
            rc, hits, sim = ctx.propagate(setup.source_records(), 1, setup.seed, 15, 1.0, 30_000)
            assert rc == 0 and hits > 0 and sim == 30_000  # (something to compare)
            cols = ctx.fetch_hits(hits)
            order = np.argsort(cols["photon_index"])
            got = {k: v[order] for k, v in cols.items()}
            want = want or got
            for k in want:
                np.testing.assert_array_equal(got[k], want[k], err_msg=f"{k} {block} {ctas}")
    ctx.close()
