"""The host memory of a context's small uploads and results: hits fetched across the call
from which it is pinned, with small and large source lists in turn."""
import numpy as np
import pytest


def _setup(pp, n):
    medium = pp.workloads.c1_setup(photons=1, seed=1).medium
    rng = np.random.default_rng(n)
    src = [pp.PointlikeIsotropicEmitter([float(c) for c in p], 0.0, 2000 // n + 1)
           for p in rng.uniform(-1, 1, (n, 3))]
    return pp.PhotonPropSetup(src, [pp.Spherical([0.0, 0.0, 6.0], 3.0)], medium,
                              pp.make_monochromatic_spectrum(450.0), 5)


@pytest.mark.gpu
def test_hits_survive_the_change(pp, gpu_ctx):
    setups = [_setup(pp, n) for n in (1, 40, 5000)]  # the last is larger than the image
    records = [s.source_records() for s in setups]
    ctx = pp.Context(0)
    setups[0].upload(ctx)
    want = [None] * len(setups)
    for call in range(150):
        i = call % len(setups)
        rc, hits, sim = ctx.propagate(records[i], len(setups[i].sources), 7, 15, 1.0, 100_000)
        assert rc == 0 and hits > 0 and sim == sum(s.photons for s in setups[i].sources)
        # other sources are uploaded before the hits are fetched
        j = (call + 1) % len(setups)
        ctx.set_sources(records[j], len(setups[j].sources), 1.0)
        cols = ctx.fetch_hits(hits)
        order = np.lexsort((cols["photon_index"], cols["source_index"]))
        got = {k: v[order] for k, v in cols.items()}
        want[i] = want[i] or got
        for k in got:
            np.testing.assert_array_equal(got[k], want[i][k], err_msg=f"call {call}: {k}")
    ctx.close()

