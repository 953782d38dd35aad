"""Many sources of few photons share groups of 64: the hits must be those of the same
sources in groups of their own, which a last source of many photons brings about, and,
photon by photon, the oracle's."""
import numpy as np
import pytest

import replay
from test_zz_no_alloc import _records_to_columns, _static_call

FIELDS = ("position", "direction", "initial_direction", "wavelength", "time", "dist_travelled",
          "abs_weight", "module_index", "n_steps", "source_index", "photon_index")
BOUNDARY = 1 << 32


def _sources(pp, n, most):
    rng = np.random.default_rng(n + most)
    lp = pp.LongitudinalParameterisation(2.0, 0.63, 0.36)
    out = []
    for i, p in enumerate(rng.uniform(-6, 6, (n, 3))):
        p, count = [float(c) for c in p], int(rng.integers(0, most + 1))
        out.append(pp.PointlikeIsotropicEmitter(p, 0.0, count) if i % 2 else
                   pp.ExtendedCherenkovEmitter(p, [0.0, 0.0, 1.0], 0.0, count, lp))
        # some ranges cross the step of the photon counter's high word
        out[-1].first_photon = [0, 17, BOUNDARY - 3, BOUNDARY + 5][i % 4]
    return out


def _targets(pp, shaped):
    rng = np.random.default_rng(1)
    at = [[float(c) for c in p] for p in rng.uniform(-12, 12, (24, 3))]
    return [pp.Circular(p, 2.0) if shaped and i % 2 else pp.Spherical(p, 1.5)
            for i, p in enumerate(at)]


def _sorted(cols, n_src):
    keep = np.asarray(cols["source_index"]) < n_src
    order = np.lexsort((np.asarray(cols["photon_index"])[keep],
                        np.asarray(cols["source_index"])[keep]))
    return {k: np.asarray(cols[k])[keep][order] for k in FIELDS}


@pytest.mark.gpu
@pytest.mark.parametrize("n, most", [(2500, 3), (5000, 40), (4000, 100), (20_000, 1)])
@pytest.mark.parametrize("shaped", [False, True])
def test_same_hits_as_in_groups_of_their_own(pp, gpu_ctx, n, most, shaped):
    torch = pytest.importorskip("torch")
    medium = pp.workloads.c1_setup(photons=1, seed=1).medium
    spectrum = pp.make_cherenkov_spectrum((300.0, 800.0), medium)
    src, targets = _sources(pp, n, most), _targets(pp, shaped)
    far = pp.PointlikeIsotropicEmitter([0.0, 0.0, 5000.0], 0.0, 20_000_000)
    ctx = pp.Context(0)
    runs = []
    for sources in (src, src + [far]):
        setup = pp.PhotonPropSetup(sources, targets, medium, spectrum, 5)
        setup.upload(ctx)
        total = sum(s.photons for s in sources)
        rc, hits, sim = ctx.propagate(setup.source_records(), len(sources), setup.seed, 15, 1.0,
                                      1_000_000)
        assert rc == 0 and sim == total and hits > 0
        runs.append(_sorted(ctx.fetch_hits(hits), n))
    ctx.close()
    if not shaped:
        setup = pp.PhotonPropSetup(src, targets, medium, spectrum, 5)
        raw = torch.empty(1_000_000 * 80, dtype=torch.uint8, device="cuda")
        rc, ctr = _static_call(pp, setup, raw.data_ptr(), 1_000_000)
        assert rc == 0 and ctr.n_ph_sim == sum(s.photons for s in src)
        runs.append(_sorted(_records_to_columns(pp, raw.cpu().numpy(), int(ctr.n_hits)), n))
    for k in FIELDS:
        for run in runs[1:]:
            np.testing.assert_array_equal(runs[0][k], run[k], err_msg=k)


@pytest.mark.gpu
def test_against_the_oracle(pp, orc, gpu_ctx):
    medium = pp.workloads.c1_setup(photons=1, seed=1).medium
    modules = [pp.HomogeneousDetector(t, 0.1, i + 1) for i, t in enumerate(_targets(pp, False))]
    setup = pp.PhotonPropSetup(_sources(pp, 3000, 12), modules, medium,
                               pp.make_cherenkov_spectrum((300.0, 800.0), medium), 5)
    ctx = pp.get_context(0)
    ctx.set_tuning(precise_math=1)
    try:
        table = pp.propagate_photons(setup)
    finally:
        ctx.set_tuning(precise_math=0)
    ref, sim, _ = orc.Run.from_setup(setup).propagate_all()
    assert table.n_ph_sim == sim
    got = dict(table)
    got["module_index"] = got["module_id"].astype("int32")
    stats = replay.compare(got, replay.oracle_columns(ref), replay.spheres_of(setup),
                           mode="precise")
    assert stats["matched"] > 0, stats


@pytest.mark.gpu
def test_histograms_of_their_own_sources(pp, gpu_ctx):
    """Tables of many pairs of few photons: a pair's counts are its hits' weights."""
    S = pp.surrogate
    n, photons, seed = 4000, 40, 3
    pairs = S.sample_pairs(n, seed=11)
    pairs.distance[:] = 0.5 + 0.5 * np.random.default_rng(2).random(n)  # close: many hits
    ctx = pp.Context(0)
    counts, hists = S.generate_tables(pairs, photons, seed=seed, ctx=ctx, n_steps=15)
    rc, hits, _ = ctx.propagate(S.cascade_records(pairs, photons), n, seed, 15, 1.0, n * photons)
    cols = ctx.fetch_hits(hits)
    ctx.close()
    assert rc == 0 and hits > 500
    want = np.bincount(cols["source_index"], cols["abs_weight"].astype(float), n)
    np.testing.assert_allclose(counts, want, rtol=1e-5)
    np.testing.assert_allclose(hists.sum(1), want, rtol=1e-5)
