"""A dense cluster in a wide target list: more spheres in one automatic grid cell than
its count can hold, as long as the cells are those of the usual density."""
import numpy as np
import pytest

from test_zz_no_alloc import _records_to_columns, _static_call

MAX_COUNT = 4095


def _targets(pp, n=5000):
    """n spheres in one of the 8 n cells of the box that two far spheres span."""
    r, margin, half = 0.05, 0.01, 170.0
    edge = 2.0 * (half + r + margin)
    cell = edge / (8.0 * (n + 2)) ** (1 / 3)
    lo = 17 * cell - 0.5 * edge  # the cell's lower corner
    p = np.random.default_rng(2).uniform(lo + 0.1, lo + cell - 0.1, (n, 3))
    fine = edge / (16.0 * (n + 2)) ** (1 / 3)
    ids = np.floor((p + 0.5 * edge) / fine).astype(int)
    assert np.unique(ids, axis=0, return_counts=True)[1].max() < MAX_COUNT - 200 < n
    centres = [[-half] * 3, [half] * 3] + [[float(c) for c in q] for q in p]
    return [pp.Spherical(c, r) for c in centres], lo + 0.5 * cell


@pytest.mark.gpu
def test_accepted_with_the_hits_of_the_unculled_loop(pp, gpu_ctx):
    torch = pytest.importorskip("torch")
    targets, middle = _targets(pp)
    medium = pp.workloads.c1_setup(photons=1, seed=1).medium
    src = pp.PointlikeIsotropicEmitter([middle, middle, middle - 15.0], 0.0, 20_000)
    setup = pp.PhotonPropSetup([src], targets, medium, pp.make_monochromatic_spectrum(450.0), 5)
    ctx = pp.Context(0)
    runs = []
    for loop in (0, 1):
        ctx.set_tuning(target_loop=loop)
        setup.upload(ctx)
        rc, hits, _ = ctx.propagate(setup.source_records(), 1, setup.seed, 15, 1.0, 20_000)
        assert rc == 0 and hits > 100
        runs.append(ctx.fetch_hits(hits))
    ctx.close()
    raw = torch.empty(20_000 * 80, dtype=torch.uint8, device="cuda")
    rc, ctr = _static_call(pp, setup, raw.data_ptr(), 20_000)
    assert rc == 0, pp._lib.last_error()
    runs.append(_records_to_columns(pp, raw.cpu().numpy(), int(ctr.n_hits)))
    order = [np.argsort(r["photon_index"]) for r in runs]
    for k in runs[0]:
        for r, o in zip(runs[1:], order[1:]):
            np.testing.assert_array_equal(runs[0][k][order[0]], r[k][o], err_msg=k)


@pytest.mark.gpu
def test_refused_cell_size_leaves_no_targets(pp, gpu_ctx):
    """A cell size that is refused leaves no tables: launches are refused too, until
    another one is set."""
    targets, middle = _targets(pp)
    medium = pp.workloads.c1_setup(photons=1, seed=1).medium
    src = pp.PointlikeIsotropicEmitter([middle, middle, middle - 15.0], 0.0, 20_000)
    setup = pp.PhotonPropSetup([src], targets, medium, pp.make_monochromatic_spectrum(450.0), 5)
    ctx = pp.Context(0)
    setup.upload(ctx)

    def run():
        return ctx.propagate(setup.source_records(), 1, setup.seed, 15, 1.0, 20_000)

    want = run()
    assert want[1] > 0
    with pytest.raises(pp._lib.PPError, match="too dense"):
        ctx.set_tuning(cell_size=500.0)
    with pytest.raises(pp._lib.PPError, match="tables are not built"):
        run()
    ctx.set_tuning(cell_size=0.0)
    assert run() == want
    ctx.close()
