"""Photons that hit early, among others of their group that do not: the culled kernel
drops their later steps and the unculled one ends a group when all of it has hit; both
give the same hits and count the same steps."""
import numpy as np
import pytest


def _lists(pp):
    rng = np.random.default_rng(8)
    cloud = [pp.Spherical([float(c) for c in p], 3.0) for p in rng.uniform(-40, 40, (300, 3))]
    big = [pp.Spherical([0.0, 0.0, 30.0], 29.0)]
    return dict(cloud=cloud, big=big, around=big + [pp.Spherical([0.0, 0.0, -60.0], 59.5)],
                many=[pp.Spherical([float(c) for c in p], 1.0)
                      for p in rng.uniform(-40, 40, (4000, 3))])


@pytest.mark.gpu
@pytest.mark.parametrize("which", ["cloud", "big", "around", "many"])
@pytest.mark.parametrize("n, steps", [(63, 15), (20_000, 1), (20_000, 15), (5_000, 300)])
def test_same_hits_and_steps(pp, gpu_ctx, which, n, steps):
    torch = pytest.importorskip("torch")
    medium = pp.workloads.c1_setup(photons=1, seed=1).medium
    src = pp.PointlikeIsotropicEmitter([0.0, 0.0, 0.0], 0.0, n)
    setup = pp.PhotonPropSetup([src], _lists(pp)[which], medium,
                               pp.make_cherenkov_spectrum((300.0, 800.0), medium), 5)
    ctx = pp.Context(0)
    raw = torch.empty(n * 80, dtype=torch.uint8, device="cuda")
    ctr = torch.zeros(64, dtype=torch.uint8, device="cuda")
    runs = []
    for loop in (0, 1):
        ctx.set_tuning(target_loop=loop)
        setup.upload(ctx)
        ctx.set_sources(setup.source_records(), 1, 1.0)
        ctx.launch(setup.seed, steps, raw.data_ptr(), n, ctr.data_ptr())
        torch.cuda.synchronize()
        counters = ctr.cpu().numpy().view(np.uint64)[:3]
        rec = raw.cpu().numpy().view(np.dtype(pp._lib.pp_hit_record))[:int(counters[0])]
        runs.append((counters, np.sort(rec, order="photon_index").tobytes()))
    ctx.close()
    assert runs[0][0][0] > 0
    np.testing.assert_array_equal(runs[0][0], runs[1][0])
    assert runs[0][1] == runs[1][1]
