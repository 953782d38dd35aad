"""The column-wise conversions of emitters and modules against the element-wise
ones they stand in for."""
import numpy as np
import pytest


def _emitters(pp, n):
    rng = np.random.default_rng(4)
    lp = pp.LongitudinalParameterisation(2.0, 0.63, 0.36)
    out = []
    for i in range(n):
        p, d = rng.normal(size=3), rng.normal(size=3)
        p = [list(p), tuple(p), p.astype(np.float32), p.reshape(3, 1)][i % 4]
        out.append([pp.PointlikeIsotropicEmitter(p, 0.1 * i, 1000 + i),
                    pp.ExtendedCherenkovEmitter(p, d, 0.2, 2000 + i, lp),
                    pp.CherenkovTrackEmitter(p, list(d), 0.3, 55.5, 3000.0 + i),
                    pp.PencilEmitter(p, d, 0.01, 0.4, 4000 + i)][i // 2 % 4])
        out[-1].first_photon = 17 * i
    return out


@pytest.mark.parametrize("n", [0, 1, 7, 8, 61, 200])
def test_emitter_records(pp, n):
    from pp_gb300 import _lib, sources
    src = _emitters(pp, n)
    got = sources.to_records(src)
    assert len(got) == max(1, n)
    for i, s in enumerate(src):
        assert bytes(got[i]) == bytes(s.to_record()), i
    if n:
        got[0].smear_table = 3  # the array is writable element by element
        assert got._keep["smear_table"][0] == 3
    assert isinstance(got[0], _lib.pp_source)


@pytest.mark.parametrize("same", [True, False])
def test_module_records(pp, same):
    class MyPOM(pp.POM):
        pass

    pos = [[1.5, -2.25, 3.1], [0.1, 0.2, 0.3], [7.0, 8.0, 9.0], [4.0, 5.0, 6.0]]
    if not same:  # positions of different array shapes
        pos[1] = np.array(pos[1]).reshape(3, 1)
    targets = [MyPOM.at(pos[0], 1), pp.DOM.at(pos[1], 2),
               pp.make_generic_multipmt_om(pos[2], 0.2159, 3),
               pp.HomogeneousDetector(pp.Spherical(pos[3], 0.3), 0.05, 4)]
    got = pp.detection.pmt_targets(targets)
    for t, r, kind in zip(targets, got, (1, 2, 3, 0)):
        want = np.asarray(t.shape.position, np.float32).reshape(3)
        assert list(r.position) == [float(v) for v in want]
        assert r.radius == np.float32(t.shape.radius) and r.kind == kind
        assert r.active_area == np.float32(t.pmt_area)
    with pytest.raises(TypeError, match="target 1: no detection model"):
        pp.detection.pmt_targets([targets[0], pp.Spherical([0, 0, 0], 1.0)])
