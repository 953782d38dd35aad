"""After the hit buffer has overflowed no warp takes another chunk of photons."""
import numpy as np
import pytest


@pytest.mark.gpu
def test_every_warp_stops_after_its_chunk(pp, gpu_ctx):
    torch = pytest.importorskip("torch")
    medium = pp.workloads.c1_setup(photons=1, seed=1).medium
    n = 100_000_000
    # a beam onto a sphere 1 cm away: nearly every photon hits in its first step
    src = pp.PencilEmitter([0.0, 0.0, 0.0], [0.0, 0.0, 1.0], 0.0, 0.0, n)
    setup = pp.PhotonPropSetup([src], [pp.Spherical([0.0, 0.0, 10.01], 10.0)], medium,
                               pp.make_monochromatic_spectrum(450.0), 5)
    ctx = pp.Context(0)
    setup.upload(ctx)
    ctx.set_sources(setup.source_records(), 1, 1.0)
    raw = torch.empty(80, dtype=torch.uint8, device="cuda")
    ctr = torch.zeros(64, dtype=torch.uint8, device="cuda")
    ctx.launch(setup.seed, 15, raw.data_ptr(), 1, ctr.data_ptr())
    torch.cuda.synchronize()
    ctx.close()
    c = np.frombuffer(ctr.cpu().numpy().tobytes()[:48],
                      np.dtype(pp._lib.pp_counters)).copy()[0]
    assert c["err_flags"] == pp._lib.PP_FLAG_OVERFLOW
    # 16 warps an SM, 8 photons a lane and chunk; 1.1: photons that scatter first
    warps = 16 * torch.cuda.get_device_properties(0).multi_processor_count
    assert c["photon_steps"] <= 1.1 * warps * 256
