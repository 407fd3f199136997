"""The all-sky exposure map at the edges of its tiles (128 pixels, 64 energies, 8 and 32
cos-theta bins) against the FP64 contraction of the same livetime rows."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("nside,C,E", [(1, 40, 20), (2, 4, 1), (8, 32, 64), (8, 36, 65), (16, 64, 130), (32, 40, 256),
                                       (16, 8, 17)])
def test_exposure_map_edges(nside, C, E):
    from oracle import oracle as O
    from xtsrcmaps_b200 import api as A
    from xtsrcmaps_b200.synth import make_job

    A.init(0)
    job = make_job("c0", seed=2)
    rng = np.random.default_rng(nside)
    logEs = np.linspace(2.0, 6.0, E) if E > 1 else np.array([3.0])
    x = rng.lognormal(12.0, 0.2, (12 * nside * nside, C)).astype(np.float32)
    w = rng.lognormal(12.0, 0.2, (12 * nside * nside, C)).astype(np.float32)
    ltf = O.livetime_efficiency_factors(logEs, job.effic_front.p0, job.effic_front.p1)
    m = A.exposure_map(A.ExpCube(x, nside, C), A.ExpCube(w, nside, C), logEs, job.aeff_front, job.aeff_back, ltf)
    cos = O.costhetas(C, 0.0, True)
    af, ab = O.aeff_value(cos, logEs, job.aeff_front), O.aeff_value(cos, logEs, job.aeff_back)
    ref = O.exposure(x.astype(np.float64), w.astype(np.float64), af, ab, ltf)
    assert m.shape == ref.shape
    assert np.max(np.abs(m - ref) / np.abs(ref).max(axis=0)) < 5e-6
