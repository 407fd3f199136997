"""Mean-PSF tables at the edges of the kernel's tiles (4 or 8 sources, 1 or 4 energies,
40 cos-theta bins per group) against the FP64 oracle."""
import numpy as np
import pytest

from helpers import max_rel, oracle_pipeline


@pytest.mark.gpu
@pytest.mark.parametrize("S,E,C", [(1, 1, 40), (3, 5, 40), (5, 37, 40), (41, 41, 40), (97, 93, 40), (9, 6, 41),
                                   (4, 4, 64), (6, 3, 3)])
def test_mean_psf_tile_edges(S, E, C):
    from xtsrcmaps_b200 import api as A
    from xtsrcmaps_b200.synth import make_job

    A.init(0)
    job = make_job("c1", seed=3, n_sources=S)
    job.energies = np.logspace(2, 6, E) if E > 1 else np.array([1e3])
    job.logEs = np.log10(job.energies)
    for cube in (job.exp_cube, job.wexp_cube):  # C bins from the 40 of the job, repeated as needed
        cube.cosbins = np.ascontiguousarray(np.tile(cube.cosbins, (1, 2))[:, :C])
        cube.nbrbins = C
    o = oracle_pipeline(job, with_map=False)
    ltf = A.livetime_efficiency_factors(job.logEs, job.effic_front)
    nf = A.normalize_rpsf(job.rpsf_front, job.scale_front)
    nb = A.normalize_rpsf(job.rpsf_back, job.scale_back)
    ex = A.compute_exposure(job.exp_cube, job.wexp_cube, job.logEs, job.src_sph, job.aeff_front, job.aeff_back, ltf)
    ps = A.compute_psf_data(nf, nb, ex, job.logEs, ltf)
    assert max_rel(ps.uPsf, o["upsf"]) < 1e-11
    assert max_rel(ps.partial_psf_integral, o["partial"], floor=1e-300) < 1e-11
