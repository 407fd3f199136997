"""The write pass's pixel pairs at the edges of its tiles: odd heights, rows narrower and
wider than a warp, energy counts of every residue modulo 4, sources in and beside the map;
dense maps and cutouts against the FP64 maps of the same tables."""
import numpy as np
import pytest

from helpers import max_rel


def _tables(S, E, H, W, pix):
    from xtsrcmaps_b200 import api as A
    from xtsrcmaps_b200.synth import make_job
    from xtsrcmaps_b200.wcs import Wcs

    A.init(0)
    job = make_job("c1", seed=9, n_sources=S)
    job.logEs = np.linspace(2.0, 6.0, E) if E > 1 else np.array([3.0])
    w = job.wcs
    wcs = Wcs(H, W, (H + 1) / 2.0, (W + 1) / 2.0, w.crval1, w.crval2, -pix, pix)
    rng = np.random.default_rng(H * 100 + W)  # around the map, a third of them beside it
    src = np.array([w.crval1, w.crval2]) + rng.uniform(-0.75, 0.75, (S, 2)) * np.array([H * pix, W * pix])
    ltf = A.livetime_efficiency_factors(job.logEs, job.effic_front)
    nf = A.normalize_rpsf(job.rpsf_front, job.scale_front)
    nb = A.normalize_rpsf(job.rpsf_back, job.scale_back)
    ex = A.compute_exposure(job.exp_cube, job.wexp_cube, job.logEs, src, job.aeff_front, job.aeff_back, ltf)
    ps = A.compute_psf_data(nf, nb, ex, job.logEs, ltf)
    return A, wcs, src, ex.exposure, ps.uPsf, ps.partial_psf_integral


@pytest.mark.gpu
@pytest.mark.parametrize("H,W,E,pix", [(33, 31, 5, 0.1), (7, 32, 4, 0.1), (64, 33, 6, 0.05), (35, 65, 37, 0.2),
                                       (1, 40, 1, 0.1), (40, 1, 3, 0.1), (50, 61, 52, 0.025), (129, 514, 8, 0.1),
                                       (2, 1100, 15, 0.05)])
def test_pair_tiles(H, W, E, pix):
    A, wcs, src, ex, u, p = _tables(5, E, H, W, pix)
    m32, _ = A.point_src_model_map_wcs(wcs, src, ex, u, p)
    m64, _ = A.point_src_model_map_wcs(wcs, src, ex, u, p, out_dtype="float64")
    assert np.isfinite(m32).all()
    assert max_rel(m32, m64) < 1e-5


@pytest.mark.gpu
@pytest.mark.parametrize("E", [5, 8, 50])
def test_pair_tiles_cutouts(E):
    A, wcs, src, ex, u, p = _tables(9, E, 61, 97, 0.1)
    rad = np.array([0.05, 0.2, 0.5, 1.0, 1.55, 1.6, 2.0, 3.0, 8.0])  # 1 to 97 pixels wide
    cut, total = A.cutout_windows(wcs, src, rad)
    m, _ = A.point_src_model_map_cutouts(wcs, src, cut, ex, u, p)
    assert m.shape == (total, E)
    from xtsrcmaps_b200.wcs import Wcs

    for s, c in enumerate(cut):
        if c["nh"] == 0 or c["nw"] == 0:
            continue
        sub = Wcs(int(c["nh"]), int(c["nw"]), wcs.crpix1 - int(c["h0"]), wcs.crpix2 - int(c["w0"]), wcs.crval1,
                  wcs.crval2, wcs.cdelt1, wcs.cdelt2)
        r, _ = A.point_src_model_map_wcs(sub, src[s:s + 1], ex[s:s + 1], u[s:s + 1], p[s:s + 1], out_dtype="float64")
        n = int(c["nh"]) * int(c["nw"])
        got = m[int(c["offset"]):int(c["offset"]) + n].reshape(r[0].shape)
        assert max_rel(got, r[0]) < 1e-5
