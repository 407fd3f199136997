"""The window pass's wide pixels (next to a source), put off to the end of a work item: a
source on a pixel's corner, edge and centre, maps of a few pixels, and more wide pixels in
an item than its list holds (64 sources within three pixels of each other, eight to a
group); dense maps and cutouts against the FP64 maps of the same tables, whose window code
is another.  Tolerance 1e-5: the FP32 window path's rounding, as for every other map."""
import numpy as np
import pytest

from helpers import max_rel

pytestmark = pytest.mark.gpu


def _job(H, W, pix, offsets, E=3):
    from xtsrcmaps_b200 import api as A
    from xtsrcmaps_b200.synth import make_job
    from xtsrcmaps_b200.wcs import Wcs

    A.init(0)
    job = make_job("c1", seed=9, n_sources=1)
    w = job.wcs
    wcs = Wcs(H, W, (H + 1) / 2.0, (W + 1) / 2.0, w.crval1, w.crval2, -pix, pix)
    off = np.asarray(offsets, np.float64) * pix
    src = np.stack([w.crval1 + off[:, 0] / np.cos(np.deg2rad(w.crval2)), w.crval2 + off[:, 1]], 1)
    logEs = np.linspace(2.0, 6.0, E)
    ltf = A.livetime_efficiency_factors(logEs, job.effic_front)
    nf = A.normalize_rpsf(job.rpsf_front, job.scale_front)
    nb = A.normalize_rpsf(job.rpsf_back, job.scale_back)
    ex = A.compute_exposure(job.exp_cube, job.wexp_cube, logEs, src, job.aeff_front, job.aeff_back, ltf)
    ps = A.compute_psf_data(nf, nb, ex, logEs, ltf)
    return A, wcs, src, ex.exposure, ps.uPsf, ps.partial_psf_integral


@pytest.mark.parametrize("H,W,pix,n", [(5, 3, 0.2, 4), (33, 32, 0.2, 5), (200, 200, 0.05, 50), (900, 64, 0.05, 64)])
def test_wide_pixels(H, W, pix, n):
    rng = np.random.default_rng(n)
    off = rng.uniform(-1.5, 1.5, (n, 2))
    off[:4] = [[0.0, 0.0], [0.5, 0.5], [0.5, 0.0], [0.01, 0.02]]
    A, wcs, src, ex, u, p = _job(H, W, pix, off)
    m32, _ = A.point_src_model_map_wcs(wcs, src, ex, u, p)
    m64, _ = A.point_src_model_map_wcs(wcs, src, ex, u, p, out_dtype="float64")
    assert np.isfinite(m32).all()
    assert max_rel(m32, m64) < 1e-5
    cut, total = A.cutout_windows(wcs, src, np.full(n, 2.2 * pix))
    mc, _ = A.point_src_model_map_cutouts(wcs, src, cut, ex, u, p)
    from xtsrcmaps_b200.wcs import Wcs

    for s in range(4):
        c = cut[s]
        sub = Wcs(int(c["nh"]), int(c["nw"]), wcs.crpix1 - int(c["h0"]), wcs.crpix2 - int(c["w0"]), wcs.crval1,
                  wcs.crval2, wcs.cdelt1, wcs.cdelt2)
        r, _ = A.point_src_model_map_wcs(sub, src[s:s + 1], ex[s:s + 1], u[s:s + 1], p[s:s + 1], out_dtype="float64")
        k = int(c["nh"]) * int(c["nw"])
        assert max_rel(mc[int(c["offset"]):int(c["offset"]) + k].reshape(r[0].shape), r[0]) < 1e-5
