"""A mean-PSF table with a row that is not finite, a source beside the map (its values are the
table's times the exposure): the values of the pixels whose points touch that row are not
finite, all others are what they are without it.  FP32 maps (dense, cutouts) against the FP64
maps of the same table, whose windows are other code; tolerance 1e-5, as for every FP32 map."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _job(E, bad, row):
    from xtsrcmaps_b200 import api as A
    from xtsrcmaps_b200.wcs import Wcs

    A.init(0)
    H, W, pix = 45, 52, 0.1
    wcs = Wcs(H, W, (H + 1) / 2.0, (W + 1) / 2.0, 120.0, -5.0, -pix, pix)
    src = np.array([[124.0, -5.0], [120.0, -9.5]])  # 1.8 and 1.9 degrees outside
    sep = np.concatenate([[0.0], 1e-4 * np.exp(np.arange(400) * np.log(70.0 / 1e-4) / 399.0)])
    d = sep[None, :, None]
    w = np.linspace(0.5, 3.0, E)[None, None, :]
    u = np.repeat((1.0 + (d / w) ** 2) ** -2.0 / w ** 2, 2, axis=0)
    part = np.cumsum(u, axis=1)
    part /= part[:, -1:]
    clean = u.copy()
    u[0, row, E // 2] = bad
    ex = np.full((2, E), 1e11)
    return A, wcs, src, ex, u, clean, part, sep


def _same(got, want, clean, bad):
    """got is not finite where want is, and what the clean table gives elsewhere."""
    fin = np.isfinite(want)
    assert 20 < (~fin).sum() < fin.sum()
    np.testing.assert_array_equal(np.isfinite(got), fin)
    np.testing.assert_allclose(got[fin], clean[fin], rtol=1e-5)
    if np.isinf(bad):
        assert not np.isnan(got).any()


@pytest.mark.parametrize("E", [1, 6, 8, 37])  # a stage of 4, 8 and 16 bytes per store
@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_dense_and_cutouts(E, bad):
    A, wcs, src, ex, u, clean, part, sep = _job(E, bad, row=318)
    m64, _ = A.point_src_model_map_wcs(wcs, src, ex, u, part, out_dtype="float64")
    c64, _ = A.point_src_model_map_wcs(wcs, src, ex, clean, part, out_dtype="float64")
    m32, _ = A.point_src_model_map_wcs(wcs, src, ex, u, part)
    _same(m32, m64, c64, bad)
    cut, total = A.cutout_windows(wcs, src, np.array([60.0, 60.0]))  # the whole map
    assert total == 2 * m32[0].size // E
    mc, _ = A.point_src_model_map_cutouts(wcs, src, cut, ex, u, part)
    _same(mc.reshape(m64.shape), m64, c64, bad)
