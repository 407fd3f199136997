"""FP32 maps with more wide pixels than the sparse pool holds (65,536 and an eighth of the map):
two sources more than 70 degrees away, every pixel's points past the separation table.  The
last pixels are evaluated point by point in the write pass.  Against the FP64 maps of the same
tables, which rise with the separation; 1e-5, as for every FP32 map."""
import numpy as np
import pytest

from helpers import max_rel


@pytest.mark.gpu
@pytest.mark.parametrize("E", [1, 6, 37])
def test_more_wide_pixels_than_records(E):
    from xtsrcmaps_b200 import api as A
    from xtsrcmaps_b200.wcs import Wcs

    A.init(0)
    H, W = 300, 261
    wcs = Wcs(H, W, (H + 1) / 2.0, (W + 1) / 2.0, 120.0, 0.0, -0.1, 0.1)
    src = np.array([[215.0, 0.0], [15.0, 4.0]])
    sep = np.concatenate([[0.0], 1e-4 * np.exp(np.arange(400) * np.log(70.0 / 1e-4) / 399.0)])
    u = np.repeat(1.0 + sep[None, :, None] * np.linspace(0.3, 2.0, E)[None, None], 2, axis=0)
    part = np.cumsum(u, axis=1)
    part /= part[:, -1:]
    ex = np.full((2, E), 1e11)
    m32, _ = A.point_src_model_map_wcs(wcs, src, ex, u, part)
    m64, _ = A.point_src_model_map_wcs(wcs, src, ex, u, part, out_dtype="float64")
    assert np.isfinite(m32).all()
    assert max_rel(m32, m64) < 1e-5
