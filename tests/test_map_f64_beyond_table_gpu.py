"""FP64 maps where rule points lie beyond the separation table, past 70 degrees or below 1e-4
degrees: whole pixels, pixels with a part of their points there, the whole sky.  The tables
rise with the separation, so that the extrapolated values do not cross zero.

Past 70 degrees against the FP64 oracle (1e-10, as for the other FP64 maps).  Pixels of 1e-5
degrees, whose solid angles carry the rounding of the directions (1e-16 of a radian on sides
of 2e-7), and the whole sky, where pixels outside the projection have no solid angle, against
the FP32 maps, which share the geometry (1e-5, the FP32 maps' rounding)."""
import numpy as np
import pytest

from helpers import max_rel

pytestmark = pytest.mark.gpu


def _job(H, W, pix, proj, sep, E):
    from oracle import oracle as O
    from xtsrcmaps_b200 import api as A
    from xtsrcmaps_b200.wcs import Wcs

    A.init(0)
    wcs = Wcs(H, W, (H + 1) / 2.0, (W + 1) / 2.0, 120.0, 0.0, -pix, pix, proj=proj)
    src = np.array([[120.0 + sep, 0.0], [120.0 - 0.5 * sep, 0.3 * sep]])
    d = np.asarray(O.separations())[None, :, None]
    u = (1.0 + d * np.linspace(0.3, 2.0, E)[None, None]) * np.array([1.0, 2.0])[:, None, None]
    part = np.cumsum(u, axis=1)
    part /= part[:, -1:]
    return O, A, (wcs, src, np.full((2, E), 1e11), u, part)


@pytest.mark.parametrize("H,W,sep", [(120, 40, 90.0), (40, 36, 70.0)])
@pytest.mark.parametrize("E", [1, 7])
def test_past_70_degrees(H, W, sep, E):
    O, A, args = _job(H, W, 1.0, "CAR", sep, E)
    ref = O.point_src_model_map_wcs(*args)
    m, info = A.point_src_model_map_wcs(*args, out_dtype="float64")
    assert (ref["map"] != 0.0).all()
    assert max_rel(m, ref["map"]) < 1e-10
    assert max_rel(info.inv_map_integral, ref["inv_integ"]) < 1e-10


@pytest.mark.parametrize("H,W,pix,proj,sep", [(36, 18, 10.0, "AIT", 3.0), (21, 20, 2e-5, "CAR", 0.0),
                                              (30, 33, 1e-5, "CAR", 2e-4)])
@pytest.mark.parametrize("E", [1, 7])
def test_ends_of_the_table_against_fp32(H, W, pix, proj, sep, E):
    O, A, args = _job(H, W, pix, proj, sep, E)
    m64, _ = A.point_src_model_map_wcs(*args, out_dtype="float64")
    m32, _ = A.point_src_model_map_wcs(*args)
    np.testing.assert_allclose(m32, m64, rtol=1e-5, equal_nan=True)
