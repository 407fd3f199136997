"""FP64 and FP32 maps of a job in which some positions are not finite: those sources' maps are
NaN, the others' are what they are without them (1e-12: the map integral's chunks differ).
The last source of the tables is one of them, so that a row past the table's end would be
one past the array's."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("H,W,E", [(33, 40, 5), (8, 8, 1)])
@pytest.mark.parametrize("dtype,tol", [("float64", 1e-12), ("float32", 1e-6)])
def test_positions_without_value(H, W, E, dtype, tol):
    from xtsrcmaps_b200 import api as A
    from xtsrcmaps_b200.wcs import Wcs

    A.init(0)
    wcs = Wcs(H, W, (H + 1) / 2.0, (W + 1) / 2.0, 120.0, -5.0, -0.1, 0.1)
    src = np.array([[np.nan, -5.0], [120.0, -5.0], [np.inf, np.nan], [120.2, -5.1], [120.0, np.nan]])
    ok = np.isfinite(src).all(axis=1)
    sep = np.concatenate([[0.0], 1e-4 * np.exp(np.arange(400) * np.log(70.0 / 1e-4) / 399.0)])
    u = np.repeat((1.0 + (sep[None, :, None] / np.linspace(0.5, 3.0, E)[None, None]) ** 2) ** -2.0, 5, axis=0)
    part = np.cumsum(u, axis=1)
    part /= part[:, -1:]
    ex = np.full((5, E), 1e11)
    m, _ = A.point_src_model_map_wcs(wcs, src, ex, u, part, out_dtype=dtype)
    r, _ = A.point_src_model_map_wcs(wcs, src[ok], ex[ok], u[ok], part[ok], out_dtype=dtype)
    assert np.isfinite(r).all() and np.isnan(m[~ok]).all()
    np.testing.assert_allclose(m[ok], r, rtol=tol)
