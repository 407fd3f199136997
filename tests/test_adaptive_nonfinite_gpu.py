"""Adaptive maps from a mean-PSF table with one infinite row, a source beside the map: values are
infinite where a region's window holds the row, none is NaN (each region reads the rows of
its own window only), and the others are what they are without it (1e-6, FP32 rounding)."""
import numpy as np
import pytest

from test_nonfinite_rows_gpu import _job

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("row", [317, 318])
def test_adaptive(row):
    A, wcs, src, ex, u, clean, part, sep = _job(6, np.inf, row)
    m, _ = A.point_src_model_map_wcs_adaptive(wcs, src, ex, u, part, rtol=1e-3, max_depth=0)
    c, _ = A.point_src_model_map_wcs_adaptive(wcs, src, ex, clean, part, rtol=1e-3, max_depth=0)
    assert np.isinf(m).any() and not np.isnan(m).any()
    fin = np.isfinite(m)
    np.testing.assert_allclose(m[fin], c[fin], rtol=1e-6)
