"""Dense FP32 maps of fewer than 32 columns, whose warps hold whole rows of pixel pairs between
two parts of rows, against the FP64 maps of the same tables (1e-5, as for every FP32 map):
one column to 31, odd and even heights, energy counts of every residue modulo 4."""
import numpy as np
import pytest

from helpers import max_rel
from test_write_pass_gpu import _tables


@pytest.mark.gpu
@pytest.mark.parametrize("H,W", [(1, 1), (70, 1), (65, 2), (33, 3), (2, 5), (41, 7), (130, 16), (1, 20), (67, 30), (64, 31)])
@pytest.mark.parametrize("E", [1, 2, 4, 37])
def test_narrow_maps(H, W, E):
    A, wcs, src, ex, u, p = _tables(3, E, H, W, 0.1)
    m32, _ = A.point_src_model_map_wcs(wcs, src, ex, u, p)
    m64, _ = A.point_src_model_map_wcs(wcs, src, ex, u, p, out_dtype="float64")
    assert np.isfinite(m32).all()
    assert max_rel(m32, m64) < 1e-5
