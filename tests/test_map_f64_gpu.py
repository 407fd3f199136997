"""The FP64 source maps against the FP64 oracle where the pass changes form: pixels of two
rows, windows of several rows, wide pixels next to a source, sources beyond the table's
last row and on a pixel centre, and energy counts at the ends of the flat indexing."""
import numpy as np
import pytest

from helpers import max_rel


@pytest.mark.gpu
@pytest.mark.parametrize("H,W,E,pix,sep", [(40, 30, 29, 0.1, 0.0), (17, 129, 2, 0.02, 3.0), (33, 31, 1, 0.2, 1.0),
                                           (12, 11, 37, 1.0, 0.3), (3, 5, 6000, 0.1, 0.05), (9, 9, 300, 0.05, 75.0),
                                           (128, 2, 5, 0.1, 40.0)])
def test_maps_f64(H, W, E, pix, sep):
    from oracle import oracle as O
    from xtsrcmaps_b200 import api as A
    from xtsrcmaps_b200.wcs import Wcs

    A.init(0)
    wcs = Wcs(H, W, (H + 1) / 2.0, (W + 1) / 2.0, 120.0, -5.0, -pix, pix)
    rng = np.random.default_rng(E)
    src = np.array([[120.0, -5.0], [120.0 + sep, -5.0], [120.0, -5.0 + sep], [120.0 + 0.3 * pix, -5.0 + 0.2 * pix]])
    S = len(src)
    d = np.asarray(O.separations())[None, :, None]
    w = 10.0 ** rng.uniform(-1.0, 0.7, (S, 1, E))
    u = (1.0 + (d / w) ** 2) ** -rng.uniform(1.5, 3.0, (S, 1, E)) / w ** 2  # a falling profile per (source, energy)
    part = np.cumsum(np.abs(u), axis=1)
    part /= part[:, -1:]
    ex = 1e11 * rng.uniform(0.5, 2.0, (S, E))
    ref = O.point_src_model_map_wcs(wcs, src, ex, u, part)
    m, info = A.point_src_model_map_wcs(wcs, src, ex, u, part, out_dtype="float64")
    assert max_rel(m, ref["map"]) < 1e-10
    assert max_rel(info.inv_map_integral, ref["inv_integ"]) < 1e-10


_FIRST_CALL = """
import sys
sys.path[:0] = [%r, %r]
import numpy as np
from test_write_pass_gpu import _tables
A, wcs, src, ex, u, p = _tables(6, 3, 61, 83, 0.2)
m, _ = A.point_src_model_map_wcs(wcs, src, ex, u, p, out_dtype="float64")
assert np.isfinite(m).all()
"""


@pytest.mark.gpu
def test_first_map_of_a_process():
    """FP64 host maps before any other map of the process: the status word that the host reads
    after the call is this call's, not what the memory held."""
    import os
    import subprocess
    import sys

    here = os.path.dirname(os.path.abspath(__file__))
    subprocess.run([sys.executable, "-c", _FIRST_CALL % (os.path.dirname(here), here)], check=True, timeout=300)
