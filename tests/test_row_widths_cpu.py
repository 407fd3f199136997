"""The widths of the separation table's rows in squared chord, as the window pass bounds them: it
takes a row's neighbours as at least 1.05 and 0.934 times as wide (rows 2 to 397)."""
import os
import re

import numpy as np


def test_neighbouring_row_widths():
    step = np.log(70.0 / 1e-4) / 399.0
    sep = np.concatenate([[0.0], 1e-4 * np.exp(np.arange(400) * step)])
    width = np.diff((2.0 * np.sin(0.5 * np.deg2rad(sep))) ** 2)
    here = os.path.dirname(os.path.abspath(__file__))
    with open(os.path.join(here, "..", "xtsrcmaps_b200", "csrc", "xts_srcmap_win.cu")) as f:
        up, dn = re.search(r"mx < fmaf\((\S+)f, w0, e1\), dn = mn >= fmaf\(-(\S+)f, w0, e0\)", f.read()).groups()
    k = np.arange(2, 398)
    assert (width[k + 1] > float(up) * width[k]).all()
    assert (width[k - 1] > float(dn) * width[k]).all()
