"""Device memory of one map call whose sources make one chunk: one set of the window path's
buffers (48 bytes of records per source and pixel, a pool of an eighth as many sparse records
of 192 bytes), not the two sets that several chunks take turns with."""
import os
import subprocess
import sys

import pytest

_CALL = """
import sys
sys.path[:0] = [%r, %r]
import numpy as np
import torch
from xtsrcmaps_b200 import api as A
from xtsrcmaps_b200.wcs import Wcs
S, n = 60, 400
A.init(0)
wcs = Wcs(n, n, (n + 1) / 2.0, (n + 1) / 2.0, 120.0, -5.0, -0.05, 0.05)
rng = np.random.default_rng(1)
d = lambda a: torch.as_tensor(np.ascontiguousarray(a), device="cuda")
args = (d(np.array([120.0, -5.0]) + rng.uniform(-8.0, 8.0, (S, 2))), d(np.full((S, 1), 1e11)),
        d(np.repeat(np.linspace(2.0, 1.0, 401)[None, :, None], S, axis=0)),
        d(np.repeat(np.linspace(0.0, 1.0, 401)[None, :, None], S, axis=0)))
out = torch.empty((S, n, n, 1), dtype=torch.float32, device="cuda")
A.point_src_model_map_wcs(wcs, *(a[:1] for a in args), out=out[:1], with_info=False)  # code and tables loaded
torch.cuda.synchronize()
before = torch.cuda.mem_get_info()[0]
A.point_src_model_map_wcs(wcs, *args, out=out, with_info=False)
torch.cuda.synchronize()
print((before - torch.cuda.mem_get_info()[0]) / (S * n * n))
"""


@pytest.mark.gpu
def test_one_chunk_takes_one_set():
    here = os.path.dirname(os.path.abspath(__file__))
    r = subprocess.run([sys.executable, "-c", _CALL % (os.path.dirname(here), here)], check=True, timeout=300,
                       capture_output=True, text=True)
    per_pixel = float(r.stdout.split()[-1])
    assert 60.0 < per_pixel < 90.0, per_pixel  # 72 bytes; the geometry and tables add less than one
