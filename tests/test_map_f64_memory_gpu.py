"""FP64 maps on a GPU whose memory is nearly full: the pass's records take fewer sources at a time
where those of the whole job do not fit (1.9 GB here, beside 1.2 GB free); the maps are what
they are with all memory free (1e-12: the map integral's chunks differ)."""
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
S, n = 40, 700
A.init(0)
wcs = Wcs(n, n, (n + 1) / 2.0, (n + 1) / 2.0, 120.0, -5.0, -0.05, 0.05)
rng = np.random.default_rng(1)
d = lambda a: torch.as_tensor(np.ascontiguousarray(a), device="cuda")
sep = np.concatenate([[0.0], 1e-4 * np.exp(np.arange(400) * np.log(70.0 / 1e-4) / 399.0)])
u = np.repeat((1.0 + (sep[None, :, None] / 0.8) ** 2) ** -2.0, S, axis=0)
part = np.cumsum(u, axis=1)
args = (d(np.array([120.0, -5.0]) + rng.uniform(-8.0, 8.0, (S, 2))), d(np.full((S, 1), 1e11)), d(u),
        d(part / part[:, -1:]))
out, ref = (torch.empty((S, n, n, 1), dtype=torch.float64, device="cuda") for _ in range(2))
call = lambda k, o: A.point_src_model_map_wcs(wcs, *(a[:k] for a in args), out_dtype="float64", out=o[:k], with_info=False)
call(1, out)  # code and tables loaded
torch.cuda.synchronize()
fill = torch.empty(torch.cuda.mem_get_info()[0] - 1200 * 10 ** 6, dtype=torch.uint8, device="cuda")
call(S, out)
torch.cuda.synchronize()
del fill
torch.cuda.empty_cache()
call(S, ref)
torch.cuda.synchronize()
assert float(((out - ref).abs() / ref.abs()).max()) < 1e-12
"""


@pytest.mark.gpu
def test_little_memory_left():
    here = os.path.dirname(os.path.abspath(__file__))
    subprocess.run([sys.executable, "-c", _CALL % (os.path.dirname(here), here)], check=True, timeout=300)
