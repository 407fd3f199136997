"""The mean PSF does not depend on what its scratch held: a call whose psf*aeff table is NaN
throughout, then one whose rows lie elsewhere in the same scratch, against the FP64 oracle."""
import ctypes as C

import numpy as np
import pytest

from helpers import max_rel, oracle_pipeline

pytestmark = pytest.mark.gpu


def _regridded(grid, n_e):
    """The King grid with n_e energies (linear between its own)."""
    from xtsrcmaps_b200.irf import IrfGrid

    e0, p0 = np.asarray(grid.logEs), np.asarray(grid.params)
    en = np.linspace(e0[0], e0[-1], n_e)
    p = np.empty((p0.shape[0], n_e, 6))
    for i in range(p0.shape[0]):
        for k in range(6):
            p[i, :, k] = np.interp(en, e0, p0[i, :, k])
    return IrfGrid(np.asarray(grid.cosths), en, p, grid.min_cos_theta)


@pytest.mark.parametrize("S", [3, 60, 700])  # the three tile shapes of the kernel
def test_scratch_holding_nan(S):
    import torch

    from oracle import oracle as O
    from xtsrcmaps_b200 import _lib as L
    from xtsrcmaps_b200 import api as A
    from xtsrcmaps_b200.synth import make_job

    A.init(0)
    dev = torch.device("cuda", 0)
    job = make_job("c1", seed=31, n_sources=S)
    job.logEs = job.logEs[::2].copy()
    job.energies = 10.0 ** job.logEs
    o = oracle_pipeline(job, with_map=False)
    E, Cn = len(job.logEs), len(o["costh"])
    up, pp = (torch.empty((S, 401, E), dtype=torch.float64, device=dev) for _ in range(2))
    vp = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    names = ("costh", "logEs", "af", "ab", "ecb", "wecb", "ltf", "exposure")
    host = dict(o, logEs=job.logEs)

    def call(nb, bad):
        c = A._Call(True, torch.empty(0, device=dev))
        gf, gb = c.grid(o["nf"], 6), c.grid(nb, 6)
        d = {k: torch.as_tensor(np.ascontiguousarray(host[k]), dtype=torch.float64, device=dev) for k in names}
        if bad:
            d["af"].fill_(float("nan"))
        L.check(L.lib().xts_compute_psf_data_noalloc(
            C.byref(gf), C.byref(gb), vp(d["costh"]), Cn, vp(d["logEs"]), E, vp(d["af"]), vp(d["ab"]), vp(d["ecb"]),
            vp(d["wecb"]), S, vp(d["ltf"]), vp(d["exposure"]), vp(up), vp(pp), c.stream))
        torch.cuda.synchronize()

    call(o["nb"], True)
    assert torch.isnan(up).all()
    # two energies more in the back grid: psf*aeff starts 401 * 2 * cos-theta nodes further on
    nb = _regridded(o["nb"], o["nb"].params.shape[1] + 2)
    call(nb, False)
    u, p = O.compute_psf_data(o["nf"], nb, o["costh"], job.logEs, o["af"], o["ab"], o["ecb"], o["wecb"], o["ltf"],
                              o["exposure"])
    assert max_rel(up.cpu().numpy(), u) < 1e-11
    assert max_rel(pp.cpu().numpy(), p, floor=1e-300) < 1e-11
