"""The work that users of this package have it do, as timed cases.

Every case goes through the package's public entry points on synthetic, seeded
inputs of the shapes, distributions and value ranges of the bundled
configurations (xtsrcmaps_b200.synth):

* ``maps``       exposure -> mean PSF -> source maps in the fused call, device arrays;
* ``maps_host``  the same call on host arrays, as a C++ or numpy host makes it;
* ``tables``     exposure and mean-PSF tables of a source catalogue, without maps;
* ``sky``        the exposure of every HEALPix pixel;
* ``cutouts``    maps in a window per source;
* ``adaptive``   maps by adaptive cubature;
* ``surrogate``  maps by the learned surrogate with its fallback;
* ``gradient``   one forward and backward pass of the surrogate's training.

``exact`` restates what each of them computes in plain torch, in 64 bits.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from xtsrcmaps_b200 import api
from xtsrcmaps_b200.irf import IrfGrid
from xtsrcmaps_b200.surrogate import Surrogate, samples
from xtsrcmaps_b200.synth import CENTER, make_job, native_to_celestial
from xtsrcmaps_b200.wcs import Wcs

BINS = 40  # cos-theta bins of a livetime cube
ROWS = 401  # rows of the separation table
HIDDEN = 128  # units of a hidden layer of the surrogate
TOLERANCE = 2e-4  # of the surrogate's values; a third to a half of them are the network's after its short training


# --------------------------------------------------------------------------- the cases
def _case(kind, S=0, H=0, W=0, E=0, pix=0.1, emin=100.0, emax=1e6, nside=64, proj="CAR", field=20.0, **more):
    return dict(kind=kind, S=S, H=H, W=W, E=E, pix=pix, emin=emin, emax=emax, nside=nside, proj=proj, field=field,
                **more)


def listed():
    return [
        # one source in a small map, from a host program's own arrays: the shortest whole call
        dict(_case("maps_host", 1, 100, 100, 20, 0.2, 100.0, 1e5, 32, field=0.0), name="one_source_host"),
        # the few sources near a target in a ragged all-sky-projection map: launches and latency
        dict(_case("maps", 7, 61, 99, 21, 0.2, 100.0, 1e5, 32, proj="AIT", field=10.0, f64=False), name="few_ait"),
        # an ordinary region of interest
        dict(_case("maps", 50, 200, 200, 37, f64=False), name="roi"),
        # a region in doubles (the reference's output type), odd sizes
        dict(_case("maps", 50, 151, 203, 29, f64=True), name="roi_doubles"),
        # a crowded region at full resolution: the largest dense maps
        dict(_case("maps", 500, 400, 400, 37, 0.05, f64=False), name="crowded"),
        # one batch of a large field's sources: the largest map, the finest pixels, the most energies
        dict(_case("maps", 40, 800, 800, 50, 0.025, 30.0, 1e6, 128, field=40.0, f64=False), name="wide_field"),
        # the crowded region with a window of 2-15 degrees around each source
        dict(_case("cutouts", 500, 400, 400, 37, 0.05), name="crowded_cutouts"),
        # the region of interest by adaptive cubature
        dict(_case("adaptive", 50, 200, 200, 37, rtol=1e-4, depth=6), name="roi_adaptive"),
        # the tables of a whole catalogue
        dict(_case("tables", 2000, E=50, emin=30.0, nside=128, field=40.0), name="catalogue_tables"),
        # exposure of the whole sky
        dict(_case("sky", E=50, emin=30.0, nside=256), name="sky_exposure"),
        # maps by the learned surrogate
        dict(_case("surrogate", 60, 400, 400, 37, 0.05), name="surrogate_maps"),
        # a training batch of the surrogate, forward and backward
        dict(_case("gradient", 50, E=37, rows=128 * 296), name="surrogate_gradient"),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["maps"] * 5 + ["maps_host", "cutouts", "adaptive", "tables", "sky", "surrogate", "gradient"])
    E = rng.randint(15, 50)
    emin, emax = rng.choice([30.0, 100.0]), rng.choice([1e5, 1e6])
    if kind == "sky":
        return _case("sky", E=E, emin=emin, emax=emax, nside=rng.choice([32, 64, 128, 256]))
    if kind == "gradient":
        return _case("gradient", rng.randint(10, 100), E=E, emin=emin, emax=emax, rows=128 * int(_log(rng, 16, 592)))
    if kind == "tables":
        return _case("tables", int(_log(rng, 1, 2000)), E=E, emin=emin, emax=emax, nside=rng.choice([32, 64, 128]),
                     field=rng.uniform(5, 40))
    # map sizes up to the value count that the kind's listed case has
    most = {"maps": 2e9, "maps_host": 5e7, "cutouts": 2e9, "adaptive": 7e7, "surrogate": 3e8}[kind]
    H = int(_log(rng, 50, 800))
    W = H if rng.random() < 0.4 else int(_log(rng, 50, 800))
    f64 = kind == "maps" and rng.random() < 0.25
    if f64:
        most = 7e7
    S = max(1, min(int(_log(rng, 1, 500)), int(most / (H * W * E))))
    pix = 0.025 * 2 ** rng.randint(0, 3)
    c = _case(kind, S, H, W, E, pix, emin, emax, rng.choice([32, 64, 128]), rng.choice(["CAR", "CAR", "AIT"]),
              round(min(H, W) * pix * rng.uniform(0.6, 1.1), 3))
    if kind == "maps":
        c["f64"] = f64
    if kind == "adaptive":
        c.update(rtol=rng.choice([1e-3, 1e-4]), depth=rng.randint(3, 6))
    return c


# --------------------------------------------------------------------------- inputs
def _wcs(c):
    return Wcs(c["H"], c["W"], (c["H"] + 1) / 2.0, (c["W"] + 1) / 2.0, CENTER[0], CENTER[1], -c["pix"], c["pix"],
               proj=c["proj"])


def _sources(c, rng):
    """[S, 2] positions: uniform over the field; where the field is as wide as the map, every
    tenth source within a degree of the map's edge, inside or just outside."""
    S, half = c["S"], 0.5 * c["field"]
    x, y = rng.uniform(-half, half, S), rng.uniform(-half, half, S)
    if c["H"] and half > 0.45 * c["H"] * c["pix"]:
        k = S // 10
        x[:k] = rng.choice([-1.0, 1.0], k) * (0.5 * c["H"] * c["pix"] + rng.uniform(-1.0, 1.0, k))
    pole = Wcs(2, 2, 1.5, 1.5, CENTER[0], CENTER[1], -1.0, 1.0)
    return np.ascontiguousarray(np.stack(native_to_celestial(pole, x, y), axis=1))


def _f64(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


def _grid_on_gpu(g):
    return IrfGrid(_f64(g.cosths), _f64(g.logEs), _f64(g.params), g.min_cos_theta)


def _cubes(nside, seed):
    """Livetime cubes [12 nside^2, BINS]: a constant times lognormal(0, 0.2), the weighted cube 0.9 of it."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    base = 2.0e5 * torch.exp(0.2 * torch.randn(12 * nside * nside, BINS, device="cuda", generator=gen))
    return api.ExpCube(base, nside, BINS), api.ExpCube((0.9 * base).contiguous(), nside, BINS)


def _tables(s):
    ex = api.compute_exposure(s["cube"], s["wcube"], s["logEs"], s["src"], s["af"], s["ab"], s["ltf"])
    return ex, api.compute_psf_data(s["nf"], s["nb"], ex, s["logEs"], s["ltf"])


def prepare(case, seed):
    c = dict(case)
    irf = make_job("c0", seed=seed % 100003 + 1)  # the instrument's tables
    logEs = np.log10(np.logspace(math.log10(c["emin"]), math.log10(c["emax"]), c["E"]))
    ltf = api.livetime_efficiency_factors(logEs, irf.effic_front)
    nf = api.normalize_rpsf(irf.rpsf_front, irf.scale_front)
    nb = api.normalize_rpsf(irf.rpsf_back, irf.scale_back)
    rng = np.random.default_rng(seed)
    s = dict(kind=c["kind"], f64=c.get("f64", False), rtol=c.get("rtol"), depth=c.get("depth"))
    s["cube"], s["wcube"] = _cubes(c["nside"], seed)
    # a survey's windows stay while its exposure grows: positions and radii of the case, not of the seed
    layout = np.random.default_rng(c["S"] * 1000 + c["H"]) if c["kind"] == "cutouts" else rng
    src = _sources(c, layout)
    if c["H"]:
        s["wcs"] = _wcs(c)
    if c["kind"] == "maps_host":
        for k in ("cube", "wcube"):
            s[k].cosbins = s[k].cosbins.cpu().numpy()
        s.update(logEs=logEs, src=src, ltf=ltf, nf=nf, nb=nb, af=irf.aeff_front, ab=irf.aeff_back)
        return s
    s.update(logEs=_f64(logEs), src=_f64(src), ltf=_f64(ltf), nf=_grid_on_gpu(nf), nb=_grid_on_gpu(nb),
             af=_grid_on_gpu(irf.aeff_front), ab=_grid_on_gpu(irf.aeff_back))
    if c["kind"] == "cutouts":
        s["cut_host"], total = api.cutout_windows(s["wcs"], src, layout.uniform(2.0, 15.0, c["S"]))
        s["cut"] = torch.as_tensor(np.frombuffer(s["cut_host"].tobytes(), dtype=np.uint8).copy(), device="cuda")
        s["out"] = torch.empty((total, c["E"]), dtype=torch.float32, device="cuda")
    elif c["kind"] in ("surrogate", "gradient"):
        t = dict(s)
        if c["kind"] == "surrogate":  # the network was trained on another field's tables
            t["src"] = _f64(_sources(dict(c, S=50, H=0, field=20.0), rng))
        u = _tables(t)[1].uPsf
        s["net"] = net = Surrogate(device="cuda", seed=seed)
        if c["kind"] == "surrogate":
            X, Y = samples(u, logEs, 2_000_000, seed=seed + 1)
            net.train(X, Y, epochs=24, seed=seed)
            net.calibrate(*samples(u, logEs, 1_000_000, seed=seed + 2), tol=TOLERANCE)
        else:
            s["X"], s["Y"] = samples(u, logEs, c["rows"], seed=seed + 1)
            net.fit_standardisation(s["X"], s["Y"])
    return s


# --------------------------------------------------------------------------- one pass
def run(s):
    kind = s["kind"]
    if kind in ("maps", "maps_host"):
        return api.point_source_maps(s["wcs"], s["src"], s["cube"], s["wcube"], s["logEs"], s["af"], s["ab"], s["nf"],
                                     s["nb"], s["ltf"], out_dtype="float64" if s["f64"] else "float32",
                                     with_info=False)[0]
    if kind == "sky":
        return api.exposure_map(s["cube"], s["wcube"], s["logEs"], s["af"], s["ab"], s["ltf"])
    if kind == "surrogate":
        return api.point_source_maps_surrogate(s["wcs"], s["src"], s["cube"], s["wcube"], s["logEs"], s["af"],
                                               s["ab"], s["nf"], s["nb"], s["ltf"], s["net"],
                                               check_tol=TOLERANCE, stats=False)[0]
    if kind == "gradient":
        return s["net"].gradient(s["X"], s["Y"])
    ex, ps = _tables(s)
    if kind == "tables":
        return {"exposure": ex.exposure, "uPsf": ps.uPsf, "partial": ps.partial_psf_integral}
    if kind == "cutouts":
        return api.point_src_model_map_cutouts(s["wcs"], s["src"], s["cut"], ex.exposure, ps.uPsf,
                                               ps.partial_psf_integral, out=s["out"], with_info=False)[0]
    return api.point_src_model_map_wcs_adaptive(s["wcs"], s["src"], ex.exposure, ps.uPsf, ps.partial_psf_integral,
                                                rtol=s["rtol"], max_depth=s["depth"], with_info=False)[0]


def work(case):
    """Bytes: the results once, the sources' livetime rows (for ``sky`` the whole cubes), the
    effective-area and King tables.  Flops: the mean PSF's contraction; the chord, table weight
    and accumulation of each rule point; two table rows per value."""
    c = case
    S, E, C = c["S"], c["E"], BINS
    irf = 8.0 * 2 * (34 * 76 + 10 * 25 * 6)
    if c["kind"] == "gradient":
        par = 5 * HIDDEN + 2 * HIDDEN * HIDDEN + HIDDEN
        return {"bytes": c["rows"] * 24.0 + 8.0 * par, "flops": 6.0 * c["rows"] * par}
    if c["kind"] == "sky":
        n = 12 * c["nside"] ** 2
        return {"bytes": n * (2 * C * 4 + 8.0 * E) + irf, "flops": n * E * C * 4.0}
    b, f = irf + S * (2 * C * 4 + 16), S * ROWS * E * C * 4.0
    if c["kind"] == "tables":
        return {"bytes": b + 8.0 * S * E * (2 * ROWS + 1), "flops": f}
    pixels = float(S * c["H"] * c["W"])
    if c["kind"] == "cutouts":  # windows of 2-15 degrees, cut at the map's edge: about half of the map
        pixels *= min(1.0, 0.45 * (20.0 / (c["H"] * c["pix"])) * (20.0 / (c["W"] * c["pix"])))
    points = {"adaptive": 17}.get(c["kind"], 12)
    return {"bytes": b + pixels * E * (8 if c.get("f64") else 4), "flops": f + pixels * (points * 20.0 + E * 4.0)}


# --------------------------------------------------------------------------- the same in 64 bits
_D2R, _TWOPI = math.pi / 180.0, 2.0 * math.pi
_STEP = math.log(70.0 / 1e-4) / 399.0  # of the separation table, in ln
_RULE = [  # Sommariva and Festa's 12-point rule of degree 7 on the square: u, v, weight; then mirrored
    (3.9383136101878902e-01, -3.6699793434042738e-01, 5.2092862230230441e-01),
    (8.0196847620659251e-01, 8.0992592975809186e-01, 2.3740240561379911e-01),
    (-1.8327327664247231e-02, 9.2596092593108370e-01, 2.4166897208389651e-01),
    (3.6699793434042738e-01, 3.9383136101878902e-01, 5.2092862230230441e-01),
    (-8.0992592975809186e-01, 8.0196847620659251e-01, 2.3740240561379911e-01),
    (-9.2596092593108370e-01, -1.8327327664247231e-02, 2.4166897208389651e-01),
]
_RULE += [(-u, -v, w) for u, v, w in _RULE]


def _separations():
    return torch.cat([torch.zeros(1, dtype=torch.float64), 1e-4 * torch.exp(torch.arange(400.0).double() * _STEP)]).cuda()


def _direction(ra, dec):
    ra, dec = ra * _D2R, dec * _D2R
    return torch.stack([torch.cos(ra) * torch.cos(dec), torch.sin(ra) * torch.cos(dec), torch.sin(dec)], dim=-1)


def _pole(w):
    a0 = w.crval1 - 360.0 if w.crval1 > 180.0 else w.crval1
    return (a0 - 180.0, 90.0 - w.crval2, 0.0) if w.crval2 >= 0 else (a0, 90.0 + w.crval2, 180.0)


def _pix2dir(w, p1, p2):
    """Directions [len(p1), len(p2), 3] of the pixel grid p1 x p2 (Calabretta and Greisen 2002)."""
    x, y = torch.meshgrid(w.cdelt1 * (_f64(p1) - w.crpix1), w.cdelt2 * (_f64(p2) - w.crpix2), indexing="ij")
    if w.proj == "CAR":
        phi, theta = x * _D2R, y * _D2R
    else:
        X, Y = x * _D2R, y * _D2R
        z2 = 1.0 - X * X / 16.0 - Y * Y / 4.0
        z = z2.clamp(min=0.0).sqrt()
        phi, theta = 2.0 * torch.atan2(0.5 * X * z, 2.0 * z2 - 1.0), torch.asin((Y * z).clamp(-1, 1))
    ap, dp, pp = _pole(w)
    sd, cd, dphi = math.sin(dp * _D2R), math.cos(dp * _D2R), phi - pp * _D2R
    st, ct = torch.sin(theta), torch.cos(theta)
    ra = ap + torch.atan2(-ct * torch.sin(dphi), st * cd - ct * sd * torch.cos(dphi)) / _D2R
    dec = torch.asin((st * sd + ct * cd * torch.cos(dphi)).clamp(-1, 1)) / _D2R
    return _direction(ra, dec)


def _sph2pix(w, ra, dec):
    ap, dp, pp = _pole(w)
    sd, cd, da, d = math.sin(dp * _D2R), math.cos(dp * _D2R), (ra - ap) * _D2R, dec * _D2R
    phi = pp + math.atan2(-math.cos(d) * math.sin(da), math.sin(d) * cd - math.cos(d) * sd * math.cos(da)) / _D2R
    theta = math.asin(max(-1.0, min(1.0, math.sin(d) * sd + math.cos(d) * cd * math.cos(da)))) / _D2R
    while phi > 180.0:
        phi -= 360.0
    while phi <= -180.0:
        phi += 360.0
    if w.proj == "CAR":
        x, y = phi, theta
    else:
        ct, h = math.cos(theta * _D2R), 0.5 * phi * _D2R
        g = math.sqrt(2.0 / (1.0 + ct * math.cos(h))) / _D2R
        x, y = 2.0 * g * ct * math.sin(h), g * math.sin(theta * _D2R)
    return w.crpix1 + x / w.cdelt1, w.crpix2 + y / w.cdelt2


def _nested(src, nside):
    """HEALPix NESTED pixel of each source (Gorski et al. 2005)."""
    order, out = nside.bit_length() - 1, []
    for ra, dec in src:
        z, tt = math.cos(0.5 * math.pi - dec * _D2R), (ra % 360.0) / 90.0
        if abs(z) <= 2.0 / 3.0:
            t1, t2 = nside * (0.5 + tt), nside * z * 0.75
            jp, jm = int(t1 - t2), int(t1 + t2)
            fp, fm = jp >> order, jm >> order
            face = fp | 4 if fp == fm else fp if fp < fm else fm + 8
            ix, iy = jm & (nside - 1), nside - (jp & (nside - 1)) - 1
        else:
            q = min(3, int(tt))
            tmp = nside * math.sqrt(3.0 * (1.0 - abs(z)))
            jp, jm = min(nside - 1, int((tt - q) * tmp)), min(nside - 1, int((1.0 - tt + q) * tmp))
            face, ix, iy = (q, nside - jm - 1, nside - jp - 1) if z >= 0 else (q + 8, jp, jm)
        out.append((face << 2 * order) + sum(((ix >> b & 1) << 2 * b) + ((iy >> b & 1) << 2 * b + 1) for b in range(order)))
    return torch.tensor(out, device="cuda")


def _between(grid, v):
    """(index of the upper neighbour, weight of it)."""
    i = torch.searchsorted(grid, v, right=True).clamp(1, len(grid) - 1)
    return i, (v - grid[i - 1]) / (grid[i] - grid[i - 1])


def _bilinear(table, ci, cw, ei, ew):
    """table [..., Mc, Me] at (c, e) -> [..., C, E]."""
    cw, ci = cw[:, None], ci[:, None]
    return ((1 - cw) * (1 - ew) * table[..., ci - 1, ei - 1] + (1 - cw) * ew * table[..., ci - 1, ei]
            + cw * (1 - ew) * table[..., ci, ei - 1] + cw * ew * table[..., ci, ei])


def _on_gpu(s):
    g = dict(s)
    for k in ("logEs", "src", "ltf"):
        g[k] = _f64(s[k].cpu().numpy() if torch.is_tensor(s[k]) else s[k])
    for k in ("af", "ab", "nf", "nb"):
        if not torch.is_tensor(s[k].params):
            g[k] = _grid_on_gpu(s[k])
    return g


def _exact_aeff(g, logEs):
    costh = 1.0 - ((torch.arange(BINS, dtype=torch.float64, device="cuda") + 0.5) / BINS) ** 2
    ci, cw = _between(g.cosths, costh)
    a = 1e4 * _bilinear(g.params[..., 0], ci, cw, *_between(g.logEs, logEs))
    return torch.where((costh >= g.min_cos_theta)[:, None], a, torch.zeros_like(a))


def _exact_tables(g):
    """Exposure [S, E], mean PSF and its partial integrals [S, ROWS, E]."""
    logEs, ltf = g["logEs"], g["ltf"]
    pix = _nested(g["src"].cpu().numpy(), g["cube"].nside)
    x, w = (torch.as_tensor(g[k].cosbins, device="cuda")[pix].double() for k in ("cube", "wcube"))
    aeff = [_exact_aeff(g[k], logEs) for k in ("af", "ab")]
    expo = (x @ (aeff[0] + aeff[1])) * ltf[0] + (w @ (aeff[0] + aeff[1])) * ltf[1]
    seps = _separations() * _D2R
    costh = 1.0 - ((torch.arange(BINS, dtype=torch.float64, device="cuda") + 0.5) / BINS) ** 2
    pa = 0.0
    for side, a in zip(("nf", "nb"), aeff):
        p = g[side].params
        king = 0.0
        for n, sig, gam in ((p[..., 0], p[..., 2], p[..., 4]), (p[..., 0] * p[..., 1], p[..., 3], p[..., 5])):
            u = 0.5 * (seps[:, None, None] / sig) ** 2
            king = king + n * (1.0 - 1.0 / gam) * (1.0 + u / gam) ** -gam
        ci, cw = _between(g[side].cosths, costh)
        pa = pa + _bilinear(king, ci, cw, *_between(g[side].logEs, logEs)) * a  # [ROWS, C, E]
    u = (torch.einsum("sc,dce->sde", x, pa) * ltf[0] + torch.einsum("sc,dce->sde", w, pa) * ltf[1]) / expo[:, None]
    t1, t2 = seps[:-1, None], seps[1:, None]
    y = _TWOPI * u * torch.sin(seps)[:, None]
    m = (y[:, 1:] - y[:, :-1]) / (t2 - t1)
    piece = 0.5 * m * (t2 * t2 - t1 * t1) + (y[:, :-1] - t1 * m) * (t2 - t1)
    part = torch.cat([torch.zeros_like(u[:, :1]), torch.cumsum(piece, dim=1)], dim=1)
    total = part[:, -1:].clone()
    return expo, u / total, part / total


def _row_weight(d2):
    """Upper table row and its weight for squared chords d2."""
    s = 2.0 / _D2R * torch.asin(0.5 * d2.sqrt())
    j = torch.where(s < 1e-4, torch.ones_like(s), 1.0 + (torch.log(s) + math.log(1e4)) / _STEP)
    idx = (1 + j.floor().long()).clamp(max=400)
    return idx, (s * 1e4 * torch.exp(_STEP * (2.0 - idx.double())) - 1.0) / math.expm1(_STEP)


def _blend(corners, u, v):
    a, b, c, d = corners
    return 0.25 * ((1 - u) * (1 - v) * a + (1 + u) * (1 - v) * b + (1 + u) * (1 + v) * c + (1 - u) * (1 + v) * d)


def _rule_means(corners, src, lut):
    out = torch.zeros(corners[0].shape[0], lut.shape[1], dtype=torch.float64, device="cuda")
    for u, v, wt in _RULE:
        idx, t = _row_weight((_blend(corners, u, v) - src).square().sum(-1))
        out += (0.25 * wt * (1.0 - t))[:, None] * lut[idx - 1] + (0.25 * wt * t)[:, None] * lut[idx]
    return out


def _adaptive_means(corners, src, lut, rtol, depth):
    """Genz and Malik's embedded rules of degrees 7 and 5 for two dimensions, regions halved along
    the larger fourth difference until the two agree to rtol at every energy."""
    l2, l4, l5 = math.sqrt(9 / 70), math.sqrt(9 / 10), math.sqrt(9 / 19)
    at = [(0, 0), (-l2, 0), (0, -l2), (l2, 0), (0, l2), (-l4, 0), (0, -l4), (l4, 0), (0, l4), (-l4, -l4), (l4, -l4),
          (-l4, l4), (l4, l4), (-l5, -l5), (-l5, l5), (l5, -l5), (l5, l5)]
    n = [1, 4, 4, 4, 4]
    w7 = [(12824 - 9120 * 2 + 400 * 4) / 19683, 980 / 6561, (1820 - 800) / 19683, 200 / 19683, 6859 / 19683 / 4]
    w5 = [(729 - 950 * 2 + 50 * 4) / 729, 245 / 486, (265 - 200) / 1458, 25 / 729, 0.0]
    w7, w5 = (_f64([x for x, k in zip(w, n) for _ in range(k)]) for w in (w7, w5))
    P, E = corners[0].shape[0], lut.shape[1]
    out = torch.zeros(P, E, dtype=torch.float64, device="cuda")
    pix = torch.arange(P, device="cuda")
    reg = torch.tensor([0.0, 0.0, 1.0, 1.0], dtype=torch.float64, device="cuda").repeat(P, 1)  # centres and half-widths
    for level in range(depth + 1):
        if not len(pix):
            break
        cs = [c[pix] for c in corners]
        f = torch.empty(len(pix), 17, E, dtype=torch.float64, device="cuda")
        for k, (o0, o1) in enumerate(at):
            v, u = reg[:, 0] + o0 * reg[:, 2], reg[:, 1] + o1 * reg[:, 3]
            idx, t = _row_weight((_blend(cs, u[:, None], v[:, None]) - src).square().sum(-1))
            f[:, k] = (1 - t)[:, None] * lut[idx - 1] + t[:, None] * lut[idx]
        v7, v5 = torch.einsum("rke,k->re", f, w7), torch.einsum("rke,k->re", f, w5)
        done = ((v5 - v7).abs() <= rtol * v7.abs()).all(dim=1) | (level == depth)
        out.index_add_(0, pix[done], (reg[done, 2] * reg[done, 3])[:, None] * v7[done])
        f, pix, reg = f[~done], pix[~done], reg[~done]
        d0, d1 = (((f[:, a] + f[:, a + 2] - 2 * f[:, 0]) - (f[:, b] + f[:, b + 2] - 2 * f[:, 0]) / 7).abs().sum(1)
                  for a, b in ((1, 5), (2, 6)))
        axis = (d1 > d0).long()
        halves = []
        for side in (-0.5, 0.5):
            r, i = reg.clone(), torch.arange(len(pix), device="cuda")
            r[i, 2 + axis] = 0.5 * reg[i, 2 + axis]
            r[i, axis] = reg[i, axis] + side * reg[i, 2 + axis]
            halves.append(r)
        pix, reg = pix.repeat(2), torch.cat(halves)
    return out


def _angle(a, b):
    return 2.0 * torch.asin(0.5 * (a - b).square().sum(-1).sqrt())


def _geometry(w):
    """Corners, centres and solid angles of the map's pixels, and its border points."""
    H, W = w.naxis1, w.naxis2
    edge = _pix2dir(w, np.arange(H + 1) + 0.5, np.arange(W + 1) + 0.5)
    cen = _pix2dir(w, np.arange(H + 1) + 1.0, np.arange(W + 1) + 1.0)
    a, b, c, d = cen[:-1, :-1], cen[:-1, 1:], cen[1:, 1:], cen[1:, :-1]

    def half(p, q, r):
        u, v = p - q, p - r
        u, v = u / u.norm(dim=-1, keepdim=True), v / v.norm(dim=-1, keepdim=True)
        return _angle(p, q) * _angle(p, r) * torch.linalg.cross(u, v).norm(dim=-1)

    omega = 0.5 * (half(a, b, d) + half(c, b, d))
    corners = [e.reshape(-1, 3) for e in (edge[:-1, :-1], edge[:-1, 1:], edge[1:, 1:], edge[1:, :-1])]
    border = torch.cat([edge[:, 0], edge[:, -1], edge[0], edge[-1]])
    return corners, a.reshape(-1, 3), omega.reshape(-1), border


def _exact_map(w, geo, sph, expo, u, part, means):
    """One source's map [H W, E] from its pixel means."""
    corners, cen, omega, border = geo
    sd = _direction(_f64(sph[0]), _f64(sph[1]))
    m = means(corners, sd, u).mul_(omega[:, None])
    p1, p2 = _sph2pix(w, sph[0] - 360.0 if sph[0] > 180.0 else sph[0], sph[1])
    factor = expo
    if 3.5 < p1 < w.naxis1 - 3.5 and 3.5 < p2 < w.naxis2 - 3.5:
        radius = float(_angle(border, sd).min()) / _D2R
        total = (_angle(cen, sd) <= radius * _D2R).double() @ m
        d = min(ROWS - 2, 1 if radius < 1.0 else int(1.0 + math.log(1e4 * radius) / _STEP))
        t = (_separations() * _D2R)[d:d + 2]
        y = _TWOPI * u[d:d + 2] * torch.sin(t)[:, None]
        slope = (y[1] - y[0]) / (t[1] - t[0])
        inside = 0.5 * slope * (t[1] ** 2 - t[0] ** 2) + (y[0] - t[0] * slope) * (t[1] - t[0]) + part[d]
        inv = torch.where(total != 0, 1.0 / total, total)
        factor = expo * inside.clamp(max=1.0) * inv
    return m.mul_(factor)


def _exact_gradient(s):
    """Gradient and loss of the network (bfloat16 hidden weights, tanh GELU), by autograd."""
    net, h = s["net"], HIDDEN
    p = net.params.double().requires_grad_(True)
    a, sizes = [], [5 * h, h, h * h, h, h * h, h, h, 1]
    for n, part in zip(sizes, torch.split(p, sizes)):
        r = part + (part.detach().float().bfloat16().double() - part.detach()) if n > h or len(a) == 6 else part
        a.append(r)
    f = torch.nn.functional.gelu
    z = (s["X"].double() - _f64(net.in_mu)) / _f64(net.in_sd)
    z = f(z @ a[0].view(h, 5).T + a[1], approximate="tanh")
    z = f(z @ a[2].view(h, h).T + a[3], approximate="tanh")
    z = f(z @ a[4].view(h, h).T + a[5], approximate="tanh")
    loss = (z @ a[6] + a[7] - (s["Y"].double() - net.out_mu) / net.out_sd).square().mean()
    return torch.autograd.grad(loss, p)[0], float(loss.detach())


def exact(case, seed):
    s = prepare(case, seed)
    kind = s["kind"]
    if kind == "gradient":
        return _exact_gradient(s)
    g = _on_gpu(s)
    if kind == "sky":
        a = _exact_aeff(g["af"], g["logEs"]) + _exact_aeff(g["ab"], g["logEs"])
        return sum((c.cosbins.double() @ a) * f for c, f in zip((g["cube"], g["wcube"]), g["ltf"]))
    expo, u, part = _exact_tables(g)
    if kind == "tables":
        return {"exposure": expo, "uPsf": u, "partial": part}
    means = _rule_means
    if kind == "adaptive":
        def means(corners, sd, lut):
            return _adaptive_means(corners, sd, lut, s["rtol"], s["depth"])
    w, src = g["wcs"], g["src"].cpu().numpy()
    E = u.shape[2]
    if kind == "cutouts":  # each window is a map of its own
        out = torch.empty(s["out"].shape, dtype=torch.float64, device="cuda")
        for i, c in enumerate(s["cut_host"]):
            n = int(c["nh"]) * int(c["nw"])
            if n:
                sub = Wcs(int(c["nh"]), int(c["nw"]), w.crpix1 - int(c["h0"]), w.crpix2 - int(c["w0"]), w.crval1,
                          w.crval2, w.cdelt1, w.cdelt2, proj=w.proj)
                out[int(c["offset"]):int(c["offset"]) + n] = _exact_map(sub, _geometry(sub), src[i], expo[i], u[i],
                                                                        part[i], means)
        return out
    geo = _geometry(w)
    out = torch.empty(len(src), w.naxis1 * w.naxis2, E, dtype=torch.float64, device="cuda")
    for i in range(len(src)):
        out[i] = _exact_map(w, geo, src[i], expo[i], u[i], part[i], means)
    out = out.view(len(src), w.naxis1, w.naxis2, E)
    return out.cpu().numpy() if kind == "maps_host" else out
