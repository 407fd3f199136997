// xts_tables.cuh -- the entries of the small per-call tables of steps (a) and (b), each
// by one thread (or, psf*aeff, one block), for the launches of xts_tables.cu.
//
//   a1 exp_costhetas        exposure/exposure.cxx:29-40
//   a2 src_cosbins (gather) exposure/exposure.cxx:42-63 + healpix/healpix.cxx:181-229
//   a3 aeff_value           irf/irf.aeff_value.cxx:11-55, math/bilerp.cxx:6-27
//   a5 exposure contraction exposure/exposure.cxx:159-263, exposure/exposure.contract.cpp:13-42
//   b2 separations          psf/psf.hxx:24-31
//   b3 King table           psf/psf.king.cxx:9-43
//   b4 bilerp               psf/psf.bilerp.cxx:6-52
#pragma once

#include <math.h>

#include "xts_geom.cuh"
#include "xts_internal.cuh"

namespace xts {

// math/bilerp.cxx:6-27: upper_bound index, weight and complement.  The
// reference asserts the value lies inside the grid; the index is clamped to the
// last interval here instead of reading past the end.
static __device__ __forceinline__ void lerp_pars(const double* g, int n, double v, bool has_lb, double lb,
                                 double* wgt, double* cmpl, int* idx) {
    if (has_lb && v < lb) { *wgt = 0.; *cmpl = 0.; *idx = 1; return; }
    int lo = 0, hi = n;  // first i with g[i] > v
    while (lo < hi) { int m = (lo + hi) >> 1; if (v < g[m]) hi = m; else lo = m + 1; }
    int i = lo < 1 ? 1 : (lo > n - 1 ? n - 1 : lo);
    double t = (v - g[i - 1]) / (g[i] - g[i - 1]);
    *wgt = t; *cmpl = 1. - t; *idx = i;
}

// a1 + a3: cos-theta bin centres and the front/back effective-area tables [C, E].
static __device__ __forceinline__ void exposure_table(int i, int C, double cosmin, int thetabin, const double* logEs,
                                                      int E, const xts_grid& af, const xts_grid& ab, double* costh,
                                                      double* front, double* back) {
    if (i >= C * E) return;
    int c = i / E, e = i - c * E;
    double f = ((double)c + 0.5) / C;
    f = thetabin ? f * f : f;
    double ct = 1. - f * (1. - cosmin);
    if (e == 0) costh[c] = ct;
    const xts_grid* gs[2] = {&af, &ab};
    double* outs[2] = {front, back};
    for (int k = 0; k < 2; ++k) {
        const xts_grid& g = *gs[k];
        double cw, cc, ew, ec; int ci, ei;
        lerp_pars(g.cosths, g.n_cos, ct, true, g.min_cos_theta, &cw, &cc, &ci);
        lerp_pars(g.logEs, g.n_e, logEs[e], false, 0., &ew, &ec, &ei);
        int Me = g.n_e;
        const double* P = g.params;
        double xx = cc * ec * P[(ci - 1) * Me + (ei - 1)];
        double xy = cc * ew * P[(ci - 1) * Me + ei];
        double yx = cw * ec * P[ci * Me + (ei - 1)];
        double yy = cw * ew * P[ci * Me + ei];
        outs[k][i] = 1e4 * (xx + xy + yx + yy);
    }
}

// The NESTED pixel of each source (exposure/exposure.cxx:42-63), -1 when the
// position is not finite.
static __device__ __forceinline__ long long src_pixel(const double* src_sph, int s, long long nside) {
    const double theta = HALFPI - src_sph[2 * s + 1] * D2R;
    const double phi = D2R * src_sph[2 * s];
    const long long pix = ang2pix_nest(theta, phi, nside);
    return pix < 0 || pix >= 12 * nside * nside ? -1 : pix;
}

// a2: livetime rows of each source's NESTED pixel, float -> double [S, C].  With
// `gathered` the cubes hold only those rows already, [S][C] in source order.
static __device__ __forceinline__ void src_cosbin(int i, const double* src_sph, int S, const float* cube,
                                                  const float* wcube, long long nside, int C, bool gathered,
                                                  double* ecb, double* wecb) {
    if (i >= S * C) return;
    int s = i / C, c = i - s * C;
    const long long pix = gathered ? s : src_pixel(src_sph, s, nside);
    if (pix < 0) {  // non-finite source position
        ecb[i] = wecb[i] = __longlong_as_double(0x7ff8000000000000ll);
        return;
    }
    ecb[i] = (double)cube[pix * C + c];
    wecb[i] = (double)wcube[pix * C + c];
}

// a5 on FP64 cores: E[s,e] = ((X.Af L0 + X.Ab L0) + W.Af L1) + W.Ab L1.
static __device__ __forceinline__ void exposure_value(int i, const double* ecb, const double* wecb, int S, int C,
                                                      const double* af, const double* ab, const double* ltf, int E,
                                                      double* out) {
    if (i >= S * E) return;
    int s = i / E, e = i - s * E;
    double ef = 0, wf = 0, eb = 0, wb = 0;
#pragma unroll 8
    for (int c = 0; c < C; ++c) {  // unrolled: eight rows of loads in flight, sums still in c order
        double x = ecb[s * C + c], w = wecb[s * C + c];
        double a = af[c * E + e], b = ab[c * E + e];
        ef = fma(x, a, ef); wf = fma(w, a, wf);
        eb = fma(x, b, eb); wb = fma(w, b, wb);
    }
    double l0 = ltf[e], l1 = ltf[E + e];
    out[i] = ((ef * l0 + eb * l0) + wf * l1) + wb * l1;
}

static __device__ __forceinline__ double sep_deg(int d) {  // psf/psf.hxx:24-31
    const double xstep = log(70. / 1e-4) / (400 - 1.);
    return d == 0 ? 0.0 : 1e-4 * exp((d - 1) * xstep);
}

static __device__ __forceinline__ double king_f2(double u, double g) {
    if (g == 1) g = 1.001;
    return (1. - 1. / g) * pow(1. + u / g, -g);
}

// b3: K[side][c][e][d] = evaluate_king(sep[d] rad, 1, params[c,e,:]) (irf/irf.hxx:22-45);
// the separation is the fastest axis of this table and of psf*aeff, so that the
// contraction below reads runs of rows of one energy.
static __device__ __forceinline__ void king_entry(int i, const xts_grid& g, double* out) {
    int McMe = g.n_cos * g.n_e;
    if (i >= ND * McMe) return;
    int ce = i / ND, d = i - ce * ND;
    const double* p = g.params + (size_t)ce * 6;
    double sep = sep_deg(d) * D2R;
    double ncore = p[0], ntail = p[1], score = p[2], stail = p[3];
    double rc = sep / score, uc = rc * rc / 2.;
    double rt = sep / stail, ut = rt * rt / 2.;
    out[i] = ncore * king_f2(uc, p[4]) + ntail * ncore * king_f2(ut, p[5]);
}

// b4 + the aeff product of b5, both sides summed: PA[c][e][d], rows padded to NDP.
// One block per (e, c), whose bilinear weights four threads look up.
constexpr int NDP = (ND + 3) / 4 * 4;

static __device__ __forceinline__ void psf_aeff_block(int e, int c, const xts_grid& pf, const xts_grid& pb,
                                                      const double* kf, const double* kb, const double* costh, int C,
                                                      const double* logEs, int E, const double* af, const double* ab,
                                                      double* pa) {
    __shared__ double wgt[4], cmpl[4];  // side 0 energy, cos-theta, side 1 energy, cos-theta
    __shared__ int idx[4];
    if (threadIdx.x < 4) {
        const int k = threadIdx.x;
        const xts_grid& g = k >> 1 ? pb : pf;
        if (k & 1) lerp_pars(g.cosths, g.n_cos, costh[c], false, 0., &wgt[k], &cmpl[k], &idx[k]);
        else lerp_pars(g.logEs, g.n_e, logEs[e], false, 0., &wgt[k], &cmpl[k], &idx[k]);
    }
    __syncthreads();
    // the padding rows enter the totals with weight 0
    if (threadIdx.x < NDP - ND) pa[((size_t)c * E + e) * NDP + ND + threadIdx.x] = 0.;
    for (int d = threadIdx.x; d < ND; d += blockDim.x) {
        double v = 0.;
        for (int side = 0; side < 2; ++side) {
            const xts_grid& g = side ? pb : pf;
            const double ew = wgt[2 * side], ec = cmpl[2 * side], cw = wgt[2 * side + 1], cc = cmpl[2 * side + 1];
            const int ei = idx[2 * side], ci = idx[2 * side + 1], Me = g.n_e;
            const double* K = (side ? kb : kf) + d;
            const size_t r0 = (size_t)((ci - 1) * Me + ei - 1) * ND, r1 = (size_t)(ci * Me + ei - 1) * ND;
            double b = cc * ec * K[r0] + cc * ew * K[r0 + ND] + cw * ec * K[r1] + cw * ew * K[r1 + ND];
            v += b * (side ? ab : af)[c * E + e];
        }
        pa[((size_t)c * E + e) * NDP + d] = v;
    }
}

// Row tables of the integral, [NDP] each: 2 pi sin(theta), half the widths of the bins that
// end there, and the row's weight in the integral over all bins.
static __device__ __forceinline__ void psf_row(int d, double* tab) {
    if (d >= NDP) return;
    const double th = D2R * sep_deg(d);
    tab[d] = d < ND ? TWOPI * sin(th) : 0.;
    const double below = d > 0 && d < ND ? 0.5 * (th - D2R * sep_deg(d - 1)) : 0.;
    const double above = d + 1 < ND ? 0.5 * (D2R * sep_deg(d + 1) - th) : 0.;
    tab[NDP + d] = below;
    tab[2 * NDP + d] = tab[d] * (below + above);
}

}  // namespace xts
