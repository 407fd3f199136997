// xts_exposure.cu -- the sources' livetime pixels and the two IRF set-up routines
// that feed step (a) (livetime-efficiency factors, King PSF normalisation); step
// (a) itself is in xts_tables.cuh and xts_tables.cu.
//
//   a2 source pixels        exposure/exposure.cxx:42-63 + healpix/healpix.cxx:181-229
//   a4 LTF                  irf/irf.cxx:70-109
//   b1 normalize_rpsf       irf/irf.normalize_rpsf.cpp:11-61, irf/irf.hxx:22-77
#include <math.h>

#include "xts_geom.cuh"
#include "xts_internal.cuh"
#include "xts_tables.cuh"

namespace xts {

__global__ void k_src_pixels(const double* src_sph, int S, long long nside, long long* pix) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < S) pix[s] = src_pixel(src_sph, s, nside);
}

int launch_src_pixels(const double* src_sph, int S, long long nside, long long* pix, cudaStream_t st) {
    if (S > 0)
        XTS_LAUNCH("k_src_pixels", st, k_src_pixels<<<(S + 127) / 128, 128, 0, st>>>(src_sph, S, nside, pix));
    return XTS_OK;
}

// a4: piecewise-linear efficiency in log E.  Row 1 from p0, row 0 from p1, and
// the break offsets b1, b2 in float, as the reference's float parameters give.
__device__ inline double ltf_single(const float* p, double logE) {
    float a0 = p[0], b0 = p[1], a1 = p[2], lb1 = p[3], a2 = p[4], lb2 = p[5];
    float b1f = __fadd_rn(__fmul_rn(__fsub_rn(a0, a1), lb1), b0);
    float b2f = __fadd_rn(__fmul_rn(__fsub_rn(a1, a2), lb2), b1f);
    double b1 = b1f, b2 = b2f;
    return logE < lb1 ? (double)a0 * logE + (double)b0
         : logE < lb2 ? (double)a1 * logE + b1
                      : (double)a2 * logE + b2;
}

__global__ void k_ltf(const double* logEs, int E, const float* p0, const float* p1, double* out) {
    int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= E) return;
    out[E + e] = ltf_single(p0, logEs[e]);
    out[e] = ltf_single(p1, logEs[e]);
}

int launch_ltf(const double* logEs, int E, const float* p0, const float* p1, double* ltf,
               cudaStream_t st) {
    XTS_LAUNCH("k_ltf", st, k_ltf<<<(E + 63) / 64, 64, 0, st>>>(logEs, E, p0, p1, ltf));
    return XTS_OK;
}

// b1: King normalisation.  64-point Gauss-Legendre below 120 MeV, analytic
// integral to 90 degrees above (irf/irf.normalize_rpsf.cpp:39-61).
__constant__ double c_gl_nodes[64];
__constant__ double c_gl_weights[64];

__device__ inline double king_f(double u, double g) {
    if (g == 1) g = 1.001;
    return (1. - 1. / g) * pow(1. + u / g, -g);
}

__device__ inline double evaluate_king(double sep, double sf, const double* p) {  // irf/irf.hxx:22-45
    double ncore = p[0], ntail = p[1], score = p[2] * sf, stail = p[3] * sf;
    double rc = sep / score, uc = rc * rc / 2.;
    double rt = sep / stail, ut = rt * rt / 2.;
    return ncore * king_f(uc, p[4]) + ntail * ncore * king_f(ut, p[5]);
}

__device__ inline double base_integral(double radius, double sf, const double* p) {  // irf/irf.hxx:48-77
    double ncore = p[0], ntail = p[1], score = p[2] * sf, stail = p[3] * sf;
    double sep = radius * D2R;
    double rc = sep / score, uc = rc * rc / 2.;
    double rt = sep / stail, ut = rt * rt / 2.;
    double fc = 1. - pow(1. + uc / p[4], 1. - p[4]);
    double ft = 1. - pow(1. + ut / p[5], 1. - p[5]);
    return ncore * fc * TWOPI * score * score + ntail * ncore * ft * TWOPI * stail * stail;
}

__global__ void k_normalize_rpsf(double* params, int Mc, int Me, const double* glog, float sp0,
                                 float sp1, float si) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= Mc * Me) return;
    int e = i % Me;
    double* p = params + (size_t)i * 6;
    double energy = pow(10.0, glog[e]);
    double tt = pow(energy * 1.e-2, (double)si);
    double sf = sqrt((double)sp0 * tt * tt + (double)sp1);
    double norm;
    if (energy < 120.) {
        double acc = 0.;
        for (int k = 0; k < 64; ++k) {
            double v = 45. * c_gl_nodes[k] + 45.;
            double x = evaluate_king(v * D2R, sf, p);
            double y = sin(v * D2R) * TWOPI * D2R;
            acc += c_gl_weights[k] * (x * y);
        }
        norm = acc * 45.;
    } else {
        norm = base_integral(90.0, sf, p);
    }
    p[0] /= norm;
    p[2] *= sf;
    p[3] *= sf;
    p[4] = p[4] == 1. ? 1.001 : p[4];
    p[5] = p[5] == 1. ? 1.001 : p[5];
}

// Gauss-Legendre nodes by Newton iteration on the Legendre recurrence
// (math/gauss_legendre.hxx:37-62), computed once on the host.
static int upload_gauss_legendre(cudaStream_t st) {
    static bool done = false;
    static int dev_done = -1;
    int dev = -1;
    cudaGetDevice(&dev);
    if (done && dev_done == dev) return XTS_OK;
    double nodes[64], wts[64];
    const int N = 64;
    for (int i = 1; i <= N; ++i) {
        double x = cos(PI * (i - 0.25) / (N + 0.5)), dp = 0.;
        for (int it = 0; it < 100; ++it) {
            double p0 = 1.0, p1 = x;
            for (int j = 2; j <= N; ++j) { double p2 = ((2 * j - 1) * x * p1 - (j - 1) * p0) / j; p0 = p1; p1 = p2; }
            dp = N * (x * p1 - p0) / (x * x - 1);
            double dx = p1 / dp;
            x -= dx;
            if (fabs(dx) <= 1e-15) break;
        }
        nodes[i - 1] = x;
        wts[i - 1] = 2.0 / ((1. - x * x) * dp * dp);
    }
    XTS_CUDA(cudaMemcpyToSymbolAsync(c_gl_nodes, nodes, sizeof(nodes), 0, cudaMemcpyHostToDevice, st));
    XTS_CUDA(cudaMemcpyToSymbolAsync(c_gl_weights, wts, sizeof(wts), 0, cudaMemcpyHostToDevice, st));
    XTS_CUDA(cudaStreamSynchronize(st));
    done = true;
    dev_done = dev;
    return XTS_OK;
}

int launch_normalize_rpsf(double* params, int Mc, int Me, const double* glog, float s0, float s1,
                          float si, cudaStream_t st) {
    int rc = upload_gauss_legendre(st);
    if (rc) return rc;
    float sp0 = s0 * s0, sp1 = s1 * s1;
    int n = Mc * Me;
    XTS_LAUNCH("k_normalize_rpsf", st, k_normalize_rpsf<<<(n + 63) / 64, 64, 0, st>>>(params, Mc, Me, glog, sp0, sp1, si));
    return XTS_OK;
}

}  // namespace xts
