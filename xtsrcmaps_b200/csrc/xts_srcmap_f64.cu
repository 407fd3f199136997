// xts_srcmap_f64.cu -- the FP64 source-map path (the reference's output type) in two
// passes over the pixels, all arithmetic in FP64.
//
// Pass A, k_pixel_rows64: per (source, pixel) the 12 rule points' squared chords (the
// biquadratic form of xts_point.cuh), their table rows and weights.  Where the points lie
// in one table row or two adjacent ones, the lower row's polynomial in q / q_k - 1
// (degree 11 over two rows, fitted in long double: below 1e-16 in t) gives every point's t,
// a point past the upper edge has t' = (t - 1) e^-step in the next row (an identity of
// the reference's formula), and three row weights times the solid angle are the pixel's
// 32-byte record.  Points over up to NW64 rows, and those beyond the table's ends (the
// reference's own formula), are evaluated one by one into a window of row weights: the
// record again up to three rows, else its extension.  Pixels with more rows than NW64 (next
// to the source) are "wide": their points are evaluated here for the map integral and again
// by the write pass.  The row weights of pixels inside the boundary radius enter the block's
// row histogram (c7, as in xts_srcmap_win.cu).
//
// Pass B, k_write_rows64: value = (sum of row weight * uPsf row) * scale in flat
// (pixel, energy) order, so stores and table reads are coalesced.
//
// One thread per pixel with asin, log and exp per point, twice (integral and write), took
// 482 + 115 us for 50 sources x 151 x 203 x 29 energies; now pass A takes 137 us, on the
// geometry stream beside the exposure and mean PSF (FP64 pipe and its latency at 16 warps
// per SM; 78 us of it the pixels of two rows), and pass B 139 us (L1 and shared-memory
// bandwidth: per value 2.3 table rows of 8 bytes and 28 of its record; without the table
// loads 66, its 356 MB take 55).  Four values per thread and turn, for loads in flight,
// took 181 us.
#include <stddef.h>

#include "xts_point.cuh"

namespace xts {

constexpr int P64 = 12;  // coefficients of a row's polynomial
constexpr double P64_C = 0.0715, P64_H = 0.0755;  // centre and half-width of its d range: [-0.004, 0.147]

struct Tab64 {
    double q[ND + 1];   // squared chord of S[k], q[401] = +inf guard
    double invq[ND];
    alignas(16) double c[ND][P64];  // (g - 1) / d as a polynomial in z = (d - P64_C) / P64_H, read 16 bytes at a time
};
static_assert(offsetof(Tab64, c) % 16 == 0 && P64 % 2 == 0, "16-byte loads of a row's polynomial");
static Tab64* g_tab64[64] = {};  // per device
static __constant__ double c_wsum64;  // sum of the 12 weights

static int build_tab64(cudaStream_t st, const Tab64** out) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return set_error(XTS_ERR_ARG, "device index %d out of range", dev);
    if (g_tab64[dev]) { *out = g_tab64[dev]; return XTS_OK; }
    static Tab64 h;
    const long double D2Rl = 0.017453292519943295769236907684886127134L;
    const double xstep = log(70. / 1e-4) / (400 - 1.);
    // T_j(z) as monomials
    long double T[P64][P64] = {};
    T[0][0] = 1.0L;
    T[1][1] = 1.0L;
    for (int j = 2; j < P64; ++j)
        for (int i = 0; i < P64; ++i) T[j][i] = (i ? 2.0L * T[j - 1][i - 1] : 0.0L) - T[j - 2][i];
    h.q[ND] = INFINITY;
    for (int k = 0; k < ND; ++k) {
        const long double S = k == 0 ? 0.0L : (long double)(1e-4 * exp((k - 1) * xstep));
        const long double x = sinl(0.5L * S * D2Rl), a0 = asinl(x);
        h.q[k] = (double)(4.0L * x * x);
        h.invq[k] = k ? (double)(1.0L / (4.0L * x * x)) : 0.;
        for (int i = 0; i < P64; ++i) h.c[k][i] = 0.;
        if (k == 0) continue;
        // the interpolant starts from the rounded q[k], as the device does
        const long double q = (long double)h.q[k], x0 = 0.5L * sqrtl(q);
        long double f[P64], m[P64] = {};
        for (int i = 0; i < P64; ++i) {
            const long double z = cosl(3.14159265358979323846264338327950288L * (i + 0.5L) / P64);
            const long double d = (long double)P64_C + (long double)P64_H * z;
            f[i] = ((asinl(x0 * sqrtl(1.0L + d)) - a0) / a0) / d;
        }
        for (int j = 0; j < P64; ++j) {
            long double s = 0;
            for (int i = 0; i < P64; ++i) s += f[i] * cosl(j * 3.14159265358979323846264338327950288L * (i + 0.5L) / P64);
            s *= (j == 0 ? 1.0L : 2.0L) / P64;
            for (int i = 0; i < P64; ++i) m[i] += s * T[j][i];
        }
        for (int i = 0; i < P64; ++i) h.c[k][i] = (double)m[i];
    }
    Tab64* d = nullptr;
    XTS_CUDA(cudaMalloc(&d, sizeof(Tab64)));
    XTS_CUDA(cudaMemcpyAsync(d, &h, sizeof(Tab64), cudaMemcpyHostToDevice, st));
    const double W = 2.0 * (2.0 * (0.25 * 5.2092862230230441e-01) + 2.0 * (0.25 * 2.3740240561379911e-01) +
                            2.0 * (0.25 * 2.4166897208389651e-01));
    XTS_CUDA(cudaMemcpyToSymbolAsync(c_wsum64, &W, sizeof(W), 0, cudaMemcpyHostToDevice, st));
    XTS_CUDA(cudaStreamSynchronize(st));
    g_tab64[dev] = d;
    *out = d;
    return XTS_OK;
}

constexpr int NW64 = 8;  // rows of an extension window

// A pixel's row weights (times its solid angle) from row `row`: n = 2 or 3 here, n = 4 ..
// NW64 in its extension; n = 0: a wide pixel.
struct __align__(16) Rec64 { double w0, w1, w2; int row, n; };

__device__ __forceinline__ int row_of(double q, const SepTab* __restrict__ tab) {
    int b = (__double2hiint(q) >> (20 - SB_BITS)) - (SB_EXP0 << SB_BITS);
    b = min(max(b, 0), NSB - 1);
    const int4 v = __ldg((const int4*)&tab->bins[b]);  // k0, -, thr
    return min(v.x + (q >= __hiloint2double(v.w, v.z)), ND - 2);  // (q = +inf is past the last row's end)
}

__device__ __forceinline__ double poly64(const double* c, double z) {
    double P = c[P64 - 1];
#pragma unroll
    for (int i = P64 - 2; i >= 0; --i) P = fma(P, z, c[i]);
    return P;
}

__device__ __forceinline__ void row_poly(const Tab64* __restrict__ t64, int k, double* c) {
#pragma unroll
    for (int i = 0; i < P64; i += 2) {
        const double2 v = __ldg((const double2*)&t64->c[k][i]);
        c[i] = v.x;
        c[i + 1] = v.y;
    }
}

// Lower row and weight t of one point by itself.
__device__ __noinline__ int point64(double q, const SepTab* __restrict__ tab, const Tab64* __restrict__ t64, double* t) {
    const int k = row_of(q, tab);
    const double d = (q - t64->q[k]) * t64->invq[k];
    if (d >= P64_C - P64_H && d <= P64_C + P64_H) {
        double c[P64];
        row_poly(t64, k, c);
        *t = REDM1 * (d * poly64(c, (d - P64_C) * (1.0 / P64_H)));
    } else {  // s < 1e-4 deg or s >= 70 deg: the reference's formula (convolve_pixel_psf_logsep.hpp:45-47)
        const double s = 2.0 * R2D * asin(0.5 * sqrt(q));
        *t = REDM1 * (s * 1e4 * exp(SEP_STEP * (1. - k)) - 1.);
    }
    return k;
}

__device__ __forceinline__ bool inside64(const SrcInfo& si, double ch2, const double* c) {
    const double x = si.dir[0] - c[0], y = si.dir[1] - c[1], z = si.dir[2] - c[2];
    const double d2 = x * x + y * y + z * z;
    if (d2 < ch2 * (1.0 - 1e-12)) return true;
    if (d2 > ch2 * (1.0 + 1e-12)) return false;
    return dir_diff(si.dir, c) <= si.radius_rad;
}

// Block (ch, s): pixels [ch npix / nch, (ch + 1) npix / nch) of source s.
__global__ void __launch_bounds__(256, 2) k_pixel_rows64(const double* __restrict__ corners,
                                                         const double* __restrict__ centers,
                                                         const double* __restrict__ omega,
                                                         const SrcInfo* __restrict__ info,
                                                         const SepTab* __restrict__ tab, const Tab64* __restrict__ t64,
                                                         int H, int W, int nch, Rec64* __restrict__ rec,
                                                         double* __restrict__ ext, double* __restrict__ hist_out) {
    __shared__ double hist[ND];
    __shared__ double win[NW64][256];  // slot j of a thread's window at win[j][t]
    const int s = blockIdx.y, ch = blockIdx.x, npix = H * W, W1 = W + 1;
    const SrcInfo si = info[s];
    for (int r = threadIdx.x; r < ND; r += blockDim.x) hist[r] = 0.;
    __syncthreads();
    double ch2 = 2.0 * sin(0.5 * si.radius_rad);
    ch2 *= ch2;
    const double em = REDM1 / (REDM1 + 1.0);  // e^-step
    const int p1 = (int)((long long)npix * (ch + 1) / nch);
    for (int pix = (int)((long long)npix * ch / nch) + threadIdx.x; pix < p1; pix += blockDim.x) {
        const int h = pix / W, w = pix - h * W;
        const PixQ g = pixel_q(pixel_geom(corners, W1, h, w, si));
        const double om = omega[pix];
        const bool inside = si.in_fov && inside64(si, ch2, centers + 3 * ((size_t)h * W1 + w));
        double q[12], mn = INFINITY, mx = -INFINITY;
#pragma unroll
        for (int p = 0; p < 12; ++p) {
            q[p] = point_q2(g, p);
            mn = fmin(mn, q[p]);
            mx = fmax(mx, q[p]);
        }
        const int k = row_of(mn, tab);
        const double qk = __ldg(&t64->q[k]), iq = __ldg(&t64->invq[k]);
        // two rows end at q[k + 2]; the last row (399) goes on past the table's end
        const double edge = k < ND - 2 ? __ldg(&t64->q[k + 1]) : INFINITY;
        const double top = k < ND - 2 ? __ldg(&t64->q[k + 2]) : qk * (1.0 + P64_C + P64_H);
        Rec64 R;
        R.row = k;
        R.n = 0;
        R.w0 = R.w1 = R.w2 = 0.;
        // (mx >= mn fails where every q is NaN, as for a source without a finite position: fmin and
        // fmax skip NaN and leave mn = +inf, mx = -inf)
        if (mx >= mn && mn >= qk && mx < top) {
            double c[P64];
            row_poly(t64, k, c);
            double T = 0., S2 = 0.;
#pragma unroll
            for (int p = 0; p < 12; ++p) {
                const double d = (q[p] - qk) * iq, wp = c_rule_uv[p][3];
                const double u = fma(REDM1 * d, poly64(c, (d - P64_C) * (1.0 / P64_H)), -1.0);
                T = fma(wp, u, T);
                S2 = fma(q[p] >= edge ? wp : 0., u, S2);
            }
            R.n = mx >= edge ? 3 : 2;
            R.w0 = om * (S2 - T);
            R.w2 = om * (em * S2);
            R.w1 = fma(om, c_wsum64, -R.w0) - R.w2;
            if (inside) {
                atomicAdd(&hist[k], R.w0);
                atomicAdd(&hist[k + 1], R.w1);
                if (R.n == 3) atomicAdd(&hist[k + 2], R.w2);
            }
        } else {
            const int k1 = row_of(mx, tab), t = threadIdx.x;
            const int n = mx >= mn ? k1 - k + 2 : 0;
            // (2 or 3 rows: points beyond the table's ends.  As wide pixels, evaluated again for every
            // energy, they took all-sky maps of 1 degree, 20 sources x 37 energies, 1654 us; 448 so)
            const bool windowed = n > 0 && n <= NW64;
            if (windowed)
                for (int j = 0; j < n; ++j) win[j][t] = 0.;
            if (windowed || inside)
                for (int p = 0; p < 12; ++p) {
                    double tp;
                    const int kp = point64(point_q2(g, p), tab, t64, &tp);
                    const double wp = c_rule_uv[p][3] * om, a = (1.0 - tp) * wp, b = tp * wp;
                    if (windowed) {
                        win[kp - k][t] += a;
                        win[kp - k + 1][t] += b;
                    } else {
                        atomicAdd(&hist[kp], a);
                        atomicAdd(&hist[kp + 1], b);
                    }
                }
            if (windowed) {
                R.n = n;
                double* x = ext + ((size_t)s * npix + pix) * NW64;
                for (int j = 0; j < n; ++j) {
                    const double v = win[j][t];
                    if (n > 3) x[j] = v;
                    if (inside) atomicAdd(&hist[k + j], v);
                }
                if (n <= 3) {
                    R.w0 = win[0][t];
                    R.w1 = win[1][t];
                    if (n == 3) R.w2 = win[2][t];
                }
            } else if (n == 0) {  // no finite point: NaN from any two rows
                R.n = 2;
                R.w0 = R.w1 = __longlong_as_double(0x7ff8000000000000ll);
            }
        }
        double2* o = (double2*)(rec + (size_t)s * npix + pix);
        o[0] = make_double2(R.w0, R.w1);
        o[1] = make_double2(R.w2, __hiloint2double(R.n, R.row));
    }
    __syncthreads();
    double* out = hist_out + ((size_t)s * nch + ch) * ND;
    for (int r = threadIdx.x; r < ND; r += blockDim.x) out[r] = hist[r];
}

constexpr int B64 = 128;  // pixels per block of the write pass

__global__ void __launch_bounds__(256) k_write_rows64(const double* __restrict__ corners,
                                                      const double* __restrict__ omega,
                                                      const SrcInfo* __restrict__ info,
                                                      const SepTab* __restrict__ tab, const Tab64* __restrict__ t64,
                                                      const Rec64* __restrict__ rec, const double* __restrict__ ext,
                                                      const double* __restrict__ upsf,
                                                      const double* __restrict__ scale, int H, int W, int E,
                                                      unsigned magic, double* __restrict__ out) {
    after_previous();
    __shared__ Rec64 sr[B64];
    __shared__ double2 wide[8][12];  // per warp the points of a wide pixel: t, row
    const int s = blockIdx.y, npix = H * W, pix0 = blockIdx.x * B64, np = min(B64, npix - pix0);
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    {
        const double2* r = (const double2*)(rec + (size_t)s * npix + pix0);
        double2* o = (double2*)sr;
        for (int k = t; k < 2 * np; k += 256) {
            double2 v = __ldg(r + k);
            o[k] = v;  // (the second half ends in n and row as its last double's words)
        }
    }
    __syncthreads();
    const double* U = upsf + (size_t)s * ND * E;
    const double* sc = scale + (size_t)s * E;
    double* o = out + ((size_t)s * npix + pix0) * E;
    const long long n = (long long)np * E;
    for (long long f = t; f < n; f += 256) {
        // pixel of the flat index: exact by the rounded-up reciprocal while f E < 2^32
        const int p = magic ? (int)__umulhi((unsigned)f, magic) : (int)(f / E);
        const int e = (int)(f - (long long)p * E);
        const Rec64& r = sr[p];
        const double* y = U + (size_t)r.row * E + e;
        double v;
        if (r.n == 2 || r.n == 3) {
            v = fma(r.w1, __ldg(y + E), r.w0 * __ldg(y));
            if (r.n == 3) v = fma(r.w2, __ldg(y + 2 * (size_t)E), v);
        } else if (r.n) {
            const double* x = ext + ((size_t)s * npix + pix0 + p) * NW64;
            v = 0.;
            for (int j = 0; j < r.n; ++j, y += E) v = fma(__ldg(x + j), __ldg(y), v);
        } else {
            continue;
        }
        __stcs(o + f, v * __ldg(sc + e));
    }
    // wide pixels: a warp each, its points one per lane, then lane = energy
    static_assert(B64 == 16 * 8, "lane l < 16 looks at pixel warp + 8 l");
    unsigned todo = __ballot_sync(0xffffffffu, lane < 16 && warp + 8 * lane < np && sr[warp + 8 * (lane & 15)].n == 0);
    while (todo) {
        const int p = warp + 8 * (__ffs(todo) - 1);
        todo &= todo - 1;
        const int pix = pix0 + p, h = pix / W, w = pix - h * W;
        if (lane < 12) {
            const SrcInfo si = info[s];
            double tt;
            const int k = point64(point_q2(pixel_q(pixel_geom(corners, W + 1, h, w, si)), lane), tab, t64, &tt);
            wide[warp][lane] = make_double2(tt, (double)k);
        }
        __syncwarp();
        const double om = omega[pix];
        for (int e = lane; e < E; e += 32) {
            double v = 0.;
            for (int i = 0; i < 12; ++i) {
                const double2 a = wide[warp][i];
                const double* y = U + (size_t)(int)a.y * E + e;
                v += c_rule_uv[i][3] * ((1.0 - a.x) * __ldg(y) + a.x * __ldg(y + E));
            }
            o[(size_t)p * E + e] = (v * om) * __ldg(sc + e);
        }
        __syncwarp();
    }
}

// Chunks per source of the histogram: about four blocks per resident one (two per SM), at
// least 4 pixels per thread.
static int rows64_chunks(int S, int npix, int nsm) {
    int n = (8 * nsm + S - 1) / S;
    const int mx = (npix + 1023) / 1024;
    return n < 1 ? 1 : (n > mx ? mx : n);
}

int launch_srcmap_f64(const double* corners, const double* centers, const double* omega, const SrcInfo* info, int S,
                      int H, int W, int E, const double* upsf, const double* partial, const double* exposure,
                      double* scale, double* inv_integ, double* correction, double* radius, int* in_fov, double* out,
                      StreamJoin& geo, cudaStream_t st) {
    int rc = upload_rule_uv(st);
    if (rc) return rc;
    const SepTab* tab = nullptr;
    const Tab64* t64 = nullptr;
    if ((rc = build_septab(st, &tab)) || (rc = build_tab64(st, &t64))) return rc;
    const int npix = H * W;
    int dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    // sources per chunk: records of at most 1 GiB (extensions 2 GiB), fewer where the GPU's
    // memory does not hold those, so that a map that fills it needs room for one source's
    long long Sc = ((long long)1 << 30) / ((long long)npix * (long long)sizeof(Rec64));
    Sc = Sc < 1 ? 1 : (Sc > S ? S : Sc);
    int nch;
    Rec64* rec;
    double *hist, *ext;
    for (;; Sc = (Sc + 1) / 2) {
        nch = rows64_chunks((int)Sc, npix, nsm);
        rec = (Rec64*)workspace(W_WIN, sizeof(Rec64) * (size_t)Sc * npix);
        ext = (double*)workspace(W_WMETA, sizeof(double) * NW64 * (size_t)Sc * npix);
        hist = (double*)workspace(W_PARTSUM, sizeof(double) * (size_t)Sc * nch * ND);
        if (rec && ext && hist) break;
        if (Sc == 1) return XTS_ERR_OOM;
        workspace_free(W_WIN);
        workspace_free(W_WMETA);
    }
    // f E < 2^32 for every flat index f < B64 E of a tile
    const unsigned magic = E > 1 && (unsigned long long)B64 * E * E < (1ull << 32) ? 0xffffffffu / (unsigned)E + 1u : 0u;
    for (int s0 = 0; s0 < S; s0 += (int)Sc) {
        const int n = S - s0 < (int)Sc ? S - s0 : (int)Sc;
        const size_t oE = (size_t)s0 * E;
        // the row pass needs the geometry only: the first chunk's runs on the geometry stream,
        // beside the exposure and mean PSF of a fused call
        const cudaStream_t rs = s0 == 0 ? geo.from : st;
        XTS_LAUNCH("k_pixel_rows64", rs, k_pixel_rows64<<<dim3(nch, n), 256, 0, rs>>>(corners, centers, omega, info + s0,
                                                                                     tab, t64, H, W, nch, rec, ext, hist));
        if ((rc = geo.join())) return rc;
        rc = launch_correction(hist, nch, info + s0, n, upsf + oE * ND, partial + oE * ND, exposure + oE, E, scale + oE,
                               inv_integ ? inv_integ + oE : nullptr, correction ? correction + oE : nullptr,
                               radius ? radius + s0 : nullptr, in_fov ? in_fov + s0 : nullptr, st);
        if (rc) return rc;
        XTS_LAUNCH("k_srcmap_f64", st, launch_next(k_write_rows64, dim3((npix + B64 - 1) / B64, n), 256, 0, st,
                                           corners, omega, info + s0, tab, t64, rec, ext, upsf + oE * ND, scale + oE, H, W,
                                           E, magic, out + (size_t)s0 * npix * E));
    }
    return XTS_OK;
}

}  // namespace xts
