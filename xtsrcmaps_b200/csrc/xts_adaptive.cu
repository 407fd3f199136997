// xts_adaptive.cu -- adaptive cubature of the pixel-mean PSF (the design of the
// reference's uncompiled math/genz_malik.hxx:18-195):
// the published Genz-Malik degree-7/5 rule for two dimensions (A.C. Genz,
// A.A. Malik, J. Comput. Appl. Math. 6 (1980) 295-302; weights as updated by
// Bernstein, Espelid and Genz), the design the reference lays out in
// math/genz_malik.hxx:18-85 and math/genz_malik.cxx:66-217 (not compiled there),
// with rectangular sub-regions and the estimate kept at the depth limit.
//
// Work is scheduled by region, not by pixel, so that pixels needing many regions
// (next to the source) do not hold up the others.  One persistent launch (a
// cooperative grid, every block resident) runs all levels: level 0 evaluates
// every (source, pixel)'s whole-pixel region and writes accepted pixels' means;
// an unaccepted region pushes its two halves onto a device-side queue; after a
// grid-wide barrier (bounded waits) the next level takes the previous level's
// queue.  A warp takes 32 regions, forms their windows a region per lane and their
// energies eight lanes (or all) to a region; accepted regions add area * R7 into their
// pixel's FP64 mean with FP64 atomics (order-free to within a few FP64 ulps).
// The queue has a fixed capacity; a region whose halves do not fit is accepted
// as it is.
//
// Decisions near the threshold are taken in FP64: when the FP32 estimate of
// max_e |R5 - R7| / |R7| lies within 5 % of rtol (and within its FP32 error, 4e-6), or the
// two fourth differences that choose the split dimension are within 0.1 % of each other (and
// their FP32 error, 4e-6 of the summed values), or the points leave the row window, the region is
// evaluated again point by point in FP64 from the FP64 mean PSF, with the
// reference design's arithmetic (math/genz_malik.hxx:127-195) and no fused
// multiply-adds, and that evaluation decides (and gives the value).  These regions are
// queued per level and taken one per warp.
//
// A region's 17 points give LUT rows and interpolation weights exactly as the
// 12-point rule's do (xts_point.cuh: FP64 chord of the corner-vector blend,
// exact row, per-row t polynomial).  When they span at most AW consecutive rows,
// four row windows are formed (the degree-7 value, degree-5 minus degree-7, and
// the two fourth divided differences that choose the split dimension) and dotted
// with the source's FP32 mean-PSF rows for every energy; otherwise the region is
// evaluated in FP64.  A region is accepted when
// max_e |R5 - R7| / |R7| <= rtol or at the depth limit; otherwise it is halved
// along the dimension with the larger summed fourth difference.
//
// k_mean_integral then sums mean * solid angle over the pixels inside the
// boundary radius (FP64, fixed order), k_correction_sums forms the scales, and
// k_scale_map64 writes value = mean * solid angle * exposure * correction.
#include "xts_point.cuh"

namespace xts {

constexpr int AT = 256;     // threads per block
constexpr int AW = 8;       // rows of a region window

// Points of the rule in half-widths along (dimension 0 = map axis h, dimension 1
// = map axis w) and the coefficients of the four windows per point.
struct GmRule {
    float off0[17], off1[17];
    float w7[17], wd[17], d0[17], d1[17];
};
static __constant__ GmRule c_gm;
struct GmRule64 { double off0[17], off1[17], w7[17], w5[17]; };  // the same rule in FP64
static __constant__ GmRule64 c_gm64;
static int upload_gm(cudaStream_t st) {
    static int dev_done = -1;
    int dev = -1;
    cudaGetDevice(&dev);
    if (dev_done == dev) return XTS_OK;
    const double l2 = 0.35856858280031809199064515390793749545406372969943071;  // sqrt(9/70)
    const double l4 = 0.94868329805051379959966806332981556011586654179756505;  // sqrt(9/10)
    const double l5 = 0.68824720161168529772162873429362352512689535661564885;  // sqrt(9/19)
    // centre; +-l2 on each axis; +-l4 on each axis; (+-l4, +-l4); (+-l5, +-l5)
    const double o[17][2] = {{0, 0},     {-l2, 0},   {0, -l2},  {l2, 0},   {0, l2},   {-l4, 0},
                             {0, -l4},   {l4, 0},    {0, l4},   {-l4, -l4}, {l4, -l4}, {-l4, l4},
                             {l4, l4},   {-l5, -l5}, {-l5, l5}, {l5, -l5},  {l5, l5}};
    const double a7 = (12824. - 9120. * 2. + 400. * 4.) / 19683., b7 = 980. / 6561.;
    const double c7 = (1820. - 400. * 2.) / 19683., d7 = 200. / 19683., f7 = 6859. / 19683. / 4.;
    const double a5 = (729. - 950. * 2. + 50. * 4.) / 729., b5 = 245. / 486.;
    const double c5 = (265. - 100. * 2.) / 1458., d5 = 25. / 729.;
    GmRule g;
    GmRule64 g64;
    for (int p = 0; p < 17; ++p) {
        const double w7 = p == 0 ? a7 : p < 5 ? b7 : p < 9 ? c7 : p < 13 ? d7 : f7;
        const double w5 = p == 0 ? a5 : p < 5 ? b5 : p < 9 ? c5 : p < 13 ? d5 : 0.;
        g64.off0[p] = o[p][0];
        g64.off1[p] = o[p][1];
        g64.w7[p] = w7;
        g64.w5[p] = w5;
        g.off0[p] = (float)o[p][0];
        g.off1[p] = (float)o[p][1];
        g.w7[p] = (float)w7;
        g.wd[p] = (float)(w5 - w7);
        // fourth differences: (f(-l2) + f(+l2) - 2 f0) - (l2/l4)^2 (f(-l4) + f(+l4) - 2 f0)
        double e0 = 0., e1 = 0.;
        if (p == 0) e0 = e1 = -2. + 2. / 7.;
        if (p == 1 || p == 3) e0 = 1.;
        if (p == 5 || p == 7) e0 = -1. / 7.;
        if (p == 2 || p == 4) e1 = 1.;
        if (p == 6 || p == 8) e1 = -1. / 7.;
        g.d0[p] = (float)e0;
        g.d1[p] = (float)e1;
    }
    XTS_CUDA(cudaMemcpyToSymbolAsync(c_gm, &g, sizeof(g), 0, cudaMemcpyHostToDevice, st));
    XTS_CUDA(cudaMemcpyToSymbolAsync(c_gm64, &g64, sizeof(g64), 0, cudaMemcpyHostToDevice, st));
    XTS_CUDA(cudaStreamSynchronize(st));
    dev_done = dev;
    return XTS_OK;
}

// One queued region: its pixel (source * npix + pixel) and its rectangle in the
// pixel's [-1, 1]^2 parameter square.
struct QRegion { int sp; float c0, c1, h0, h1; };

// Shared memory: the separation tables, then per warp the row windows of its 32
// regions ([32][AW] float4 (w7, wd, d0, d1), one float4 of padding per region so that
// lanes' 16-byte accesses fall in different banks) and the 17 points of the region
// that the warp evaluates in FP64.
constexpr int ADAPT_BLOCKS = 2;  // per SM
constexpr int TH = 4, TW = 8;    // pixels of a warp's patch at level 0
constexpr int WSTRIDE = AW + 1;
constexpr int NWARP = AT / 32;
struct Point64 { double t; int idx; };
constexpr size_t AO_SQ = 0;
constexpr size_t AO_COEF = (8 * (ND + 1) + 15) / 16 * 16;
constexpr size_t AO_WIN = AO_COEF + sizeof(float4) * 2 * ND;
constexpr size_t AO_P64 = AO_WIN + sizeof(float4) * NWARP * 32 * WSTRIDE;
constexpr size_t A_SMEM = AO_P64 + sizeof(Point64) * NWARP * 17;

// One region of a warp's batch, as its lane holds it.
struct LaneRegion {
    int sp, s, h, w;  // source * npix + pixel, source, map row and column
    float c0, c1, h0, h1;
};

// What the levels share.
struct LevelArgs {
    const double* corners; const SrcInfo* info; const float* lut; const double* upsf;
    int H, W, E, EP;
    float rtol;
    double* mean;
};

__device__ __forceinline__ double shfl_d(double v, int src) { return __shfl_sync(0xffffffffu, v, src); }

// A region again in FP64 by the whole warp, with the reference design's arithmetic
// (math/genz_malik.hxx:127-195 as restated by the oracle): lane p blends rule point p
// from the pixel's corner vectors, s = 2 asin(|p - src| / 2), the logsep row and
// weight; then lane = energy: f = (1 - t) U[i - 1] + t U[i], R7 and R5 summed over the
// points in order, the fourth differences summed over the energies in order, no fused
// multiply-adds.  Returns true when the region is accepted, after adding (at level 0:
// storing) area * R7 into its mean; otherwise sets *dim (at level 0 the mean is
// cleared).  All arguments are warp-uniform.
__device__ __noinline__ bool gm_region64(const LevelArgs& A, const LaneRegion& R, Point64* pts, bool last, bool level0,
                                         int* dim) {
    const int lane = threadIdx.x & 31, W1 = A.W + 1, E = A.E;
    const double* U = A.upsf + (size_t)R.s * ND * E;
    double* mean = A.mean + (size_t)R.sp * E;
    __syncwarp();
    if (lane < 17) {
        const double* a = A.corners + 3 * ((size_t)R.h * W1 + R.w);            // LL
        const double* b = A.corners + 3 * ((size_t)R.h * W1 + R.w + 1);        // LR
        const double* c = A.corners + 3 * ((size_t)(R.h + 1) * W1 + R.w + 1);  // UR
        const double* d = A.corners + 3 * ((size_t)(R.h + 1) * W1 + R.w);      // UL
        const double* src = A.info[R.s].dir;
        const double u = __dadd_rn(R.c1, __dmul_rn(c_gm64.off1[lane], R.h1));
        const double v = __dadd_rn(R.c0, __dmul_rn(c_gm64.off0[lane], R.h0));
        const double nn = __dmul_rn(__dsub_rn(1.0, u), __dsub_rn(1.0, v));
        const double pn = __dmul_rn(__dadd_rn(1.0, u), __dsub_rn(1.0, v));
        const double pp = __dmul_rn(__dadd_rn(1.0, u), __dadd_rn(1.0, v));
        const double np = __dmul_rn(__dsub_rn(1.0, u), __dadd_rn(1.0, v));
        double q2 = 0.;
        for (int k = 0; k < 3; ++k) {
            const double bl = __dadd_rn(__dadd_rn(__dadd_rn(__dmul_rn(nn, a[k]), __dmul_rn(pn, b[k])), __dmul_rn(pp, c[k])),
                                        __dmul_rn(np, d[k]));
            const double qk = __dsub_rn(__dmul_rn(0.25, bl), src[k]);
            q2 = __dadd_rn(q2, __dmul_rn(qk, qk));
        }
        const double sd = 2.0 * R2D * asin(0.5 * sqrt(q2));
        const double j = sd < 1e-4 ? 1. : __dadd_rn(1., __dmul_rn(RECIPSTEP, __dadd_rn(LN_1E4, log(sd))));
        int idx = 1 + (int)(unsigned short)j;
        idx = idx > 400 ? 400 : idx;
        pts[lane].idx = idx;
        pts[lane].t = __dmul_rn(REDM1, __dsub_rn(__dmul_rn(__dmul_rn(sd, 1e4), exp(__dmul_rn(SEP_STEP, 2. - idx))), 1.));
    }
    __syncwarp();
    auto value = [&](int p, int e) {
        const int i = pts[p].idx;
        const double t = pts[p].t;
        return __dadd_rn(__dmul_rn(__dsub_rn(1.0, t), U[(size_t)(i - 1) * E + e]), __dmul_rn(t, U[(size_t)i * E + e]));
    };
    auto r7 = [&](int e, double* five) {  // R7 (and R5) at energy e
        double v7 = 0., v5 = 0.;
#pragma unroll
        for (int p = 0; p < 17; ++p) {
            const double fv = value(p, e);
            v7 = __dadd_rn(v7, __dmul_rn(c_gm64.w7[p], fv));
            v5 = __dadd_rn(v5, __dmul_rn(c_gm64.w5[p], fv));
        }
        *five = v5;
        return v7;
    };
    double rel = 0., first = 0., second = 0.;  // R7 of the lane's first two energies
    for (int e = lane; e < min(E, last ? 64 : E); e += 32) {
        double v5;
        const double v7 = r7(e, &v5);
        if (e < 32) first = v7;
        else if (e < 64) second = v7;
        const double err = fabs(__dsub_rn(v5, v7));
        const double r = v7 != 0. ? err / fabs(v7) : (err != 0. ? INFINITY : 0.);
        rel = r > rel ? r : rel;
    }
    if (!last) {
        for (int o = 16; o > 0; o >>= 1) rel = fmax(rel, __shfl_xor_sync(0xffffffffu, rel, o));
    }
    const bool accept = last || rel <= (double)A.rtol;
    if (!accept) {
        double dd0 = 0., dd1 = 0.;
        for (int e0 = 0; e0 < E; e0 += 32) {
            const int e = e0 + lane;
            double g0 = 0., g1 = 0.;
            if (e < E) {
                double f[9];
#pragma unroll
                for (int p = 0; p < 9; ++p) f[p] = value(p, e);
                const double f0 = __dmul_rn(2., f[0]);
                g0 = fabs(__dsub_rn(__dsub_rn(__dadd_rn(f[1], f[3]), f0),
                                    __dmul_rn(1. / 7., __dsub_rn(__dadd_rn(f[5], f[7]), f0))));
                g1 = fabs(__dsub_rn(__dsub_rn(__dadd_rn(f[2], f[4]), f0),
                                    __dmul_rn(1. / 7., __dsub_rn(__dadd_rn(f[6], f[8]), f0))));
            }
            const int n = min(32, E - e0);
            for (int k = 0; k < n; ++k) {
                dd0 = __dadd_rn(dd0, shfl_d(g0, k));
                dd1 = __dadd_rn(dd1, shfl_d(g1, k));
            }
        }
        *dim = dd0 >= dd1 ? 0 : 1;
    }
    const double area = __dmul_rn(R.h0, R.h1);
    for (int e = lane; e < E; e += 32) {
        double v = 0., v5;
        if (accept) v = __dmul_rn(area, e < 32 ? first : e < 64 ? second : r7(e, &v5));
        if (level0) mean[e] = v;
        else if (accept) atomicAdd(mean + e, v);
    }
    return accept;
}

// The two halves of a region (lower half first) at q[k], q[k + 1].
__device__ __forceinline__ void store_halves(QRegion* q, int k, const LaneRegion& R, int dim) {
    QRegion a{R.sp, R.c0, R.c1, R.h0, R.h1}, b = a;
    if (dim == 0) {
        a.h0 = b.h0 = 0.5f * R.h0;
        a.c0 = R.c0 - 0.5f * R.h0;
        b.c0 = R.c0 + 0.5f * R.h0;
    } else {
        a.h1 = b.h1 = 0.5f * R.h1;
        a.c1 = R.c1 - 0.5f * R.h1;
        b.c1 = R.c1 + 0.5f * R.h1;
    }
    q[k] = a;
    q[k + 1] = b;
}

// One region decided in FP64, its halves queued (or its value kept when the queue is full).
__device__ __noinline__ void gm_fp64(const LevelArgs& A, const LaneRegion& R, Point64* pts, bool last, bool level0,
                                     QRegion* qout, int* qcount, int qcap) {
    int dim = 0, k = 0;
    if (gm_region64(A, R, pts, last, level0, &dim)) return;
    if ((threadIdx.x & 31) == 0) k = atomicAdd(qcount, 2);
    k = __shfl_sync(0xffffffffu, k, 0);
    if (k + 2 > qcap) gm_region64(A, R, pts, true, level0, &dim);
    else if ((threadIdx.x & 31) == 0) store_halves(qout, k, R, dim);
}

struct Queue64 { QRegion* q; int* count; int cap; };

__device__ __forceinline__ LaneRegion lane_region(const QRegion& r, int npix, int W) {
    LaneRegion R;
    R.sp = r.sp; R.c0 = r.c0; R.c1 = r.c1; R.h0 = r.h0; R.h1 = r.h1;
    R.s = r.sp / npix;
    const int pix = r.sp - R.s * npix;
    R.h = pix / W;
    R.w = pix - R.h * W;
    return R;
}

enum { GM_ACCEPT = 0, GM_SPLIT0 = 1, GM_SPLIT1 = 2, GM_FP64 = 3, GM_NONE = 4 };

// The windowed regions of `mask` (lane = region): G lanes per region, lane q of the
// group the energies q, q + G, ... (table rows and means are read and written in runs
// of G consecutive values).  Returns each lane's decision for its own region; accepted
// regions' values are added to (at level 0 stored in) their means, and at level 0 the
// means of the others are cleared.
template <int G>
__device__ __forceinline__ int gm_decide(const LevelArgs& A, const LaneRegion& R, const float4* win, int rmin, int nr,
                                         unsigned mask, bool last, bool level0) {
    constexpr int NS = 8;  // energies per lane: E <= G * NS
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, q = lane & (G - 1), E = A.E;
    int mine = GM_NONE;
    for (int r0 = 0; r0 < 32; r0 += 32 / G) {
        if (!((mask >> r0) & ((1u << (32 / G)) - 1))) continue;  // warp-uniform
        const int rg = r0 + lane / G;
        const bool on = (mask >> rg) & 1;
        const int row = __shfl_sync(full, rmin, rg), nrow = __shfl_sync(full, nr, rg);
        const int n = on ? nrow : 0;
        const int sp = __shfl_sync(full, R.sp, rg), s = __shfl_sync(full, R.s, rg);
        const float area = __shfl_sync(full, R.h0, rg) * __shfl_sync(full, R.h1, rg);
        const float* y0 = A.lut + ((size_t)s * ND + row) * A.EP + q;
        const float4* wr = win + rg * WSTRIDE;
        float v7[NS], vd[NS];
#pragma unroll
        for (int c = 0; c < NS; ++c) v7[c] = vd[c] = 0.f;
        // two rows at a time, so that their loads are in flight together
        auto dot = [&](const float2* w, float* u, float* v) {
            const float* y = y0;
            for (int j = 0; j < n; j += 2, y += 2 * A.EP) {
                const bool two = j + 1 < n;
                const float2 wa = w[2 * j], wb = two ? w[2 * j + 2] : make_float2(0.f, 0.f);
                const float* yb = y + A.EP;  // (past the last row: not read, as 0 x inf is no 0)
                float fa[NS], fb[NS];
#pragma unroll
                for (int c = 0; c < NS; ++c)
                    if (G * c < E) {  // uniform
                        const bool in = q + G * c < E;
                        fa[c] = in ? __ldg(y + G * c) : 0.f;
                        fb[c] = in && two ? __ldg(yb + G * c) : 0.f;
                    }
#pragma unroll
                for (int c = 0; c < NS; ++c)
                    if (G * c < E) {
                        u[c] = fmaf(wb.x, fb[c], fmaf(wa.x, fa[c], u[c]));
                        v[c] = fmaf(wb.y, fb[c], fmaf(wa.y, fa[c], v[c]));
                    }
            }
        };
        dot((const float2*)wr, v7, vd);
        int code = GM_ACCEPT;
        if (!last) {
            float rel = 0.f;
#pragma unroll
            for (int c = 0; c < NS; ++c)
                if (G * c < E) {
                    const float x7 = fabsf(v7[c]), xd = fabsf(vd[c]);
                    // 0 / 0 (an all-zero energy, or a lane past E) counts as no error
                    rel = fmaxf(rel, xd == 0.f ? 0.f : (x7 != 0.f ? __fdividef(xd, x7) : 3.4e38f));
                }
#pragma unroll
            for (int o = G / 2; o > 0; o >>= 1) rel = fmaxf(rel, __shfl_xor_sync(full, rel, o));
            const bool accept = rel <= A.rtol;
            if (fabsf(rel - A.rtol) <= fmaxf(0.05f * A.rtol, 4e-6f)) code = GM_FP64;
            if (__any_sync(full, !accept && code != GM_FP64)) {  // the fourth differences of regions to be split
                float a0[NS], a1[NS];
#pragma unroll
                for (int c = 0; c < NS; ++c) a0[c] = a1[c] = 0.f;
                if (!accept) dot((const float2*)wr + 1, a0, a1);
                float dd0 = 0.f, dd1 = 0.f, sx = 0.f;
#pragma unroll
                for (int c = 0; c < NS; ++c)
                    if (G * c < E) {
                        dd0 += fabsf(a0[c]);
                        dd1 += fabsf(a1[c]);
                        sx += fabsf(v7[c]);
                    }
#pragma unroll
                for (int o = G / 2; o > 0; o >>= 1) {
                    dd0 += __shfl_xor_sync(full, dd0, o);
                    dd1 += __shfl_xor_sync(full, dd1, o);
                    sx += __shfl_xor_sync(full, sx, o);
                }
                // the fourth differences cancel most of the values they are formed from, so
                // their FP32 error is measured against the values (sx), not against themselves
                const bool near_dim = fabsf(dd0 - dd1) <= 1e-3f * (dd0 + dd1) + 4e-6f * sx;
                if (!accept && code != GM_FP64) code = near_dim ? GM_FP64 : dd0 >= dd1 ? GM_SPLIT0 : GM_SPLIT1;
            }
        }
        if (on && (code == GM_ACCEPT || (level0 && code != GM_FP64))) {
            double* m = A.mean + (size_t)sp * E + q;
#pragma unroll
            for (int c = 0; c < NS; ++c)
                if (q + G * c < E) {
                    const double v = code == GM_ACCEPT ? (double)(area * v7[c]) : 0.;
                    if (level0) m[G * c] = v;
                    else atomicAdd(m + G * c, v);
                }
        }
        const int got = __shfl_sync(full, code, ((lane - r0) & (32 / G - 1)) * G);
        if (lane >= r0 && lane < r0 + 32 / G && ((mask >> lane) & 1)) mine = got;
    }
    return mine;
}

// One batch of up to 32 regions (lane = region, `on` marks the lanes that hold one).
template <int G>
__device__ __forceinline__ void gm_batch(const LevelArgs& A, const LaneRegion& R, bool on, const double* sq,
                                         const float4* scoef, float4* win, Point64* pts, bool last, bool level0,
                                         QRegion* qout, int* qcount, int qcap, const Queue64& q64) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    int rmin = 0, nr = 0;
    if (on) {
        const PixGeom g = pixel_geom(A.corners, A.W + 1, R.h, R.w, A.info[R.s]);
        int ix[17];
        float tt[17];
        int rmax = 0;
        rmin = ND;
#pragma unroll
        for (int p = 0; p < 17; ++p) {
            const double u = R.c1 + c_gm.off1[p] * R.h1;  // along w
            const double v = R.c0 + c_gm.off0[p] * R.h0;  // along h
            const double x = fma(g.Dx, u * v, fma(g.Cx, v, fma(g.Bx, u, g.Ax)));
            const double y = fma(g.Dy, u * v, fma(g.Cy, v, fma(g.By, u, g.Ay)));
            const double z = fma(g.Dz, u * v, fma(g.Cz, v, fma(g.Bz, u, g.Az)));
            ix[p] = point_row(fma(x, x, fma(y, y, z * z)), sq, scoef, &tt[p]);
            rmin = min(rmin, ix[p] - 1);
            rmax = max(rmax, ix[p]);
        }
        nr = rmax - rmin + 1;
        if (nr <= AW) {  // the region's row windows
            float4* wr = win + lane * WSTRIDE;
            for (int j = 0; j < nr; ++j) wr[j] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int p = 0; p < 17; ++p) {
                const float b = tt[p], a = 1.f - b;
                float4* wj = wr + (ix[p] - 1 - rmin);
                float4 lo = wj[0], hi = wj[1];
                lo.x += a * c_gm.w7[p]; lo.y += a * c_gm.wd[p]; lo.z += a * c_gm.d0[p]; lo.w += a * c_gm.d1[p];
                hi.x += b * c_gm.w7[p]; hi.y += b * c_gm.wd[p]; hi.z += b * c_gm.d0[p]; hi.w += b * c_gm.d1[p];
                wj[0] = lo;
                wj[1] = hi;
            }
        }
    }
    __syncwarp();
    const unsigned narrow = __ballot_sync(full, on && nr <= AW);
    int code = GM_NONE;
    for (unsigned mask = narrow; mask;) {
        const int c = gm_decide<G>(A, R, win, rmin, nr, mask, last, level0);
        if ((mask >> lane) & 1) code = c;
        mask = 0;
        // the halves of the split regions: one reservation per warp
        const unsigned split = __ballot_sync(full, code == GM_SPLIT0 || code == GM_SPLIT1);
        if (split) {
            int k = 0;
            if (lane == 0) k = atomicAdd(qcount, 2 * __popc(split));
            k = __shfl_sync(full, k, 0) + 2 * __popc(split & ((1u << lane) - 1));
            const bool is = (split >> lane) & 1, fits = is && k + 2 <= qcap;
            if (fits) store_halves(qout, k, R, code == GM_SPLIT0 ? 0 : 1);
            mask = __ballot_sync(full, is && !fits);  // queue full: keep their estimates
            last = true;
            if (is) code = GM_NONE;
        }
    }
    if (on && nr > AW) code = GM_FP64;  // points too far apart for a window (next to the source)
    // regions for FP64: queued for the level's second phase, one region per warp there
    const unsigned near = __ballot_sync(full, code == GM_FP64);
    if (near) {
        int k = 0;
        if (lane == 0) k = atomicAdd(q64.count, __popc(near));
        k = __shfl_sync(full, k, 0) + __popc(near & ((1u << lane) - 1));
        const bool fits = code == GM_FP64 && k < q64.cap;
        if (fits) q64.q[k] = QRegion{R.sp, R.c0, R.c1, R.h0, R.h1};
        unsigned over = __ballot_sync(full, code == GM_FP64 && !fits);
        while (over) {  // that queue full: here
            const int l = __ffs(over) - 1;
            over &= over - 1;
            LaneRegion Q;
            Q.sp = __shfl_sync(full, R.sp, l); Q.s = __shfl_sync(full, R.s, l);
            Q.h = __shfl_sync(full, R.h, l); Q.w = __shfl_sync(full, R.w, l);
            Q.c0 = __shfl_sync(full, R.c0, l); Q.c1 = __shfl_sync(full, R.c1, l);
            Q.h0 = __shfl_sync(full, R.h0, l); Q.h1 = __shfl_sync(full, R.h1, l);
            gm_fp64(A, Q, pts, last, level0, qout, qcount, qcap);
        }
    }
    __syncwarp();  // the windows are reused by the next batch
}

__device__ __forceinline__ void load_tables(const SepTab* septab, double* sq, float4* scoef) {
    for (int k = threadIdx.x; k < ND + 1; k += blockDim.x) sq[k] = septab->q[k];
    for (int k = threadIdx.x; k < 2 * ND; k += blockDim.x) scoef[k] = ((const float4*)septab->coef)[k];
    __syncthreads();
}

// Grid-wide barrier of a cooperative launch: the last block to arrive resets the
// count and advances the generation; the others poll it with a bounded wait.
// Returns false (in every thread of the block) when the wait ran out.
constexpr int GRID_WAIT_LIMIT = 1 << 24;  // polls of ~100 ns: about a second or more

__device__ __forceinline__ bool grid_barrier(unsigned* bar, unsigned nblocks, unsigned* gen) {
    __syncthreads();
    bool ok = true;
    if (threadIdx.x == 0) {
        const unsigned g = *gen;
        __threadfence();
        const unsigned arrived = atomicAdd(&bar[0], 1u) + 1u;
        if (arrived == nblocks) {
            atomicExch(&bar[0], 0u);
            __threadfence();
            atomicAdd(&bar[1], 1u);
        } else {
            int it = 0;
            while (atomicAdd(&bar[1], 0u) == g && ++it < GRID_WAIT_LIMIT) __nanosleep(100);
            ok = it < GRID_WAIT_LIMIT;
        }
        __threadfence();
        *gen = g + 1u;
    }
    return __syncthreads_and(ok);
}

// All levels in one persistent launch (cooperative: every block resident).  Level
// 0: item k = (source, pixel) k, the whole pixel as one region; level L >= 1: item k
// = region k of level L - 1's queue.  Levels are separated by grid barriers.
//
// A warp takes 32 items: geometry and row windows with one region per lane, then the
// energies of 32 / G regions at a time with G lanes per region (G = 8 for E <= 64,
// else 32), so table rows and FP64 means move in runs of consecutive values.  Level 0
// takes pixels in TH x TW patches, whose points share table rows (1.03 -> 0.69 ms against
// runs of 32 pixels, L1 misses on the rows).  Regions that need FP64 are queued and
// follow the level's others, one per warp: inside the batches, whose neighbours tend to
// need it together, they held the level's end up (2.0 of 4.9 ms, 0.5 now).  50 sources,
// 200 x 200, 37 energies, rtol 1e-4, depth 6 (4.1 M regions, 0.1 M in FP64): 2.45 ms,
// 26.1 with one region per thread throughout.  What is left: table rows from L2 below
// level 0 (a queue's neighbours are of different patches), the levels' last batches, and
// the FP64 pipe.  Two blocks of 128 registers per SM: 2.52 ms, three of 80: 2.91.
template <int G>
__global__ void __launch_bounds__(AT, ADAPT_BLOCKS)
k_adaptive_levels(LevelArgs A, const SepTab* __restrict__ septab, int S, int max_depth, QRegion* __restrict__ q,
                  long long qcap, int cap64, int* __restrict__ counts, int* __restrict__ work,
                  int* __restrict__ count64, unsigned* __restrict__ bar,
                  int* __restrict__ status) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ unsigned gen_s;
    double* sq = (double*)(smem + AO_SQ);
    float4* scoef = (float4*)(smem + AO_COEF);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float4* win = (float4*)(smem + AO_WIN) + warp * 32 * WSTRIDE;
    Point64* pts = (Point64*)(smem + AO_P64) + warp * 17;
    if (threadIdx.x == 0) gen_s = atomicAdd(&bar[1], 0u);
    load_tables(septab, sq, scoef);
    const int npix = A.H * A.W, pw = (A.W + TW - 1) / TW, per_src = pw * ((A.H + TH - 1) / TH);
    for (int level = 0; level <= max_depth; ++level) {
        const bool last = level >= max_depth, level0 = level == 0;
        QRegion* qout = q + (size_t)(level & 1) * qcap;
        const QRegion* qin = q + (size_t)((level - 1) & 1) * qcap;
        const int n = level0 ? 0 : (int)min((long long)counts[level - 1], qcap);
        const long long nb = level0 ? (long long)S * per_src : (n + 31) / 32;
        const Queue64 q64{q + 2 * (size_t)qcap, count64 + level, cap64};
        // batches from the level's counter, the next one taken ahead: batches next to
        // sources cost several times the others
        int nxt = 0;
        if (lane == 0) nxt = atomicAdd(work + level, 1);
        for (;;) {
            const int item = __shfl_sync(0xffffffffu, nxt, 0);
            if (item >= nb) break;
            if (lane == 0) nxt = atomicAdd(work + level, 1);
            QRegion r{0, 0.f, 0.f, 1.f, 1.f};
            bool on;
            if (level0) {  // a TH x TW patch of pixels, whose points share table rows
                const int s = item / per_src, p = item - s * per_src, ph = p / pw;
                const int h = ph * TH + lane / TW, w = (p - ph * pw) * TW + lane % TW;
                on = h < A.H && w < A.W;
                if (on) r.sp = s * npix + h * A.W + w;
            } else {
                on = item * 32 + lane < n;
                if (on) r = qin[item * 32 + lane];
            }
            gm_batch<G>(A, lane_region(r, npix, A.W), on, sq, scoef, win, pts, last, level0, qout, counts + level,
                        (int)qcap, q64);
        }
        // the level's regions for FP64, spread over all warps
        if (!grid_barrier(bar, gridDim.x, &gen_s)) {
            if (threadIdx.x == 0) atomicExch(status, 1);
            return;
        }
        const int n64 = min(*q64.count, q64.cap);
        for (int k = blockIdx.x + gridDim.x * warp; k < n64; k += gridDim.x * NWARP)
            gm_fp64(A, lane_region(q64.q[k], npix, A.W), pts, last, level0, qout, counts + level, (int)qcap);
        if (level == max_depth) break;
        if (!grid_barrier(bar, gridDim.x, &gen_s)) {
            if (threadIdx.x == 0) atomicExch(status, 1);
            return;
        }
    }
}

// The adaptive map from its FP64 means: value = mean * omega * exposure * correction.
__global__ void k_scale_map64(const double* __restrict__ mean, float* __restrict__ out,
                              const double* __restrict__ omega, const double* __restrict__ scale, int npix, int E) {
    __shared__ double sc[256];
    const int s = blockIdx.y;
    for (int e = threadIdx.x; e < E; e += blockDim.x) sc[e] = scale[(size_t)s * E + e];
    __syncthreads();
    const unsigned n = (unsigned)npix * (unsigned)E;
    const double* m = mean + (size_t)s * n;
    float* o = out + (size_t)s * n;
    for (unsigned k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const unsigned pix = k / (unsigned)E;
        o[k] = (float)(m[k] * omega[pix] * sc[k - pix * (unsigned)E]);
    }
}

// c8 + c10 and the solid angle: value = mean * omega * exposure * correction.
// out[s][pix][e] *= omega[pix] (FP64 product rounded to FP32) * scale[s][e]; four
// consecutive values per thread (one 16-byte load and store, one division), the
// source's first values up to a 16-byte boundary and its last ones one by one.
__device__ __forceinline__ float scale_value(float v, const double* omega, const float* sc, unsigned pix,
                                             unsigned e) {
    return (float)((double)v * omega[pix]) * sc[e];
}
__global__ void k_scale_map(float* __restrict__ out, const double* __restrict__ omega,
                            const double* __restrict__ scale, int npix, int E) {
    __shared__ float sc[256];
    const int s = blockIdx.y;
    for (int e = threadIdx.x; e < E; e += blockDim.x) sc[e] = (float)scale[(size_t)s * E + e];
    __syncthreads();
    const unsigned n = (unsigned)npix * (unsigned)E, uE = (unsigned)E;
    float* o = out + (size_t)s * n;
    const unsigned mis = (unsigned)(((uintptr_t)o >> 2) & 3u);  // o is 4-byte aligned
    const unsigned head = min((4u - mis) & 3u, n);
    const unsigned nq = (n - head) >> 2, tail0 = head + 4 * nq;
    const unsigned tid = blockIdx.x * blockDim.x + threadIdx.x, nth = gridDim.x * blockDim.x;
    if (tid < head) o[tid] = scale_value(o[tid], omega, sc, tid / uE, tid % uE);
    if (tid < n - tail0) {
        const unsigned k = tail0 + tid;
        o[k] = scale_value(o[k], omega, sc, k / uE, k % uE);
    }
    float4* o4 = reinterpret_cast<float4*>(o + head);
    for (unsigned q = tid; q < nq; q += nth) {
        const unsigned k = head + 4 * q;
        unsigned pix = k / uE, e = k - pix * uE;
        float4 v = o4[q];
        float* f = reinterpret_cast<float*>(&v);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            f[i] = scale_value(f[i], omega, sc, pix, e);
            if (++e == uE) { e = 0; ++pix; }
        }
        o4[q] = v;
    }
}

bool srcmap_adaptive_supported(int E) { return E >= 1 && E <= 256; }

int launch_adaptive_map(const double* corners, const SrcInfo* info, const double* upsf, int S, int H, int W, int E,
                        double rtol, int max_depth, double* mean64, int* status, cudaStream_t st) {
    int rc = upload_gm(st);
    if (rc) return rc;
    const SepTab* tab = nullptr;
    rc = build_septab(st, &tab);
    if (rc) return rc;
    const int npix = H * W;
    // the mean PSF rows in FP32, [S][401][E]
    const int EP = (E + 3) & ~3;  // table rows padded to whole float4s
    float* lut = (float*)workspace(W_LUT, sizeof(float) * (size_t)S * ND * EP + 16);
    // two region queues (ping-pong) and one for FP64, their counters per level and the grid barrier
    long long cap = 4LL * S * npix;
    cap = cap < (1 << 20) ? (1 << 20) : cap;
    cap = cap > (1 << 26) ? (1 << 26) : cap;
    const int cap64 = 1 << 20;  // regions of one level decided in FP64 (more are decided where they arise)
    QRegion* q = (QRegion*)workspace(W_SPARSE, sizeof(QRegion) * (2 * (size_t)cap + cap64) + 16);
    int* counts = (int*)workspace(W_WMETA, sizeof(int) * 128);
    if (!lut || !q || !counts) return XTS_ERR_OOM;
    unsigned* bar = (unsigned*)(counts + 32);
    int* work = counts + 40;     // batches taken per level
    int* count64 = counts + 64;  // regions for FP64 per level
    XTS_LAUNCH("k_lut_scaled", st, k_lut_scaled<<<lut_scaled_grid(S), 256, 0, st>>>(upsf, nullptr, S, E, EP, lut,
                                                                                       nullptr, nullptr));
    typedef void (*LevelsFn)(LevelArgs, const SepTab*, int, int, QRegion*, long long, int, int*, int*, int*,
                             unsigned*, int*);
    const LevelsFn levels = E <= 64 ? k_adaptive_levels<8> : k_adaptive_levels<32>;
    XTS_CUDA(cudaFuncSetAttribute(levels, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)A_SMEM));
    XTS_CUDA(cudaMemsetAsync(counts, 0, sizeof(int) * 128, st));
    int dev = 0, nsm = 148, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    XTS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, levels, AT, A_SMEM));
    const unsigned G = (unsigned)(nsm * (per_sm > 0 ? per_sm : 1));
    // one cooperative launch: every block resident, so the grid barriers between levels complete
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(G);
    cfg.blockDim = dim3(AT);
    cfg.dynamicSmemBytes = A_SMEM;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const LevelArgs la{corners, info, lut, upsf, H, W, E, EP, (float)rtol, mean64};
    cudaError_t le = cudaSuccess;
    XTS_LAUNCH("k_adaptive_map", st, le = cudaLaunchKernelEx(&cfg, levels, la, tab, S, max_depth, q, cap, cap64, counts,
                                                             work, count64, bar, status));
    if (le != cudaSuccess) return cuda_error(le, "cooperative launch of k_adaptive_levels");
    return XTS_OK;
}

// The map integral of FP32 pixel means: block (c, s) takes pixels
// [c npix / nc, (c + 1) npix / nc) of source s; warp w of the block the runs of 32
// pixels w, w + 8, ... of that range.  Per run each lane tests one pixel against the
// source's boundary; then, for the inside pixels in order, lane l adds energies l,
// l + 32, ... (a pixel's E means are contiguous, so the loads coalesce).  Per block the
// warps' partial sums are added in a fixed order into sums[s][c][e].
constexpr int MI_WARPS = 8;
constexpr int MI_EQ = 8;  // energies per lane: E <= 256
template <typename T>
__global__ void __launch_bounds__(32 * MI_WARPS) k_mean_integral(const double* __restrict__ centers,
                                                                 const double* __restrict__ omega,
                                                                 const SrcInfo* __restrict__ info,
                                                                 const T* __restrict__ mean, int H, int W, int E,
                                                                 int nc, double* __restrict__ sums_out) {
    __shared__ double part[MI_WARPS][AT];
    const int s = blockIdx.y, t = threadIdx.x, lane = t & 31, wp = t >> 5;
    const SrcInfo si = info[s];
    const int npix = H * W, W1 = W + 1;
    double ch2 = 2.0 * sin(0.5 * si.radius_rad);
    ch2 *= ch2;
    const int p_lo = (int)((long long)npix * blockIdx.x / nc), p_hi = (int)((long long)npix * (blockIdx.x + 1) / nc);
    const int nq = (E + 31) >> 5;
    double acc[MI_EQ];
#pragma unroll
    for (int q = 0; q < MI_EQ; ++q) acc[q] = 0.;
    if (si.in_fov) {
        const T* m = mean + (size_t)s * npix * E;
        // 32 pixels per round: each lane tests its own pixel against the boundary, then
        // the warp sums the inside pixels' rows (lane = energy), two rows per step so
        // that two loads are in flight
        for (int pix0 = p_lo + 32 * wp; pix0 < p_hi; pix0 += 32 * MI_WARPS) {
            const int pix = pix0 + lane;
            bool inside = false;
            double om = 0.;
            if (pix < p_hi) {
                const int h = pix / W, w = pix - h * W;
                const double* c = centers + 3 * (h * W1 + w);
                const double x = si.dir[0] - c[0], y = si.dir[1] - c[1], z = si.dir[2] - c[2];
                const double d2 = x * x + y * y + z * z;
                if (d2 < ch2 * (1.0 - 1e-12)) inside = true;
                else if (d2 > ch2 * (1.0 + 1e-12)) inside = false;
                else inside = dir_diff(si.dir, c) <= si.radius_rad;
                if (inside) om = omega[pix];
            }
            unsigned mask = __ballot_sync(0xffffffffu, inside);
            while (mask) {
                const int l1 = __ffs(mask) - 1;
                mask &= mask - 1;
                const int l2 = mask ? __ffs(mask) - 1 : -1;
                if (l2 >= 0) mask &= mask - 1;
                const double om1 = __shfl_sync(0xffffffffu, om, l1);
                const double om2 = __shfl_sync(0xffffffffu, om, l2 < 0 ? l1 : l2);
                const T* mp1 = m + (size_t)(pix0 + l1) * E;
                const T* mp2 = m + (size_t)(pix0 + (l2 < 0 ? l1 : l2)) * E;
                T v1[MI_EQ], v2[MI_EQ];
#pragma unroll
                for (int q = 0; q < MI_EQ; ++q) {
                    const int e = lane + 32 * q;
                    const bool on = q < nq && e < E;
                    v1[q] = on ? mp1[e] : (T)0;
                    v2[q] = on && l2 >= 0 ? mp2[e] : (T)0;
                }
#pragma unroll
                for (int q = 0; q < MI_EQ; ++q) {
                    acc[q] += (double)v1[q] * om1;
                    if (l2 >= 0) acc[q] += (double)v2[q] * om2;
                }
            }
        }
    }
#pragma unroll
    for (int q = 0; q < MI_EQ; ++q) {
        const int e = lane + 32 * q;
        if (q < nq && e < E) part[wp][e] = acc[q];
    }
    __syncthreads();
    for (int e = t; e < E; e += 32 * MI_WARPS) {
        double v = 0.;
        for (int k = 0; k < MI_WARPS; ++k) v += part[k][e];
        sums_out[((size_t)s * nc + blockIdx.x) * E + e] = v;
    }
}

// Chunks of the FP32 mean-map integral per source: enough blocks for every SM.
int mean_integral_chunks(int S, int npix) {
    int nc = (2400 + (S > 0 ? S : 1) - 1) / (S > 0 ? S : 1);
    const int mx = (npix + 255) / 256;
    return nc < 1 ? 1 : (nc > mx ? mx : nc);
}

int launch_mean_integral(const double* centers, const double* omega, const SrcInfo* info, const float* mean, int S,
                         int H, int W, int E, int nch, double* sums, cudaStream_t st) {
    if (E < 1 || E > AT) return set_error(XTS_ERR_ARG, "map integral of pixel means: E (%d) above %d", E, AT);
    XTS_LAUNCH("k_mean_integral", st, k_mean_integral<float><<<dim3(nch, S), 32 * MI_WARPS, 0, st>>>(
                                          centers, omega, info, mean, H, W, E, nch, sums));
    return XTS_OK;
}

int launch_mean_integral64(const double* centers, const double* omega, const SrcInfo* info, const double* mean, int S,
                           int H, int W, int E, int nch, double* sums, cudaStream_t st) {
    if (E < 1 || E > AT) return set_error(XTS_ERR_ARG, "map integral of pixel means: E (%d) above %d", E, AT);
    XTS_LAUNCH("k_mean_integral", st, k_mean_integral<double><<<dim3(nch, S), 32 * MI_WARPS, 0, st>>>(
                                              centers, omega, info, mean, H, W, E, nch, sums));
    return XTS_OK;
}

int launch_scale_map64(const double* mean, float* out, const double* omega, const double* scale, int S, int npix,
                       int E, cudaStream_t st) {
    const unsigned n = (unsigned)npix * (unsigned)E;
    unsigned gx = (n + 255) / 256;
    if (gx > 1024) gx = 1024;
    XTS_LAUNCH("k_scale_map", st, k_scale_map64<<<dim3(gx, S), 256, 0, st>>>(mean, out, omega, scale, npix, E));
    return XTS_OK;
}

int launch_scale_map(float* out, const double* omega, const double* scale, int S, int npix, int E,
                     cudaStream_t st) {
    const unsigned n = (unsigned)npix * (unsigned)E;
    unsigned gx = (n + 255) / 256;
    if (gx > 1024) gx = 1024;
    XTS_LAUNCH("k_scale_map", st, k_scale_map<<<dim3(gx, S), 256, 0, st>>>(out, omega, scale, npix, E));
    return XTS_OK;
}

}  // namespace xts
