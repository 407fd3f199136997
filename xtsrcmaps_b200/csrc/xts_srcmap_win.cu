// xts_srcmap_win.cu -- the FP32 source-map path in two passes over the pixels.
//
// Pass A, k_pixel_windows (geometry, once per pixel and source): the 12 rule
// points of the pixel give LUT rows and interpolation weights (xts_point.cuh);
// their weights times the pixel's solid angle are summed into a dense window of
// at most RW consecutive table rows.  For pixels inside the boundary radius of
// an in-FOV source the window also enters the block's FP64 row histogram, whose
// dot product with uPsf is the map integral of c7 (model_map.map_integral.cxx:4-48):
//     sum_pix omega * value(pix, e) = sum_r Hist[r] * uPsf[r][e].
// The rule points' squared chords are FP32 offsets from the pixel centre's FP64
// squared chord (the biquadratic form of xts_point.cuh), six mirror pairs as packed
// FP32 operations: one FP64 table search per pixel, none per point.  A work item is a
// group of up to eight sources and a part of the map; a pixel's own geometry is formed
// once for the group.  The histogram takes each window row of a
// pixel inside the radius by one FP64 shared-memory atomic add.  Every pixel's
// window is written once as a 16-byte record (3 FP32 weights and the first row /
// row count), with the 8 weights of a window longer than 3 rows in a 32-byte
// extension.  Pixels whose points leave the 8-row window (those next to the
// source) are "wide": their points are redone in FP64, a thread per point, into a
// sparse record of their 24 (row, weight) pairs from a shared pool, or, if the pool
// is full, again point by point in pass B.
//
// Pass B, k_srcmap_win (the write pass, d1 + d2 + c8 + c10): the source's scaled
// table Y' = uPsf * exposure * correction (FP32, [401][EQ] float4, EQ odd so
// different rows fall in different shared-memory bank groups) is brought into
// shared memory by one TMA bulk copy; each thread reads the window records of two
// pixels of neighbouring rows and forms value[e] = sum_j W[j] * Y'[row_j][e] of both from
// one load of each table row (rows rbase + j, or the 24 rows of a sparse record).  Values
// are staged and written by TMA bulk stores, so the pass streams the
// window records in and the map out; the next tile's records are loaded while
// the current one is computed.
#include <vector>

#include "xts_point.cuh"

namespace xts {

// ============================================================================ pass A
constexpr int WT = 256;     // pixels per tile == threads per block
constexpr int NSG_MAX = 8;  // sources per group: one pixel's source-independent geometry serves the group

// A source as the window pass needs it: the boundary test's limits beside its direction.
struct WinSrc {
    double dir[3], ch2, radius_rad;  // ch2: squared chord of the boundary radius
    int in_fov, pad;
};
__device__ __forceinline__ WinSrc win_source(const SrcInfo& si) {
    WinSrc w;
    w.dir[0] = si.dir[0]; w.dir[1] = si.dir[1]; w.dir[2] = si.dir[2];
    const double c = 2.0 * sin(0.5 * si.radius_rad);
    w.ch2 = c * c;
    w.radius_rad = si.radius_rad;
    w.in_fov = si.in_fov;
    w.pad = 0;
    return w;
}

// Shared memory of the window pass for nsg sources per group.
constexpr size_t WA_OFF_WTS = sizeof(SepTab);  // (the tables first)
constexpr size_t WA_OFF_BAR = WA_OFF_WTS + sizeof(float) * WT * RW;
constexpr size_t WA_OFF_SRC = WA_OFF_BAR + 16;
// Wide pixels put off: map pixel, source of the group | inside << 8, omega's bits, sparse
// record (-1: none).  The dense pass keeps an item's (what does not fit is found again by its
// records, wide_left), the cutouts' pass a warp's of a run.
constexpr int WIDE_CAP = 128;
constexpr size_t WA_OFF_WIDE = WA_OFF_SRC + sizeof(WinSrc) * NSG_MAX;
constexpr size_t WA_OFF_HIST = WA_OFF_WIDE + sizeof(int4) * WIDE_CAP;
static_assert(WA_OFF_WIDE % 16 == 0 && WA_OFF_HIST % 16 == 0, "alignment");
constexpr size_t wa_smem(int nsg) { return WA_OFF_HIST + sizeof(double) * ND * (size_t)nsg; }
constexpr size_t WA_OFF_WARP = (wa_smem(1) + 15) / 16 * 16;  // the cutouts' pass: [WT] wide pixels, 32 per warp
constexpr size_t WA_CUT_SMEM = WA_OFF_WARP + sizeof(int4) * WT;

constexpr int NSP = 24;  // entries of a sparse record: 12 points x 2 rows
constexpr int META_OVERFLOW = -0x7fffffff - 1;  // wide pixel without a sparse record
constexpr int REC_ROWS = 3;  // window rows held by the 16-byte main record
constexpr float EMSTEP = (float)(REDM1 / (REDM1 + 1.0));  // e^-step: t in row k + 1 = (t in row k - 1) e^-step

// Per (source, pixel) the main record rec = {w0, w1, w2, meta}: meta >= 0 is the
// window's first row (bits 0-15) and row count (bits 16-23), with the weights of
// windows longer than REC_ROWS rows in ext (two float4, w0..w7); meta < 0 marks a
// wide pixel (sparse record -1 - meta, or META_OVERFLOW).
struct PassA {
    const SepBin* sbin;    // shared: row bins
    const float4* scoef;   // shared: per-row records
    const double* sq;      // shared: squared chords of the rows
    const float* sd1;      // shared: their steps q[k + 1] - q[k]
    double* hist;          // shared: the block's map-integral rows ([sources of the group][ND])
    float* wts;            // shared: [RW][WT] windows
    float4* rec;
    float4* ext;
    float2* sparse;
    int sparse_cap;
    int* sparse_count;
    int4* wide;            // shared: wide pixels [WIDE_CAP]
};

// Shared tables of pass A: one bulk copy per block, in flight while the caller clears the
// histogram and prepares its sources; tables_ready() (by every thread, after a block
// barrier) waits for it.
__device__ __forceinline__ PassA pass_a_tables(unsigned char* smem, const SepTab* septab, float4* rec, float4* ext,
                                               float2* sparse, int sparse_cap, int* sparse_count) {
    PassA A;
    const SepTab* tab = (const SepTab*)smem;
    A.sbin = tab->bins;
    A.scoef = (const float4*)tab->coef;
    A.sq = tab->q;
    A.sd1 = tab->d1;
    A.hist = (double*)(smem + WA_OFF_HIST);
    A.wts = (float*)(smem + WA_OFF_WTS);
    A.rec = rec; A.ext = ext; A.sparse = sparse; A.sparse_cap = sparse_cap; A.sparse_count = sparse_count;
    A.wide = (int4*)(smem + WA_OFF_WIDE);
    if (threadIdx.x == 0) {
        const unsigned bar = smem_u32(smem + WA_OFF_BAR);
        mbar_init(bar, 1);
        bulk_load(smem, septab, (unsigned)sizeof(SepTab), bar);
    }
    return A;
}
// False (in every thread) when the bounded wait ran out: the block sets *status and returns.
__device__ __forceinline__ bool tables_ready(unsigned char* smem, int* status) {
    const bool ok = mbar_wait(smem_u32(smem + WA_OFF_BAR), 0);
    if (__syncthreads_and(ok)) return true;
    if (threadIdx.x == 0) {
        atomicExch(status, 1);
        mbar_wait(smem_u32(smem + WA_OFF_BAR), 0);  // bounded: let the copy land before the block exits
    }
    return false;
}

// Source-independent geometry of one pixel: its rule points are the bilinear
// blend P(u, v) = M + B u + C v + D uv of the corners, so relative to a source s
// with A = M - s the squared chord is q(u, v) = |A + B u + C v + D uv|^2, whose
// coefficients split into source-dependent ones (|A|^2, 2 A.B, 2 A.C, 2 A.D) and
// the rest (|B|^2, |C|^2, 2 B.C, 2 B.D, 2 C.D, |D|^2; FP64 products rounded once).  The
// latter enter each mirror pair's chord offset through eb (even part) and ob (odd part),
// formed once per pixel for a group of sources.  Mirror pairs k and k + 3 have the same weight (the rule's points are
// three orbits of quarter turns) and go through packed FP32 FMAs together: x holds pair k,
// y pair k + 3.
struct PixBase {
    double m[3];      // M, the corners' average (FP64)
    float b2[3], c2[3], d2[3];  // 2B, 2C, 2D
    float bc2;        // 2 B.C
    float2 eb[3], ob[3];
    float om;         // solid angle
    float off;        // bound on |chord of M - chord of the pixel's centre| per chord: 4.2 |M - centre|
};

__device__ __forceinline__ float2 pair_c(int k, int j) { return make_float2(c_pair[k][j], c_pair[k + 3][j]); }

__device__ __forceinline__ PixBase pixel_base(const double* __restrict__ corners, const double* __restrict__ centers,
                                              const double* __restrict__ omega, int W1, int h, int w, size_t om_idx) {
    const double* a = corners + 3 * (h * W1 + w);            // LL
    const double* b = corners + 3 * (h * W1 + w + 1);        // LR
    const double* c = corners + 3 * ((h + 1) * W1 + w + 1);  // UR
    const double* d = corners + 3 * ((h + 1) * W1 + w);      // UL
    const double* pc = centers + 3 * ((size_t)h * W1 + w);
    PixBase P;
    double bb = 0., cc = 0., bd2 = 0., cd2 = 0., dd = 0., bc = 0.;
    float mc = 0.f;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const double ac = a[i] + c[i], bd = b[i] + d[i], bad = b[i] - d[i], ca = c[i] - a[i];
        P.m[i] = 0.25 * (ac + bd);
        const double B2 = 0.5 * (ca + bad), C2 = 0.5 * (ca - bad), D2 = 0.5 * (ac - bd);
        P.b2[i] = (float)B2;
        P.c2[i] = (float)C2;
        P.d2[i] = (float)D2;
        bb = fma(B2, B2, bb);
        cc = fma(C2, C2, cc);
        bd2 = fma(B2, D2, bd2);
        cd2 = fma(C2, D2, cd2);
        dd = fma(D2, D2, dd);
        bc = fma(B2, C2, bc);
        const float x = (float)(P.m[i] - pc[i]);
        mc = fmaf(x, x, mc);
    }
    // |B|^2, |C|^2, 2 B.D, 2 C.D, |D|^2 and 2 B.C from the doubled vectors
    const float q4 = 0.25f * (float)bb, q5 = 0.25f * (float)cc, q6 = 0.5f * (float)bd2, q7 = 0.5f * (float)cd2;
    const float q8 = 0.25f * (float)dd;
    P.bc2 = 0.5f * (float)bc;
    P.off = fmaf(4.2f, sqrtf(mc), 4e-12f);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        P.eb[k] = __ffma2_rn(make_float2(q8, q8), pair_c(k, 7),
                             __ffma2_rn(make_float2(q5, q5), pair_c(k, 4), __fmul2_rn(make_float2(q4, q4), pair_c(k, 3))));
        P.ob[k] = __ffma2_rn(make_float2(q7, q7), pair_c(k, 6), __fmul2_rn(make_float2(q6, q6), pair_c(k, 5)));
    }
    P.om = omega ? (float)omega[om_idx] : 1.f;  // omega NULL: the pixel means (unit solid angle)
    return P;
}

// Lower table row of the squared chord q: one bin load and one FP64 compare.
__device__ __forceinline__ int row_lower(double q, const SepBin* bins) {
    int b = (__double2hiint(q) >> (20 - SB_BITS)) - (SB_EXP0 << SB_BITS);
    b = min(max(b, 0), NSB - 1);
    const SepBin sb = bins[b];
    return sb.k0 + (q >= sb.thr);
}

// Point p of a wide pixel (next to the source) with FP64 chords from the corners, for its
// sparse record and its map-integral rows alike.
__device__ __forceinline__ void wide_point(const int4& e, int p, const SepBin* sbin, const float4* scoef,
                                           float2* sparse, const double* __restrict__ corners, int W1, double dx,
                                           double dy, double dz, double* hist, int* rlo, int* rhi) {
    const int h = e.x / (W1 - 1);
    SrcInfo sd;
    sd.dir[0] = dx; sd.dir[1] = dy; sd.dir[2] = dz;
    const PixQ g = pixel_q(pixel_geom(corners, W1, h, e.x - h * (W1 - 1), sd));
    float tt;
    const int idx = point_row_bin(point_q2(g, p), sbin, scoef, &tt);
    const float wo = c_rule_w32[p] * __int_as_float(e.z);
    const float wa = (1.f - tt) * wo, wb = tt * wo;
    if (e.w >= 0) {
        float2* sr = sparse + (size_t)e.w * NSP;
        sr[2 * p] = make_float2(wa, __int_as_float(idx - 1));
        sr[2 * p + 1] = make_float2(wb, __int_as_float(idx));
    }
    if (e.y >> 8) {
        atomicAdd(&hist[idx - 1], (double)wa);
        atomicAdd(&hist[idx], (double)wb);
        if (rlo) {
            atomicMin(rlo, idx - 1);
            atomicMax(rhi, idx);
        }
    }
}
// Wide pixels a thread per (point, pixel), neighbouring lanes on different pixels (their
// rows differ, so the histogram's atomics rarely meet).  The pixel's own lane did its
// twelve points one after another before, a run next to a source having a few such lanes.
// The dense pass takes an item's together at its end (50 sources x 200 x 200: 105 -> 82 us,
// 500 x 400 x 400: 1.24 -> 1.22 ms; a warp's at once, source by source: 93 us and 1.35 ms);
// the cutouts' pass, whose items are small and all next to a source, a warp's at once
// (1.00 -> 0.93 ms, 0.94 with the pixels' second-order terms in FP64; at the item's end 1.02).
__device__ __forceinline__ void wide_of_warp(bool wide, const int4& e, const PassA& A,
                                             const double* __restrict__ corners, int W1, const WinSrc& si,
                                             int4* list, int* rlo, int* rhi) {
    const unsigned mask = __ballot_sync(0xffffffffu, wide);
    if (!mask) return;
    const int lane = threadIdx.x & 31, n = __popc(mask);
    if (wide) list[__popc(mask & ((1u << lane) - 1))] = e;
    __syncwarp();
    for (int k = lane; k < 12 * n; k += 32) {
        const int p = k / n;
        wide_point(list[k - p * n], p, A.sbin, A.scoef, A.sparse, corners, W1, si.dir[0], si.dir[1], si.dir[2], A.hist, rlo,
                   rhi);
    }
    __syncwarp();
}
__device__ __forceinline__ void wide_of_item(int n, const PassA& A, const double* __restrict__ corners, int W1,
                                             const WinSrc* src) {
    for (int k = threadIdx.x; k < 12 * n; k += WT) {
        const int p = k / n;
        const int4 e = A.wide[k - p * n];
        const int j = e.y & 0xff;
        wide_point(e, p, A.sbin, A.scoef, A.sparse, corners, W1, src[j].dir[0], src[j].dir[1], src[j].dir[2],
                   A.hist + j * ND, nullptr, nullptr);
    }
}

// The item's wide pixels that found the list full: marked by z = 1 in their records (omega
// and the inside test in x and y).  Kept out of the pass's common path and its registers:
// called there the pass takes 1.28 ms (500 x 400 x 400), inlined there 1.35, inlined here 1.27.
__device__ __noinline__ void wide_left(const PassA A, const double* __restrict__ corners, int W1,
                                          const WinSrc* src, int ns, int s0, int npix, int pa, int pb) {
    for (int j = 0; j < ns; ++j)
        for (int pix = pa + threadIdx.x; pix < pb; pix += WT) {
            float4* rec = A.rec + (size_t)(s0 + j) * npix + pix;
            const float4 r = *rec;
            const int meta = __float_as_int(r.w);
            if (meta >= 0 || r.z == 0.f) continue;
            const int4 e = make_int4(pix, r.y != 0.f ? 256 : 0, __float_as_int(r.x), meta == META_OVERFLOW ? -1 : -1 - meta);
            for (int p = 0; p < 12; ++p)
                wide_point(e, p, A.sbin, A.scoef, A.sparse, corners, W1, src[j].dir[0], src[j].dir[1], src[j].dir[2],
                           A.hist + j * ND, nullptr, nullptr);
            *rec = make_float4(0.f, 0.f, 0.f, r.w);
        }
}

// One (source, pixel): the pixel's window for source si, record index kk.  Pixels
// whose centre lies within the boundary radius (squared chord ch2) add their window
// rows to hist (the source's map-integral rows); the rows they touch widen
// [*rlo, *rhi] when those are given.  (h, w) and W1 locate the pixel's corners for
// the rare wide pixel: on the item's list (CUT: returned with true).
template <bool CUT>
__device__ __forceinline__ bool window_source(const PixBase& P, const WinSrc& si,
                                              const double* __restrict__ corners, const double* __restrict__ centers,
                                              int W1, int h, int w,
                                              size_t kk, const PassA& A, double* hist, int* rlo, int* rhi, int j,
                                              int* nwide, int4* entry) {
    const int t = threadIdx.x;
    const double Ax = P.m[0] - si.dir[0], Ay = P.m[1] - si.dir[1], Az = P.m[2] - si.dir[2];
    const double a0 = fma(Ax, Ax, fma(Ay, Ay, Az * Az));  // q at the centre of the blend
    bool inside = false;
    if (si.in_fov) {
        // |a0 - the centre's squared chord| <= |M - centre| (|A| + chord) <= 4 |M - centre|: the
        // centre's own chord decides only within that of the boundary's
        const float gap = (float)(si.ch2 - a0);
        if (fabsf(gap) > P.off) {
            inside = gap > 0.f;
        } else {
            const double* pc = centers + 3 * ((size_t)h * W1 + w);
            const double x = si.dir[0] - pc[0], y = si.dir[1] - pc[1], z = si.dir[2] - pc[2];
            const double d2 = x * x + y * y + z * z;
            if (d2 < si.ch2 * (1.0 - 1e-12)) inside = true;
            else if (d2 > si.ch2 * (1.0 + 1e-12)) inside = false;
            else inside = dir_diff(si.dir, pc) <= si.radius_rad;
        }
    }
    // q(point) - a0 in FP32: 2 A.B u + 2 A.C v + (2 A.D + 2 B.C) uv + the pixel's part
    const float ax = (float)Ax, ay = (float)Ay, az = (float)Az;
    const float f1 = fmaf(ax, P.b2[0], fmaf(ay, P.b2[1], az * P.b2[2]));
    const float f2 = fmaf(ax, P.c2[0], fmaf(ay, P.c2[1], az * P.c2[2]));
    const float f3 = fmaf(ax, P.d2[0], fmaf(ay, P.d2[1], fmaf(az, P.d2[2], P.bc2)));
    float2 dq2[6];  // pairs (k, k + 3): the points themselves, then their mirror images
    float mn = INFINITY, mx = -INFINITY;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float2 E = __ffma2_rn(make_float2(f3, f3), pair_c(k, 2), P.eb[k]);
        const float2 O = __ffma2_rn(make_float2(f2, f2), pair_c(k, 1),
                                    __ffma2_rn(make_float2(f1, f1), pair_c(k, 0), P.ob[k]));
        dq2[k] = __fadd2_rn(E, O);
        dq2[k + 3] = __ffma2_rn(O, make_float2(-1.f, -1.f), E);
        mn = fminf(mn, fminf(fminf(dq2[k].x, dq2[k].y), fminf(dq2[k + 3].x, dq2[k + 3].y)));
        mx = fmaxf(mx, fmaxf(fmaxf(dq2[k].x, dq2[k].y), fmaxf(dq2[k + 3].x, dq2[k + 3].y)));
    }
    const float om = P.om;
    auto edge = [&](int k) { return (float)(A.sq[k] - a0); };  // q[k] - a0 in FP32
    // Most pixels' points lie in the centre's table row, or in it and one
    // neighbour.  Then one row's polynomial (fitted over two rows) gives every
    // point's t relative to the lower row kl, u = t - 1; a point past the upper
    // edge eb has t' = u e^-step in row kl + 1.  With T = sum w u over all points
    // and S2 = sum w u over those past eb, the three row weights are
    //     s0 = om (S2 - T),  s2 = om e^-step S2,  s1 = om sum(w) - s0 - s2.
    const int kc = row_lower(a0, A.sbin);  // the centre's lower table row
    if (kc >= 2 && kc <= ND - 4) {
        // rows kc (and kc + 1), or kc - 1 and kc; eb = +inf for one row.  The outer edges are
        // bounds from row kc's width: a row is 5.27 (the widest) to 6.98 % wider than the one
        // below it, so a few pixels more than need be go on to the general path.  The inner
        // edges are FP64 differences, rounded.  The case is made opaque to the compiler:
        // specialising the point loop per case would run up to three copies of it per warp,
        // each with a part of the lanes.
        const float w0 = A.sd1[kc], e0 = edge(kc), e1 = edge(kc + 1);
        const bool up = mn >= e0 && mx < fmaf(1.05f, w0, e1), dn = mn >= fmaf(-0.934f, w0, e0) && mx < e1;
        int kl = up ? kc : (dn ? kc - 1 : -1);
        float eb = (mn >= e0 && mx < e1) ? INFINITY : (up ? e1 : e0);
        asm volatile("" : "+r"(kl), "+f"(eb));
        if (kl >= 0) {  // (warp-divergent: a warp's pixels usually agree)
            const float4 c0 = A.scoef[2 * kl], c1 = A.scoef[2 * kl + 1];
            const float eL = (float)(__hiloint2double(__float_as_int(c1.w), __float_as_int(c1.z)) - a0);
            // zz = (dl - C)/H and REDM1 dl, dl = q / q_kl - 1 = (dq - eL) / q_kl, as FMAs in dq
            const float kz = c0.x * (1.f / DPOLY_H), z0 = fmaf(-eL, kz, -DPOLY_C / DPOLY_H);
            const float kr = c0.x * (float)REDM1, r0 = -eL * kr;
            const float2 kz2 = make_float2(kz, kz), z02 = make_float2(z0, z0), kr2 = make_float2(kr, kr);
            const float2 r02 = make_float2(r0, r0), p0 = make_float2(c0.y, c0.y), p1 = make_float2(c0.z, c0.z);
            const float2 p2 = make_float2(c0.w, c0.w), p3 = make_float2(c1.x, c1.x), p4 = make_float2(c1.y, c1.y);
            float2 T2 = make_float2(0.f, 0.f), S22 = T2;
#pragma unroll
            for (int k = 0; k < 6; ++k) {
                const float2 dq = dq2[k];
                const float2 zz = __ffma2_rn(dq, kz2, z02);
                const float2 P4 = __ffma2_rn(__ffma2_rn(__ffma2_rn(__ffma2_rn(p4, zz, p3), zz, p2), zz, p1), zz, p0);
                const float2 u = __ffma2_rn(__ffma2_rn(dq, kr2, r02), P4, make_float2(-1.f, -1.f));
                const float wp = c_rule_w32[k % 3];
                T2 = __ffma2_rn(make_float2(wp, wp), u, T2);
                S22 = __ffma2_rn(make_float2(dq.x >= eb ? wp : 0.f, dq.y >= eb ? wp : 0.f), u, S22);
            }
            const float T = T2.x + T2.y, S2 = S22.x + S22.y;
            const float s0 = om * (S2 - T), s2 = om * (EMSTEP * S2);
            const float s1 = fmaf(om, c_rule_wsum, -s0) - s2;
            const bool two = eb != INFINITY;
            const int nent = two ? 3 : 2;
            if (inside) {
                atomicAdd(&hist[kl], (double)s0);
                atomicAdd(&hist[kl + 1], (double)s1);
                if (two) atomicAdd(&hist[kl + 2], (double)s2);
                if (rlo) {
                    atomicMin(rlo, kl);
                    atomicMax(rhi, kl + nent - 1);
                }
            }
            A.rec[kk] = make_float4(s0, s1, s2, __int_as_float(kl | (nent << 16)));
            return false;
        }
    }
    float dqs[12];  // the rule's points in order: pair k at k, its mirror image at k + 6
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        dqs[k] = dq2[k].x;
        dqs[k + 3] = dq2[k].y;
        dqs[k + 6] = dq2[k + 3].x;
        dqs[k + 9] = dq2[k + 3].y;
    }
    // General path: the window of RW rows around the centre's row, the row edges
    // as FP32 offsets from a0.
    const int base = min(max(kc - RW / 2, 0), ND - RW);
    float d[RW];
#pragma unroll
    for (int j = 0; j < RW; ++j) d[j] = edge(base + j);
    float* wd = A.wts + t;  // slot j at wd[j * WT]: lanes hit consecutive words
#pragma unroll
    for (int j = 0; j < RW; ++j) wd[j * WT] = 0.f;
    bool wide = false;
    int lo = RW, hi = -1;
#pragma unroll
    for (int p = 0; p < 12; ++p) {
        const float dq = dqs[p];
        int r = 0;
        float dlo = d[0];
#pragma unroll
        for (int j = 1; j < RW; ++j) {
            const bool ge = dq >= d[j];
            r += ge;
            dlo = ge ? d[j] : dlo;
        }
        const int k = base + r;  // the point's lower table row
        const float wo = c_rule_w32[p] * om;
        if (dq >= d[0] && r < RW - 1 && k >= 1) {
            const float4 c0 = A.scoef[2 * k], c1 = A.scoef[2 * k + 1];
            const float dl = (dq - dlo) * c0.x;  // q / q_k - 1
            float tt;
            if (dl >= -0.002f && dl <= 0.072f) {
                const float zz = fmaf(dl, 1.f / DPOLY_H, -DPOLY_C / DPOLY_H);
                const float P4 = fmaf(fmaf(fmaf(fmaf(c1.y, zz, c1.x), zz, c0.w), zz, c0.z), zz, c0.y);
                tt = (float)REDM1 * (dl * P4);
            } else {
                tt = t_exact(a0 + (double)dq, k + 1);
            }
            wd[r * WT] += (1.f - tt) * wo;
            wd[(r + 1) * WT] += tt * wo;
            lo = min(lo, r);
            hi = max(hi, r + 1);
        } else {
            wide = true;
        }
    }
    if (!wide) {
        // map integral (c7): the window's rows of a pixel inside the radius
        if (inside) {
#pragma unroll
            for (int j = 0; j < RW; ++j)
                if (j >= lo && j <= hi) atomicAdd(&hist[base + j], (double)wd[j * WT]);
            if (rlo) {
                atomicMin(rlo, base + lo);
                atomicMax(rhi, base + hi);
            }
        }
        const int nent = hi - lo + 1;
        float f[RW];
#pragma unroll
        for (int j = 0; j < RW; ++j) f[j] = j < nent ? wd[min(j + lo, RW - 1) * WT] : 0.f;
        const int meta = (base + lo) | (nent << 16);
        A.rec[kk] = make_float4(f[0], f[1], f[2], __int_as_float(meta));
        if (nent > REC_ROWS) {
            A.ext[2 * kk] = make_float4(f[0], f[1], f[2], f[3]);
            A.ext[2 * kk + 1] = make_float4(f[4], f[5], f[6], f[7]);
        }
    } else {
        int slot = atomicAdd(A.sparse_count, 1);
        if (slot >= A.sparse_cap) slot = -1;
        const float meta = __int_as_float(slot >= 0 ? -1 - slot : META_OVERFLOW);
        const int4 e = make_int4(h * (W1 - 1) + w, j | (inside ? 256 : 0), __float_as_int(om), slot);
        if (CUT) {
            A.rec[kk] = make_float4(0.f, 0.f, 0.f, meta);
            *entry = e;
            return true;
        }
        const int at = atomicAdd(nwide, 1);
        const float full = at >= WIDE_CAP ? 1.f : 0.f;
        if (at < WIDE_CAP) A.wide[at] = e;
        A.rec[kk] = make_float4(full * om, inside ? full : 0.f, full, meta);
    }
    return false;
}

// This lane's pixel of the warp's next run of 32 from pixel p0 on.
__device__ __forceinline__ int next_run(int* counter, int p0) {
    int c = 0;
    if ((threadIdx.x & 31) == 0) c = atomicAdd(counter, 32);
    return p0 + __shfl_sync(0xffffffffu, c, 0) + (threadIdx.x & 31);
}

// The dense map: block b takes item b = (g, p), part p of the P parts of group g (nsg
// sources; tiles [p nt / P, (p + 1) nt / P) of WT pixels), forms each pixel's
// source-independent geometry once and the windows of the group's sources from it,
// and adds the item's non-zero rows to hist_out[s] (cleared before the launch) with
// FP64 atomics.  Items are small (about 8 per resident block), so blocks retire
// steadily: the hardware balances them, and kernels of a higher-priority stream
// (exposure and PSF beside this pass) get their slots as they free up.
__global__ void __launch_bounds__(WT, 3) k_pixel_windows(const double* __restrict__ corners, const double* __restrict__ centers,
                                                      const double* __restrict__ omega, const SrcInfo* __restrict__ info,
                                                      const SepTab* __restrict__ septab, int S, int H, int W,
                                                      int P, int nsg,
                                                      double* __restrict__ hist_out, float4* __restrict__ rec,
                                                      float4* __restrict__ ext, float2* __restrict__ sparse,
                                                      int sparse_cap, int* __restrict__ sparse_count,
                                                      int* __restrict__ status) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int next_s, nwide_s;
    const PassA A = pass_a_tables(smem, septab, rec, ext, sparse, sparse_cap, sparse_count);
    WinSrc* ssrc = (WinSrc*)(smem + WA_OFF_SRC);
    const int t = threadIdx.x;
    if (t == 0) next_s = nwide_s = 0;
    const int npix = H * W, W1 = W + 1;
    const int nt = (npix + WT - 1) / WT;
    const int item = blockIdx.x;
    const int g = item / P, p = item - g * P, s0 = g * nsg, ns = min(nsg, S - s0);
    if (t < ns) ssrc[t] = win_source(info[s0 + t]);
    for (int r = t; r < ns * ND; r += WT) A.hist[r] = 0.;
    __syncthreads();
    if (!tables_ready(smem, status)) return;
    // warps take runs of 32 pixels from the item as they finish the last one: pixels next to
    // a source or at a row's edge cost several times the others
    const int pa = (int)((long long)p * nt / P) * WT, pb = min((int)((long long)(p + 1) * nt / P) * WT, npix);
    for (int pix = next_run(&next_s, pa); pix - (t & 31) < pb; pix = next_run(&next_s, pa)) {
        if (pix >= pb) continue;
        const int h = pix / W, w = pix - h * W;
        const PixBase Q = pixel_base(corners, centers, omega, W1, h, w, (size_t)pix);
        for (int j = 0; j < ns; ++j) {
            window_source<false>(Q, ssrc[j], corners, centers, W1, h, w, (size_t)(s0 + j) * npix + pix, A,
                                 A.hist + j * ND, nullptr, nullptr, j, &nwide_s, nullptr);
        }
    }
    __syncthreads();
    wide_of_item(min(nwide_s, WIDE_CAP), A, corners, W1, ssrc);
    if (nwide_s > WIDE_CAP) wide_left(A, corners, W1, ssrc, ns, s0, npix, pa, pb);
    __syncthreads();
    for (int r = t; r < ns * ND; r += WT) {
        const double v = A.hist[r];
        if (v != 0.) atomicAdd(hist_out + (size_t)s0 * ND + r, v);
    }
}

// Cutouts: one persistent launch over a work queue of (source, run) items, run = `run`
// consecutive pixels of the source's window (row-major, nw wide; a multiple of WT).  A
// block takes the next item from the queue (one atomic), builds its pixels' records
// and the item's map-integral rows in shared memory, and adds the rows it touched
// to hist_out[s] with FP64 atomics.  item_src[i] is the source of item i, tile_off[s]
// its first item and tile_off[S] the number of items.
__global__ void __launch_bounds__(WT, 3) k_pixel_windows_cut(const double* __restrict__ corners,
                                                          const double* __restrict__ centers,
                                                          const double* __restrict__ omega,
                                                          const SrcInfo* __restrict__ info,
                                                          const xts_cutout* __restrict__ cut,
                                                          const int* __restrict__ item_src,
                                                          const long long* __restrict__ tile_off,
                                                          unsigned long long* __restrict__ queue,
                                                          const SepTab* __restrict__ septab, int S, int W, int run,
                                                          double* __restrict__ hist_out, float4* __restrict__ rec,
                                                          float4* __restrict__ ext, float2* __restrict__ sparse,
                                                          int sparse_cap, int* __restrict__ sparse_count,
                                                          int* __restrict__ status) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ long long item_s;
    __shared__ int rmin_s, rmax_s, next_s;
    const PassA A = pass_a_tables(smem, septab, rec, ext, sparse, sparse_cap, sparse_count);
    WinSrc* ssrc = (WinSrc*)(smem + WA_OFF_SRC);
    const int t = threadIdx.x, W1 = W + 1;
    for (int r = t; r < ND; r += WT) A.hist[r] = 0.;
    __syncthreads();
    if (!tables_ready(smem, status)) return;
    const long long n_items = tile_off[S];
    for (;;) {
        if (t == 0) {
            const long long it = (long long)atomicAdd(queue, 1ull);
            item_s = it;
            rmin_s = ND;
            rmax_s = -1;
            next_s = 0;
            if (it < n_items) ssrc[0] = win_source(info[item_src[it]]);
        }
        __syncthreads();  // also orders the previous item's flush before this item's adds
        const long long item = item_s;
        if (item >= n_items) break;
        const int s = item_src[item];
        const xts_cutout cw = cut[s];
        const int npix = cw.nh * cw.nw, p0 = (int)((item - tile_off[s]) * run), p1 = min(npix, p0 + run);  // (<= 2^30)
        for (int pix = next_run(&next_s, p0); pix - (t & 31) < p1; pix = next_run(&next_s, p0)) {
            int4 e;
            bool wide = false;
            if (pix < p1) {
                const int i = pix / cw.nw, j = pix - i * cw.nw;
                const int h = cw.h0 + i, w = cw.w0 + j;
                const PixBase P = pixel_base(corners, centers, omega, W1, h, w, (size_t)h * W + w);
                wide = window_source<true>(P, ssrc[0], corners, centers, W1, h, w, (size_t)(cw.offset + pix), A, A.hist,
                                           &rmin_s, &rmax_s, 0, nullptr, &e);
            }
            wide_of_warp(wide, e, A, corners, W1, ssrc[0], (int4*)(smem + WA_OFF_WARP) + (t & ~31), &rmin_s, &rmax_s);
        }
        __syncthreads();
        for (int r = rmin_s + t; r <= rmax_s; r += WT) {
            const double v = A.hist[r];
            if (v != 0.) atomicAdd(hist_out + (size_t)s * ND + r, v);
            A.hist[r] = 0.;
        }
        __syncthreads();  // the flush has read rmin_s / rmax_s before thread 0 resets them
    }
}

// ============================================================================ pass B
// Work unit: a pair of pixels (2i, w), (2i + 1, w) per lane, 32 consecutive pairs of the
// source's map in (i, w) order per warp and tile.  Per float4 of output and table row an
// LDS.128 returns 512 bytes to the warp (four cycles of the SM's 128 bytes), whether or
// not the lanes' rows agree; a pair's two windows overlap (a table row is 3.4 % of the
// separation wide), so one load of their common rows feeds both pixels: about 3 rows per
// pair instead of 2 x 2.5.  Sums go quad by quad as packed FMAs straight into the stage,
// 4, 8 or 16 bytes per store as E allows (an even E at 4 bytes per lane has 2- to 4-way
// bank conflicts; those of the 16-byte stores, whose lanes are E floats apart, stay: 8-way
// for 32 energies, 4-way for 16 and 48, 2-way for 8, 24 and 40, none for 4 times an odd
// number: a call of 50 sources x 200 x 200 takes 375 us with 32 energies, 287 with 40, 387
// with 48 and 325 with 52).  Without its stores the pass takes 1.40 ms of 2.34 (400 x 400 x 37 x
// 500 sources; one pixel per lane at a time: 2.2), so HBM bounds it; where few warps fit
// beside the table (E = 50: 10) that is what it gains: 40 sources x 800 x 800 x 50 1.33 ->
// 1.04 ms.
constexpr int BQ = 13;   // float4 quads of a table row at most: E <= 52
constexpr int BWMAX = 16;  // warps per block at most
constexpr int NU = 6;    // common rows of a pair on the fast path

// Table row stride in float4 units: ceil(E/4), made odd.
static int win_row_quads(int E) {
    int nq = (E + 3) / 4;
    return (nq & 1) ? nq : nq + 1;
}

// Shared memory of a block of nw warps: the source's table, per warp two stages (the
// pair's upper and lower pixels) of 32 pixels and the alignment pads, an mbarrier.
struct WinLayout { size_t tab, stage, bar, total; };
static __host__ __device__ int stage_floats(int E) { return (32 * E + 8 + 3) / 4 * 4; }
static __host__ __device__ WinLayout win_layout(int E, int EQ, int nw) {
    WinLayout L;
    L.tab = 0;                                            // [ND + RW][EQ] float4 (RW zero guard rows)
    L.stage = (size_t)(ND + RW) * EQ * 16;
    L.bar = L.stage + sizeof(float) * (size_t)nw * 2 * stage_floats(E);
    L.total = L.bar + 16;
    return L;
}
// Warps per block: as many as shared memory holds beside the table, at most BWMAX; 12
// above 32 energies where the window records come from HBM (more than twice the 126 MB L2).
// Reads between the map's writes cost HBM more than their bytes (a bare copy of the pass's
// traffic at 400 x 400 x 37 x 500: 2.32-2.40 ms with the records, 1.86-1.90 without), and
// with more warps more so: 2.34 ms with 12, 2.40 with 14, 2.50 with 16, 2.56 with 10.  Fewer
// energies leave the pass short of loads in flight instead: 500 x 400 x 400 x 20 1.72 ms with
// 12, 1.45 with 16; x 28 (300 sources) 1.23 and 1.13; x 36 1.39 and 1.44.  37 energies:
// 35 sources 234 and 205 us, 100 (256 MB of records) 520 and 522, 125 628 and 645.
// Small jobs take as few warps per block as give every SM a block.
static int win_warps(int E, size_t rec_bytes, long long pairs, int nsm) {
    int nw = rec_bytes > ((size_t)256 << 20) && E > 32 ? 12 : BWMAX;
    const long long share = (pairs + 32LL * nsm - 1) / (32LL * nsm);
    if (share < nw) nw = share < 1 ? 1 : (int)share;
    while (nw > 0 && win_layout(E, win_row_quads(E), nw).total > 227 * 1024) --nw;
    return nw;
}

// A source's pixels in the write pass: the dense map (H x W, records from s * npix,
// output from (s_base + s) * npix) or a cutout window (records and output from
// cut[s].offset).
template <bool CUT>
struct SrcSpan {
    const xts_cutout* cut;
    int S, s_base, H, W, by;  // by: pairs per block and tile
    __device__ __forceinline__ int rows(int s) const { return !CUT ? H : s < S ? cut[s].nh : 0; }
    __device__ __forceinline__ int cols(int s) const { return !CUT ? W : s < S ? cut[s].nw : 0; }
    __device__ __forceinline__ long long rec_base(int s) const {
        return CUT ? cut[s].offset : (long long)s * ((long long)H * W);
    }
    __device__ __forceinline__ long long out_base(int s) const {
        return CUT ? cut[s].offset : (long long)(s_base + s) * ((long long)H * W);
    }
    __device__ __forceinline__ int pairs(int s) const { return (rows(s) + 1) / 2 * cols(s); }
    __device__ __forceinline__ int tiles(int s) const { return (pairs(s) + by - 1) / by; }
};

// One lane's place in a source's pairs and the main records of its pixels (hasB: the
// pair has a lower pixel).
struct PixPair { int i, col, pix; bool on, hasB; float4 ra, rb; };

template <bool CUT>
__device__ __forceinline__ void load_pair(PixPair& P, const SrcSpan<CUT>& sp, const float4* win, int s, bool more) {
    P.ra = P.rb = make_float4(0.f, 0.f, 0.f, 0.f);
    P.on = P.hasB = false;
    P.pix = 0;
    if (more) {
        const int H = sp.rows(s), W = sp.cols(s);
        P.on = 2 * P.i < H;
        P.hasB = 2 * P.i + 1 < H;
        P.pix = 2 * P.i * W + P.col;
        const float4* r = win + sp.rec_base(s) + P.pix;
        if (P.on) P.ra = __ldg(r);
        if (P.hasB) P.rb = __ldg(r + W);
    }
}

__device__ __forceinline__ int rec_rows(const float4& r) { const int m = __float_as_int(r.w); return m < 0 ? 0 : m >> 16; }
__device__ __forceinline__ int rec_first(const float4& r) { const int m = __float_as_int(r.w); return m < 0 ? 0 : m & 0xffff; }

// A quad of one pixel's values into the stage (dst: the pixel's quad, VW floats aligned),
// of which the first n count.
template <int VW>
__device__ __forceinline__ void store_quad(float* dst, int n, float2 lo, float2 hi) {
    if (VW == 4) {
        *(float4*)dst = make_float4(lo.x, lo.y, hi.x, hi.y);
    } else if (VW == 2) {
        *(float2*)dst = lo;
        if (n > 2) *(float2*)(dst + 2) = hi;
    } else {
        dst[0] = lo.x;
        if (n > 1) dst[1] = lo.y;
        if (n > 2) dst[2] = hi.x;
        if (n > 3) dst[3] = hi.y;
    }
}

// Both pixels' values from their K common rows (first row lo); packed FP32 FMAs.  Rows
// past a pixel's own window carry weight 0 (the table ends in RW zero rows), which adds
// nothing only where the table is finite: the caller sees to that.
template <int NQ, int K, int VW>
__device__ __forceinline__ void pair_values(const float4* tab, int EQ, const float4& ra, const float4& rb, int oa, int ob,
                                            int lo, bool hasB, float* da, float* db, int E) {
    const float4* row[K];
    float2 wa[K], wb[K];
#pragma unroll
    for (int j = 0; j < K; ++j) {
        row[j] = tab + (lo + j) * EQ;
        const float a = j == oa ? ra.x : j == oa + 1 ? ra.y : j == oa + 2 ? ra.z : 0.f;
        const float b = j == ob ? rb.x : j == ob + 1 ? rb.y : j == ob + 2 ? rb.z : 0.f;
        wa[j] = make_float2(a, a);
        wb[j] = make_float2(b, b);
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        float2 a0 = make_float2(0.f, 0.f), a1 = a0, b0 = a0, b1 = a0;
#pragma unroll
        for (int j = 0; j < K; ++j) {
            const float4 y = row[j][q];
            const float2 y0 = make_float2(y.x, y.y), y1 = make_float2(y.z, y.w);
            a0 = __ffma2_rn(wa[j], y0, a0);
            a1 = __ffma2_rn(wa[j], y1, a1);
            b0 = __ffma2_rn(wb[j], y0, b0);
            b1 = __ffma2_rn(wb[j], y1, b1);
        }
        const int n = q < NQ - 1 ? 4 : E - 4 * (NQ - 1);
        store_quad<VW>(da + 4 * q, n, a0, a1);
        if (hasB) store_quad<VW>(db + 4 * q, n, b0, b1);
    }
}

template <int NQ, int VW>
__device__ __forceinline__ void pair_values_k(int kmax, const float4* tab, int EQ, const float4& ra, const float4& rb,
                                              int oa, int ob, int lo, bool hasB, float* da, float* db, int E) {
    if (kmax <= 3) pair_values<NQ, 3, VW>(tab, EQ, ra, rb, oa, ob, lo, hasB, da, db, E);
    else if (kmax <= 4) pair_values<NQ, 4, VW>(tab, EQ, ra, rb, oa, ob, lo, hasB, da, db, E);
    else pair_values<NQ, NU, VW>(tab, EQ, ra, rb, oa, ob, lo, hasB, da, db, E);
}

// A wide pixel's values where the sparse pool was full: point by point from the table with a
// compensated sum.
__device__ __forceinline__ void point_values(const float4* tab, int EQ, int E, const double* corners,
                                             const double* omega, const SrcInfo* info, const SepTab* septab, int W1,
                                             int h, int w, size_t om, float* dst) {
    const SrcInfo si = *info;
    const PixGeom g = pixel_geom(corners, W1, h, w, si);
    const float o = omega ? (float)omega[om] : 1.f;
    const float* Y = (const float*)tab;
    const int ES = 4 * EQ;
    // the points' rows and weights once for all energies (formed again for each, an all-sky
    // map of 1 degree, 50 sources x 360 x 180 x 37, most of its pixels past the table's end
    // and beyond the pool, took 15.5 ms; so 1.7)
    int at[12];
    float wa[12], wb[12];
#pragma unroll
    for (int p = 0; p < 12; ++p) {
        float tt;
        at[p] = (point_row(point_q(g, p), septab->q, (const float4*)septab->coef, &tt) - 1) * ES;
        const float wgt = (float)c_rule_uv[p][3];
        wa[p] = (1.f - tt) * wgt;
        wb[p] = tt * wgt;
    }
#pragma unroll 1
    for (int e = 0; e < E; ++e) {
        float acc1 = 0.f, comp = 0.f;
#pragma unroll
        for (int p = 0; p < 12; ++p) {
            const float* yl = Y + at[p] + e;
            const float term = fmaf(wa[p], yl[0], wb[p] * yl[ES]);
            const float s2 = acc1 + term;
            comp += fabsf(acc1) >= fabsf(term) ? (acc1 - s2) + term : (term - s2) + acc1;
            acc1 = s2;
        }
        dst[e] = (acc1 + comp) * o;
    }
}

// One pixel's values by itself: a window of any length or a sparse record.
template <int NQ>
__device__ __forceinline__ void record_values(const float4* tab, int EQ, int E, const float4& rec, const float4* ext,
                                              const float2* sparse, float* dst) {
    const int meta = __float_as_int(rec.w);
    const int n = meta < 0 ? NSP : meta >> 16, r0 = meta < 0 ? 0 : meta & 0xffff;
    const float2* se = sparse + (size_t)(meta < 0 ? -1 - meta : 0) * NSP;
    float4 wx = rec, wy = make_float4(0.f, 0.f, 0.f, 0.f);
    if (meta >= 0 && n > REC_ROWS) {
        wx = __ldg(ext);
        wy = __ldg(ext + 1);
    }
    float4 acc[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) acc[q] = make_float4(0.f, 0.f, 0.f, 0.f);
    // Four entries' loads in flight (one at a time, as the compiler chose for 45 to 48 energies
    // once the function grew: 1 source x 224 x 224 x 45 27.7 us, 22.0 before, 19.9 so).  The
    // warps next to a source, whose pixels are all of this kind, are the last of a small job.
    for (int j = 0; j < n; j += 4) {
        float2 e[4];  // weight, row
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (meta < 0) {
                e[i] = __ldg(se + j + i);  // (NSP is a multiple of four)
            } else {
                const float lo4 = i == 0 ? wx.x : i == 1 ? wx.y : i == 2 ? wx.z : wx.w;
                const float hi4 = i == 0 ? wy.x : i == 1 ? wy.y : i == 2 ? wy.z : wy.w;
                e[i] = make_float2(j ? hi4 : lo4, __int_as_float(r0 + j + i));  // (n <= 8)
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (j + i >= n) break;
            const float wj = e[i].x;
            const float4* yr = tab + __float_as_int(e[i].y) * EQ;
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                const float4 y = yr[q];
                acc[q].x = fmaf(wj, y.x, acc[q].x);
                acc[q].y = fmaf(wj, y.y, acc[q].y);
                acc[q].z = fmaf(wj, y.z, acc[q].z);
                acc[q].w = fmaf(wj, y.w, acc[q].w);
            }
        }
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q)
        store_quad<1>(dst + 4 * q, q < NQ - 1 ? 4 : E - 4 * (NQ - 1), make_float2(acc[q].x, acc[q].y),
                      make_float2(acc[q].z, acc[q].w));
}

// Both for the kernel's rare pixels, in one function, or (dense maps up to 24 energies) one
// each: with the one, those kernels spilled 28 to 36 bytes of registers in their common path
// (28 sources x 757 x 757 x 15 energies: 326 us, 295 with two; 22 energies, 14 sources: 207 and
// 181), while the cutouts' kernel (37 energies, 500: 1,250 us, 1,300 with two) and the dense one
// of more energies (5 x 125 x 125 x 47: 22.0 and 24.0) lose by two.
template <int NQ>
__device__ __noinline__ void record_values_call(const float4* tab, int EQ, int E, const float4& rec, const float4* ext,
                                                const float2* sparse, float* dst) {
    record_values<NQ>(tab, EQ, E, rec, ext, sparse, dst);
}
__device__ __noinline__ void point_values_call(const float4* tab, int EQ, int E, const double* corners,
                                               const double* omega, const SrcInfo* info, const SepTab* septab, int W1,
                                               int h, int w, size_t om, float* dst) {
    point_values(tab, EQ, E, corners, omega, info, septab, W1, h, w, om, dst);
}
template <int NQ>
__device__ __noinline__ void pixel_values(const float4* tab, int EQ, int E, const float4& rec, const float4* ext,
                                          const float2* sparse, const double* corners, const double* omega,
                                          const SrcInfo* info, const SepTab* septab, int W1, int h, int w, size_t om,
                                          float* dst) {
    if (__float_as_int(rec.w) == META_OVERFLOW) point_values(tab, EQ, E, corners, omega, info, septab, W1, h, w, om, dst);
    else record_values<NQ>(tab, EQ, E, rec, ext, sparse, dst);
}

// A warp's 32 pairs in a map of fewer than 32 columns, five runs of consecutive pixels one
// after the other over both stages (whose pads hold the residues): the first pairs' upper and
// lower pixels (n1 each), both rows of the whole rows of pairs (pixels pixm .. pixl - 1), the
// last pairs' upper and lower pixels (rem each, from pixl).  Written pixel by pixel with plain
// stores, 300 x 400 x 31 x 37 values took 585 us, so 434; 20 columns 457 and 363.
struct NarrowRuns { int at[5], pixm, pixl, rem; };
__device__ __forceinline__ NarrowRuns narrow_runs(int pix0, int n1, int nv, int W, unsigned ob, int E) {
    NarrowRuns r;
    auto after = [&](int at, int pix) {
        return at + ((int)((ob + (unsigned)pix) * (unsigned)E - (unsigned)at) & 3);
    };
    const int nf = (nv - n1) / W;
    r.rem = nv - n1 - nf * W;
    r.pixm = (pix0 / (2 * W) + 1) * 2 * W;
    r.pixl = r.pixm + 2 * nf * W;
    r.at[0] = after(0, pix0);
    r.at[1] = after(r.at[0] + n1 * E, pix0 + W);
    r.at[2] = after(r.at[1] + n1 * E, r.pixm);
    r.at[3] = after(r.at[2] + 2 * nf * W * E, r.pixl);
    r.at[4] = after(r.at[3] + r.rem * E, r.pixl + W);
    return r;
}

// Warps run independently: each owns 32 pairs of the tile, its stages and its own TMA bulk
// stores, so no block barrier is needed except when the block moves on to the next
// source's table.  One block per SM.
// NARROW: a dense map of fewer than 32 columns (the cutouts' windows, wide and narrow ones, go
// through the form without it; one form for both had cost the wide maps and the cutouts up to
// 5 % in registers and code).
template <int NQ, bool CUT, bool NARROW>
__global__ void __launch_bounds__(32 * BWMAX, 1)
k_srcmap_win(const float4* __restrict__ win, const float4* __restrict__ ext, const float2* __restrict__ sparse,
             const float* __restrict__ lut, const double* __restrict__ corners, const double* __restrict__ omega,
             const SrcInfo* __restrict__ info, const SepTab* __restrict__ septab, const xts_cutout* __restrict__ cut,
             const long long* __restrict__ tile_off,
             int S, int s_base, int H, int W, int E, int EQ, int* status, float* __restrict__ out) {
    after_previous();
    extern __shared__ __align__(16) unsigned char smem[];
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31, nthr = blockDim.x;
    const WinLayout L = win_layout(E, EQ, nthr >> 5);
    float4* tab = (float4*)(smem + L.tab);
    const unsigned bar = smem_u32(smem + L.bar), full = 0xffffffffu;
    const int sf = stage_floats(E);
    float* stage = (float*)(smem + L.stage) + warp * 2 * sf;
    const int W1 = W + 1;
    const SrcSpan<CUT> sp{cut, S, s_base, H, W, nthr};
    const long long T = CUT ? tile_off[S] : (long long)S * sp.tiles(0);
    const long long f0 = T * blockIdx.x / gridDim.x, f1 = T * (blockIdx.x + 1) / gridDim.x;
    const unsigned tab_bytes = (unsigned)(ND * EQ * 16);

    for (int k = t; k < RW * EQ; k += nthr) tab[ND * EQ + k] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (t == 0) mbar_init(bar, 1);
    __syncthreads();

    int cur = -1;
    bool finite = true;  // the source's whole table: else each pixel's values by its own rows
    unsigned phase = 0;
    // (source, tile) of f, advanced by counting: no 64-bit division per tile
    int s, tile;
    if (CUT) {  // the source whose items hold f0: the last s with tile_off[s] <= f0
        int a = 0, b = S;
        while (b - a > 1) {
            const int mid = (a + b) >> 1;
            if (tile_off[mid] <= f0) a = mid; else b = mid;
        }
        s = a;
        while (s < S && tile_off[s + 1] <= f0) ++s;  // skip sources without tiles
        tile = (int)(f0 - tile_off[s]);
    } else {
        s = (int)(f0 / sp.tiles(0));
        tile = (int)(f0 - (long long)s * sp.tiles(0));
    }
    // the lane's pair of a tile: (i, col) by one division per source, then by steps of nthr
    PixPair P;
    int step_i = 0, step_c = 0;
    auto place = [&](int src, int tl) {
        const int Wn = max(sp.cols(src), 1), y = tl * nthr + t;
        P.i = y / Wn;
        P.col = y - P.i * Wn;
        step_i = nthr / Wn;
        step_c = nthr - step_i * Wn;
    };
    place(min(s, S - 1), tile);
    load_pair(P, sp, win, s, f0 < f1 && s < S && tile * nthr + t < sp.pairs(s));
    for (long long f = f0; f < f1; ++f) {
        int sn = s, tn = tile + 1;  // the next tile
        while (tn >= sp.tiles(sn) && sn < S) { tn = 0; ++sn; }
        // the next tile's records, in flight while this tile is computed
        const PixPair C = P;
        const int Ws = sp.cols(s);
        if (sn == s) {
            P.i += step_i;
            P.col += step_c;
            if (P.col >= Ws) { P.col -= Ws; ++P.i; }
        } else if (sn < S) {
            place(sn, tn);
        }
        load_pair(P, sp, win, sn, f + 1 < f1 && sn < S && tn * nthr + t < sp.pairs(sn));
        if (s != cur) {
            __syncthreads();  // every warp is done with the previous source's table
            if (t == 0) {
                fence_async_shared();
                bulk_load(tab, lut + (size_t)s * ND * EQ * 4, tab_bytes, bar);
            }
            cur = s;
            const bool ok = mbar_wait(bar, phase);
            phase ^= 1;
            if (!__syncthreads_and(ok)) {
                if (t == 0) {
                    atomicExch(status, 1);
                    mbar_wait(bar, phase ^ 1);  // bounded: let the copy land before the block exits
                }
                if ((lane & 7) == 0) bulk_wait_all();
                return;
            }
            // (one float4 at a time cost jobs of a few sources 1 to 2 us)
            float2 z0 = make_float2(0.f, 0.f), z1 = z0;  // 0, or NaN
#pragma unroll 4
            for (int k = t; k < ND * EQ; k += nthr) {
                const float4 y = tab[k];
                z0 = __ffma2_rn(make_float2(y.x, y.y), make_float2(0.f, 0.f), z0);
                z1 = __ffma2_rn(make_float2(y.z, y.w), make_float2(0.f, 0.f), z1);
            }
            finite = __syncthreads_and((z0.x + z0.y) + (z1.x + z1.y) == 0.f);
        }
        const int nv = __popc(__ballot_sync(full, C.on));  // lanes with pixels (the first nv)
        // runs of consecutive pixels: lanes [0, n1) end a map row, lanes [n1, nv) begin the
        // next pair's; a pixel's stage position is its flat output index modulo 4
        const int n1 = min(Ws - __shfl_sync(full, C.col, 0), nv);
        const bool narrow = CUT && Ws < 32;  // more runs than two: written by plain stores
        const int pix0 = __shfl_sync(full, C.pix, 0), pix1 = __shfl_sync(full, C.pix, n1 & 31);
        const unsigned ob = (unsigned)sp.out_base(s), uE = (unsigned)E;  // (residues: 32 bits suffice)
        auto residue = [&](int pix, int l) { return (int)(((ob + (unsigned)pix - (unsigned)l) * uE) & 3u); };
        int mA0 = residue(pix0, 0), mB0 = residue(pix0 + Ws, 0);
        int mA1 = mA0 + ((residue(pix1, n1) - mA0) & 3), mB1 = mB0 + ((residue(pix1 + Ws, n1) - mB0) & 3);
        if (narrow) mA0 = mA1 = mB0 = mB1 = 0;
        float* da = stage + (lane < n1 ? mA0 : mA1) + lane * E;
        float* db = stage + sf + (lane < n1 ? mB0 : mB1) + lane * E;
        NarrowRuns nr;
        if (NARROW) {
            nr = narrow_runs(pix0, n1, nv, Ws, ob, E);
            const int l = lane - (nv - nr.rem);  // of the last pairs
            if (l >= 0) {
                da = stage + nr.at[3] + l * E;
                db = stage + nr.at[4] + l * E;
            } else if (lane >= n1) {
                da = stage + nr.at[2] + (C.pix - nr.pixm) * E;
                db = da + Ws * E;
            } else {
                da = stage + nr.at[0] + lane * E;
                db = stage + nr.at[1] + lane * E;
            }
        }

        // the stages are reused only now: the previous bulk stores' read-out overlapped the loads
        if ((lane & 7) == 0) bulk_wait_read();
        __syncwarp();
        const int na = rec_rows(C.ra), nb = rec_rows(C.rb), fa = rec_first(C.ra), fb = C.hasB ? rec_first(C.rb) : fa;
        const int lo = min(fa, fb), n = max(fa + na, fb + nb) - lo;
        const bool own = C.on && (!finite || __float_as_int(C.ra.w) < 0 || __float_as_int(C.rb.w) < 0 ||
                                  na > REC_ROWS || nb > REC_ROWS || n > NU);
        const int kmax = __reduce_max_sync(full, C.on ? n : 0);
        if (!__any_sync(full, own)) {
            if (C.on) {
                if (!(E & 3)) pair_values_k<NQ, 4>(kmax, tab, EQ, C.ra, C.rb, fa - lo, fb - lo, lo, C.hasB, da, db, E);
                else if (!(E & 1)) pair_values_k<NQ, 2>(kmax, tab, EQ, C.ra, C.rb, fa - lo, fb - lo, lo, C.hasB, da, db, E);
                else pair_values_k<NQ, 1>(kmax, tab, EQ, C.ra, C.rb, fa - lo, fb - lo, lo, C.hasB, da, db, E);
            }
        } else if (C.on) {
            int h = 2 * C.i, w = C.col;  // (the lower pixel: h + 1)
            const size_t k = (size_t)(sp.rec_base(s) + C.pix);
            if (CUT) {
                h += cut[s].h0;
                w += cut[s].w0;
            }
            for (int b = 0; b < (C.hasB ? 2 : 1); ++b) {
                const float4* x = ext + 2 * (k + (b ? Ws : 0));
                const size_t om = (size_t)(h + b) * W + w;
                if (CUT || NQ > 6)
                    pixel_values<NQ>(tab, EQ, E, b ? C.rb : C.ra, x, sparse, corners, omega, info + s, septab, W1, h + b, w,
                                     om, b ? db : da);
                else if (__float_as_int(b ? C.rb.w : C.ra.w) == META_OVERFLOW)
                    point_values_call(tab, EQ, E, corners, omega, info + s, septab, W1, h + b, w, om, b ? db : da);
                else
                    record_values_call<NQ>(tab, EQ, E, b ? C.rb : C.ra, x, sparse, b ? db : da);
            }
        }
        fence_async_shared();
        __syncwarp();
        const unsigned hb = __ballot_sync(full, C.hasB);
        if (NARROW) {  // as below, a run after the other
            const int l = lane & 7, lower = (lane >> 3) & 1;
            const bool second = lane >= 16;
            const int l0 = second ? nv - nr.rem : 0, cnt = second ? nr.rem : n1;
            const bool on = cnt > 0 && (!lower || ((hb >> l0) & 1));
#pragma unroll 1
            for (int k = 0; k < (nr.pixl > nr.pixm ? 2 : 1); ++k) {  // (a map of odd height has no last lower row)
                const int pix = k ? nr.pixm : (second ? nr.pixl : pix0) + lower * Ws;
                const int n = k ? (lane < 8 ? min(nr.pixl, H * W) - nr.pixm : 0) : on ? cnt : 0;
                const int at = k ? nr.at[2] : second ? (lower ? nr.at[4] : nr.at[3]) : lower ? nr.at[1] : nr.at[0];
                if (n <= 0) continue;
                const float* src = stage + at;
                float* dst = out + (sp.out_base(s) + pix) * E;
                const int nf = n * E, head = min((int)((4u - (unsigned)at) & 3u), nf), body = (nf - head) & ~3;
                if (l == 0 && body > 0) bulk_store(dst + head, src + head, (unsigned)body * 4u);
                const int e = l < 4 ? l : head + body + l - 4;
                if (l < 4 ? e < head : e < nf) dst[e] = src[e];
            }
        } else if (!narrow) {
            // eight lanes per run: a TMA bulk store of its 16-byte aligned body, lanes for the edges
            const int l = lane & 7, lower = (lane >> 3) & 1;
            const bool second = lane >= 16;
            const int l0 = second ? n1 : 0, cnt = (second ? nv : n1) - l0;
            if (cnt > 0 && (!lower || ((hb >> l0) & 1))) {
                const int m = lower ? (second ? mB1 : mB0) : (second ? mA1 : mA0);
                const float* src = stage + lower * sf + m + l0 * E;
                float* dst = out + (sp.out_base(s) + (second ? pix1 : pix0) + lower * Ws) * E;
                const int nf = cnt * E, head = min((int)((4u - (unsigned)(m + l0 * E)) & 3u), nf);
                const int body = (nf - head) & ~3;
                if (l == 0 && body > 0) bulk_store(dst + head, src + head, (unsigned)body * 4u);
                const int e = l < 4 ? l : head + body + l - 4;
                if (l < 4 ? e < head : e < nf) dst[e] = src[e];
            }
        } else {
            for (int l = 0; l < nv; ++l) {
                const int pix = __shfl_sync(full, C.pix, l);
                for (int e = lane; e < E; e += 32) {
                    float* o = out + (sp.out_base(s) + pix) * E + e;
                    o[0] = stage[l * E + e];
                    if ((hb >> l) & 1) o[(size_t)Ws * E] = stage[sf + l * E + e];
                }
            }
            __syncwarp();
        }
        s = sn;
        tile = tn;
    }
    if ((lane & 7) == 0) bulk_wait_all();
}

// Resident blocks per SM of a kernel at a launch shape, asked of the driver once per kernel,
// shape and device (the answer does not change); the kernel's shared-memory limit is raised
// to the largest shape asked for.  Calls are serialised by the library's lock.
template <typename F>
static int resident_blocks(F* kernel, int threads, size_t smem, int dev, int* out) {
    struct Known { const void* k; int threads, dev, blocks; size_t smem; };
    static std::vector<Known> known;
    size_t limit = 0;
    for (const Known& n : known) {
        if (n.k != (const void*)kernel || n.dev != dev) continue;
        if (n.threads == threads && n.smem == smem) { *out = n.blocks; return XTS_OK; }
        if (n.smem > limit) limit = n.smem;
    }
    if (smem > limit)
        XTS_CUDA(cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    XTS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(out, (const void*)kernel, threads, smem));
    known.push_back(Known{(const void*)kernel, threads, dev, *out, smem});
    return XTS_OK;
}

struct WriteArgs {
    const float4* win; const float4* ext; const float2* sparse; const float* lut;
    const double* corners; const double* omega; const SrcInfo* info; const SepTab* tab;
    const xts_cutout* cut; const long long* tile_off;  // cutouts (cut != NULL): tile_off [S + 1] in tiles of pairs
    int S, s_base, H, W, E, EQ;
    int* status; float* out;
};

template <int NQ>
static int launch_write_pass(unsigned G, int warps, size_t smem, cudaStream_t st, const WriteArgs& a, int* per_sm,
                             bool query) {
    const int BT = 32 * warps;
    if (query) {
        int pd = 0, pn = 0, pc = 0, dev = 0, rc;
        cudaGetDevice(&dev);
        if ((rc = resident_blocks(k_srcmap_win<NQ, false, false>, BT, smem, dev, &pd))) return rc;
        if ((rc = resident_blocks(k_srcmap_win<NQ, false, true>, BT, smem, dev, &pn))) return rc;
        if ((rc = resident_blocks(k_srcmap_win<NQ, true, false>, BT, smem, dev, &pc))) return rc;
        *per_sm = pd < pc ? pd : pc;
        if (pn < *per_sm) *per_sm = pn;
        return XTS_OK;
    }
    if (a.cut)
        XTS_LAUNCH("k_srcmap", st, launch_next(
                                       k_srcmap_win<NQ, true, false>, G, BT, smem, st, a.win, a.ext, a.sparse, a.lut,
                                       a.corners, a.omega, a.info, a.tab, a.cut, a.tile_off, a.S, a.s_base, a.H, a.W, a.E, a.EQ, a.status, a.out));
    else
        XTS_LAUNCH("k_srcmap", st, launch_next(
                                       a.W < 32 ? k_srcmap_win<NQ, false, true> : k_srcmap_win<NQ, false, false>, G, BT, smem, st, a.win, a.ext, a.sparse, a.lut,
                                       a.corners, a.omega, a.info, a.tab, nullptr, nullptr, a.S, a.s_base, a.H, a.W, a.E, a.EQ, a.status, a.out));
    return XTS_OK;
}

typedef int (*WritePassFn)(unsigned, int, size_t, cudaStream_t, const WriteArgs&, int*, bool);
static const WritePassFn k_write_pass[BQ] = {
    launch_write_pass<1>, launch_write_pass<2>, launch_write_pass<3>, launch_write_pass<4>, launch_write_pass<5>,
    launch_write_pass<6>, launch_write_pass<7>, launch_write_pass<8>, launch_write_pass<9>, launch_write_pass<10>,
    launch_write_pass<11>, launch_write_pass<12>, launch_write_pass<13>};

// ============================================================================ host
bool srcmap_win_supported(int E) {
    return E >= 1 && E <= 4 * BQ && win_warps(E, 0, 1LL << 40, 1) > 0;
}

// Sources per group of the dense window pass: a pixel's own geometry (a third of the work
// of one source) is formed once per group, while there are items (group, tile) for every
// resident block twice over.
static int window_group(int n, int ntile, int G) {
    int nsg = NSG_MAX;
    while (nsg > 1 && (long long)((n + nsg - 1) / nsg) * ntile < 2LL * G) nsg >>= 1;
    return nsg;
}
constexpr int ITEMS = 8;  // work items per resident block
// Parts per source group (n sources of ntile tiles, G blocks): about ITEMS items per
// resident block (500 sources x 400 x 400: 1.52 ms at 4, 1.34 at 8, 1.35 at 16; 40 x 800 x
// 800: 383 us at 8, 397 at 16), at most one part per tile.
static int window_parts(int n, int nsg, int ntile, int G) {
    const long long ng = (n + nsg - 1) / nsg;
    long long P = ((long long)ITEMS * G + ng - 1) / ng;
    if (P > ntile) P = ntile;
    return P < 1 ? 1 : (int)P;
}

// Window records of one source chunk: a 16-byte main record and a 32-byte
// extension slot per (source, pixel); only windows of more than REC_ROWS rows
// write and read their extension.
static size_t win_bytes_per_source(int npix) { return (size_t)npix * 48; }

// When the sources come in several chunks (host-mode copy-out, or records above
// the buffer budget) and a geometry stream is given, the window pass of chunk k + 1
// (geometry stream) may run while chunk k is corrected and written (launching
// stream): window records, sparse records, row histograms and scaled tables are
// double-buffered and events order each buffer's reuse.  Splitting a device-mode
// job into chunks only for this overlap was measured slower (c1: 0.375 ms in 2
// chunks, 0.392 in 4, 0.320 in one), so a device-mode job is one chunk.

int launch_srcmap_win(const double* corners, const double* centers, const double* omega,
                      const SrcInfo* info, int S, int H, int W, int E,
                      const double* upsf, const double* partial, const double* exposure,
                      double* scale, double* inv_integ, double* correction, double* radius,
                      int* in_fov, int* status, float* out, int chunk_sources,
                      int (*on_chunk)(void*, int, int, cudaStream_t), void* on_chunk_ctx,
                      StreamJoin& geo, cudaStream_t st, bool means_only) {
    int rc = upload_rule_uv(st);
    if (rc) return rc;
    const SepTab* tab = nullptr;
    rc = build_septab(st, &tab);
    if (rc) return rc;
    const cudaStream_t gs = geo.from;
    const bool pipe = gs != st;
    const int npix = H * W;
    const int EQ = win_row_quads(E);
    // sources per chunk: window records and their extensions of at most 4 GiB; two sets of
    // buffers where there is more than one chunk
    const size_t budget = (size_t)4 << 30;
    int Sc = (int)(budget / win_bytes_per_source(npix));
    if (chunk_sources > 0 && chunk_sources < Sc) Sc = chunk_sources;
    if (g_tuning.chunk_sources > 0 && g_tuning.chunk_sources < Sc) Sc = g_tuning.chunk_sources;
    Sc = Sc < 1 ? 1 : (Sc > S ? S : Sc);
    int dev = 0, nsm = 148, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const int nw = win_warps(E, (size_t)Sc * npix * 16, (long long)Sc * ((H + 1) / 2) * W, nsm);
    const WinLayout L = win_layout(E, EQ, nw);
    const size_t rec_n = (size_t)Sc * npix + 4, ext_n = (size_t)Sc * npix * 2 + 4;
    const size_t lut_n = (size_t)Sc * ND * EQ * 4 + 4;
    // sparse records for wide pixels: room for 1/8 of the chunk's pixels (at least 64k)
    long long cap = (long long)Sc * npix / 8;
    cap = cap < 65536 ? 65536 : cap;
    cap = cap > (long long)Sc * npix ? (long long)Sc * npix : cap;
    const size_t sp_n = (size_t)NSP * cap + 2, nset = Sc < S ? 2 : 1;
    float4* rec0 = (float4*)workspace(W_WIN, sizeof(float4) * nset * rec_n);
    float4* ext0 = (float4*)workspace(W_WMETA, sizeof(float4) * nset * ext_n);
    float* lut0 = (float*)workspace(W_LUT, sizeof(float) * nset * lut_n);
    float2* sparse0 = (float2*)workspace(W_SPARSE, sizeof(float2) * nset * sp_n);
    // pass A: one block per work item, items sized for about 8 per block of the
    // resident set (at most window_blocks_per_sm blocks per SM)
    int resident = 0;
    if ((rc = resident_blocks(k_pixel_windows, WT, wa_smem(NSG_MAX), dev, &resident))) return rc;
    resident = resident < 1 ? 1 : resident;
    if (g_tuning.window_blocks_per_sm > 0 && g_tuning.window_blocks_per_sm < resident)
        resident = g_tuning.window_blocks_per_sm;
    const int ntile = (npix + WT - 1) / WT, nsg = window_group(Sc, ntile, resident * nsm);
    const int nparts = window_parts(Sc, nsg, ntile, resident * nsm);
    const size_t hist_n = (size_t)Sc * ND + 1;  // the last double: the sparse records' count
    double* hist0 = (double*)workspace(W_PARTSUM, sizeof(double) * nset * hist_n);
    if (!rec0 || !ext0 || !lut0 || !sparse0 || !hist0) return XTS_ERR_OOM;
    const WritePassFn wp = k_write_pass[(E + 3) / 4 - 1];
    rc = wp(0, nw, L.total, st, WriteArgs{}, &per_sm, true);
    if (rc) return rc;
    if (per_sm < 1) return set_error(XTS_ERR_ARG, "source-map write pass does not fit on an SM (E=%d)", E);
    cudaEvent_t evA[2], evB[2];  // window pass of a buffer done; write pass of a buffer done
    pipe_events(evA, evB);
    int k = 0;
    for (int s0 = 0; s0 < S; s0 += Sc, ++k) {
        const int n = S - s0 < Sc ? S - s0 : Sc, b = k & 1;
        const size_t oE = (size_t)s0 * E;
        float4* rec = rec0 + b * rec_n;
        float4* ext = ext0 + b * ext_n;
        float* lut = lut0 + b * lut_n;
        float2* sparse = sparse0 + b * sp_n;
        double* hist = hist0 + b * hist_n;
        int* sparse_count = (int*)(hist + (size_t)n * ND);
        // the window pass is geometry only: it runs on the geometry stream, once
        // the write pass that last read its buffers is done
        if (pipe && k >= 2) XTS_CUDA(cudaStreamWaitEvent(gs, evB[b], 0));
        const int n_items = (n + nsg - 1) / nsg * nparts;  // one block per item
        XTS_CUDA(cudaMemsetAsync(hist, 0, sizeof(double) * ((size_t)n * ND + 1), gs));
        XTS_LAUNCH("k_pixel_windows", gs, k_pixel_windows<<<n_items, WT, wa_smem(nsg), gs>>>(
                                              corners, centers, means_only ? nullptr : omega, info + s0, tab, n, H, W,
                                              nparts, nsg, hist, rec, ext, sparse, (int)cap,
                                              sparse_count, status));
        if (Sc >= S) {  // one chunk: nothing else follows on the geometry stream
            if ((rc = geo.join())) return rc;
        } else if (pipe) {
            XTS_CUDA(cudaEventRecord(evA[b], gs));
            XTS_CUDA(cudaStreamWaitEvent(st, evA[b], 0));
        }
        if (means_only) {
            XTS_LAUNCH("k_lut_scaled", st, k_lut_scaled<<<lut_scaled_grid(n), 256, 0, st>>>(
                                               upsf + oE * ND, nullptr, n, E, EQ * 4, lut, nullptr, nullptr));
        } else {
            rc = launch_correction(hist, 1, info + s0, n, upsf + oE * ND, partial + oE * ND,
                                   exposure + oE, E, scale + oE, inv_integ ? inv_integ + oE : nullptr,
                                   correction ? correction + oE : nullptr, radius ? radius + s0 : nullptr,
                                   in_fov ? in_fov + s0 : nullptr, st, lut, EQ * 4);
            if (rc) return rc;
        }
        const long long T = (long long)n * (((H + 1) / 2 * W + 32 * nw - 1) / (32 * nw));
        long long G = (long long)nsm * (g_tuning.write_blocks_per_sm > 0 && g_tuning.write_blocks_per_sm < per_sm
                                            ? g_tuning.write_blocks_per_sm : per_sm);
        if (G > T) G = T;
        WriteArgs wa{rec, ext, sparse, lut, corners, means_only ? nullptr : omega, info + s0, tab, nullptr, nullptr,
                     n, s0, H, W, E, EQ, status, out};
        rc = wp((unsigned)G, nw, L.total, st, wa, nullptr, false);
        if (rc) return rc;
        if (on_chunk && (rc = on_chunk(on_chunk_ctx, s0, n, st))) return rc;
        if (pipe && Sc < S) XTS_CUDA(cudaEventRecord(evB[b], st));
    }
    return geo.join();
}

// ============================================================================ cutouts
// Items of the cutout work queue: tile_off[s] = the first (source, tile) item of
// source s (runs of `run` pixels of its window), tile_off[S] = the item count.  One
// block; the sources in runs of 1024 with a block scan.
// For the write pass the same of tiles of `by` pixel pairs: pair_off.
__global__ void __launch_bounds__(1024) k_cut_tiles(const xts_cutout* __restrict__ cut, int S, int by, int run,
                                                    long long* __restrict__ tile_off,
                                                    long long* __restrict__ pair_off) {
    // (two scans, one block each)
    if (blockIdx.x) tile_off = pair_off;
    __shared__ long long part[32];
    __shared__ long long carry_s;
    const int t = threadIdx.x, lane = t & 31, wp = t >> 5;
    if (t == 0) carry_s = 0;
    __syncthreads();
    for (int s0 = 0; s0 < S; s0 += 1024) {
        const int s = s0 + t;
        long long n = 0;
        if (s < S)
            n = blockIdx.x ? ((long long)(cut[s].nh + 1) / 2 * cut[s].nw + by - 1) / by
                           : ((long long)cut[s].nh * cut[s].nw + run - 1) / run;
        long long inc = n;
        for (int o = 1; o < 32; o <<= 1) {
            const long long v = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += v;
        }
        if (lane == 31) part[wp] = inc;
        __syncthreads();
        long long before = carry_s;
        for (int k = 0; k < wp; ++k) before += part[k];
        if (s < S) tile_off[s] = before + inc - n;
        __syncthreads();
        if (t == 1023) carry_s = before + inc;
        __syncthreads();
    }
    if (t == 0) tile_off[S] = carry_s;
}

// item_src[i] = the source of item i (one block per source).
__global__ void k_cut_item_src(const long long* __restrict__ tile_off, int* __restrict__ item_src) {
    const int s = blockIdx.x;
    for (long long i = tile_off[s] + threadIdx.x; i < tile_off[s + 1]; i += blockDim.x) item_src[i] = s;
}

int launch_srcmap_win_cut(const double* corners, const double* centers, const double* omega, const SrcInfo* info,
                          const xts_cutout* cut, int S, int H, int W, int E, const double* upsf,
                          const double* partial, const double* exposure, double* scale, double* inv_integ,
                          double* correction, double* radius, int* in_fov, int* status, float* out, cudaStream_t st) {
    int rc = upload_rule_uv(st);
    if (rc) return rc;
    const SepTab* tab = nullptr;
    if ((rc = build_septab(st, &tab))) return rc;
    const long long npix = (long long)H * W;
    const int EQ = win_row_quads(E);
    int dev = 0, nsm = 148, resident = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const int nw = win_warps(E, (size_t)S * npix * 16, (long long)S * npix / 2, nsm);
    const WinLayout L = win_layout(E, EQ, nw);
    // buffers sized for the largest windows (every window the whole map): nothing here
    // depends on the windows' sizes on the host, so the call needs no synchronisation
    const long long max_items = (long long)S * ((npix + WT - 1) / WT);
    // pixels per item: eight tiles where there are plenty (an item's queue access, barriers and
    // flush of its rows are then shared by eight pixels per thread), one in small jobs
    const int run = max_items >= 16384 ? 8 * WT : max_items >= 4096 ? 2 * WT : WT;
    const size_t rec_n = (size_t)S * npix + 4;
    float4* rec = (float4*)workspace(W_WIN, sizeof(float4) * rec_n);
    float4* ext = (float4*)workspace(W_WMETA, sizeof(float4) * 2 * rec_n);
    float* lut = (float*)workspace(W_LUT, sizeof(float) * ((size_t)S * ND * EQ * 4 + 4));
    long long cap = (long long)S * npix / 8;
    cap = cap < 65536 ? 65536 : cap;
    float2* sparse = (float2*)workspace(W_SPARSE, sizeof(float2) * ((size_t)NSP * cap + 2));
    double* hist = (double*)workspace(W_PARTSUM, sizeof(double) * ((size_t)S * ND + 1));
    char* items = (char*)workspace(W_CUT_ITEMS, 2 * align_up(sizeof(long long) * (S + 1), 256) +
                                                    align_up(sizeof(int) * (size_t)max_items, 256) + 256);
    if (!rec || !ext || !lut || !sparse || !hist || !items) return XTS_ERR_OOM;
    long long* pair_off = (long long*)items;
    items += align_up(sizeof(long long) * (S + 1), 256);
    long long* tile_off = (long long*)items;
    int* item_src = (int*)(items + align_up(sizeof(long long) * (S + 1), 256));
    unsigned long long* queue = (unsigned long long*)(items + align_up(sizeof(long long) * (S + 1), 256) +
                                                      align_up(sizeof(int) * (size_t)max_items, 256));
    int* sparse_count = (int*)(hist + (size_t)S * ND);
    XTS_CUDA(cudaMemsetAsync(hist, 0, sizeof(double) * ((size_t)S * ND + 1), st));
    XTS_CUDA(cudaMemsetAsync(queue, 0, sizeof(unsigned long long), st));
    XTS_LAUNCH("k_cut_tiles", st, k_cut_tiles<<<2, 1024, 0, st>>>(cut, S, 32 * nw, run, tile_off, pair_off));
    XTS_LAUNCH("k_cut_item_src", st, k_cut_item_src<<<S, 256, 0, st>>>(tile_off, item_src));
    if ((rc = resident_blocks(k_pixel_windows_cut, WT, WA_CUT_SMEM, dev, &resident))) return rc;
    resident = resident < 1 ? 1 : resident;
    if (g_tuning.queue_blocks_per_sm > 0 && g_tuning.queue_blocks_per_sm < resident) resident = g_tuning.queue_blocks_per_sm;
    // pass A: one persistent wave pulling (source, tile) items from the queue
    XTS_LAUNCH("k_pixel_windows", st, k_pixel_windows_cut<<<(unsigned)(resident * nsm), WT, WA_CUT_SMEM, st>>>(
                                          corners, centers, omega, info, cut, item_src, tile_off, queue, tab, S, W, run,
                                          hist, rec, ext, sparse, (int)cap, sparse_count, status));
    rc = launch_correction(hist, 1, info, S, upsf, partial, exposure, E, scale, inv_integ, correction, radius, in_fov,
                           st, lut, EQ * 4);
    if (rc) return rc;
    const WritePassFn wp = k_write_pass[(E + 3) / 4 - 1];
    if ((rc = wp(0, nw, L.total, st, WriteArgs{}, &per_sm, true))) return rc;
    if (per_sm < 1) return set_error(XTS_ERR_ARG, "source-map write pass does not fit on an SM (E=%d)", E);
    WriteArgs wa{rec, ext, sparse, lut, corners, omega, info, tab, cut, pair_off, S, 0, H, W, E, EQ, status, out};
    if (g_tuning.write_blocks_per_sm > 0 && g_tuning.write_blocks_per_sm < per_sm) per_sm = g_tuning.write_blocks_per_sm;
    // pass B: one persistent wave over the same items, split evenly between the blocks
    return wp((unsigned)(nsm * per_sm), nw, L.total, st, wa, nullptr, false);
}

}  // namespace xts
