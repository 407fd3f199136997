// xts_psf.cu -- step (b): exposure-weighted mean King PSF tables.
//
//   b2 separations            psf/psf.hxx:24-31
//   b3 King table [D,Mc,Me]   psf/psf.king.cxx:9-43
//   b4 bilerp -> [C,D,E]      psf/psf.bilerp.cxx:6-52
//   b5 corrected_exposure_psf psf/psf.corrected_exposure_psf.cxx:12-120
//   b6 mean_psf               psf/psf.mean_psf.cxx:6-33
//   b7 partial/total, normalise psf/psf.partial_total_integral.cxx:8-52, psf/psf.normalize.cxx:7-24
//
// Front and back both use the front livetime-efficiency factors
// (psf.psf_lookup_table_and_partial_integrals.cxx:151-156), so the two sides'
// psf*aeff tables are summed before the contraction over cos-theta:
//   mean[s,d,e] = (sum_c (X[s,c] L0[e] + W[s,c] L1[e]) (Pf Af + Pb Ab)[c,d,e]) / exposure[s,e]
// which is the reference's four DGEMMs and three sums reassociated.
#include <math.h>

#include "xts_internal.cuh"
#include "xts_tables.cuh"

namespace xts {

// b5, b6 and b7 in one kernel: a block forms the mean PSF of TS sources at TE energies
// over all 401 rows in shared memory, integrates it and writes uPsf and the partial
// integrals once (three passes over them in memory before).
//
// Contraction: FP64 tensor-core products (m8n8k4, FP64 sums): the TS sources' livetime
// and weighted-livetime rows (from shared memory) against 8 rows of one energy's psf*aeff
// per tile, read from L2 with a tile's loads in flight during the previous one's products.
// On the FMA pipe the same tile is held to under half of the pipe's rate by shared memory:
// every broadcast of a livetime pair returns 512 bytes to the warp for four FMAs (2000
// sources x 50 energies: 0.48 ms for the contraction against 0.37 here, 0.26 without the
// loads).  The tile's products also go into the total integral, a fixed linear function of
// the rows, so the scan needs no pass of its own for it.
//
// Integral (psf.partial_total_integral.cxx:8-52, psf.normalize.cxx:7-24): per (s, e)
// the exact integral of the linear interpolant of 2 pi u(theta) sin(theta) over each
// separation bin, its prefix sums, both divided by the total.  One warp per (s, e): a
// lane integrates a run of 13 bins, the runs are joined by a shuffle scan.  The
// reference forms the bin integral as 0.5 m (t2^2 - t1^2) + b (t2 - t1) with the slope m
// and intercept b of the interpolant; that is exactly the trapezoid 0.5 (t2 - t1)(y1 + y2),
// used here without its division (the two agree to a few ulp), and the normalisation
// multiplies by 1/total.  uPsf is written before the prefix sums take its place in the tile.
//
// 2000 sources x 50 energies: 0.56 ms (contraction 0.37, scan 0.06, write-out 0.13 of
// 640 MB), where a contraction kernel and a scan kernel with the energy as its inner stride
// took 0.64 + 0.94.  The pitch of the tile (NDP = 4 mod 16 doubles) keeps both the row-wise
// accesses and the (row, energy)-wise ones of the write-out free of bank conflicts.
constexpr int PSF_MAX_C = 64;
constexpr int PSF_MAX_E = 1226;
constexpr int PM_THREADS = 384;
constexpr int PSF_KS = 10;                      // k steps (4 cos-theta bins each) loaded at a time
constexpr int PSCAN_ROWS = (ND - 1 + 31) / 32;  // bins per lane

// Row pitch of the livetime rows in shared memory: whole groups of PSF_KS k steps (zeros
// past C) and 4 mod 16 doubles, so that a fragment's 8 x 4 elements fall in different banks.
__host__ __device__ constexpr int psf_row_pitch(int C) {
    const int K = (C + 4 * PSF_KS - 1) / (4 * PSF_KS) * (4 * PSF_KS);
    return K + (20 - K % 16) % 16;
}

static constexpr size_t psf_mean_smem(int TS, int TE, int C) {
    const size_t tabs = sizeof(double) * 2 * NDP, rows = sizeof(double) * 2 * (size_t)psf_row_pitch(C) * TS;
    return sizeof(double) * ((size_t)TS * TE * NDP + 2 * (size_t)TS * TE + PM_THREADS / 32 * (size_t)TS) + (tabs > rows ? tabs : rows) + 16;
}

__device__ __forceinline__ void dmma(double* c, double a, double b) {  // C[8][8] += A[8][4] B[4][8]
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
        : "+d"(c[0]), "+d"(c[1]) : "d"(a), "d"(b));
}

// Per-lane run of the (s, e) row y: cum[k] = its prefix integral over bins d0 .. d0 + k.
__device__ __forceinline__ double scan_run(const double* y, const double* st, const double* hdt, int d0, double* cum) {
    double run = 0.0;
    const int d1 = min(ND, d0 + PSCAN_ROWS);
    if (d0 < ND) {
        double y1 = y[d0 - 1] * st[d0 - 1];
#pragma unroll
        for (int k = 0; k < PSCAN_ROWS; ++k) {
            const int d = d0 + k;
            if (d < d1) {
                const double y2 = y[d] * st[d];
                run = fma(hdt[d], y1 + y2, run);
                y1 = y2;
            }
            cum[k] = run;
        }
    }
    return run;
}

template <int TS, int TE>
__global__ void __launch_bounds__(PM_THREADS, 2) k_psf_mean(const double* __restrict__ pa,
                                                           const double* __restrict__ tab, int C, int E,
                                                           const double* __restrict__ ecb,
                                                           const double* __restrict__ wecb, int S,
                                                           const double* __restrict__ ltf,
                                                           const double* __restrict__ expo, double* __restrict__ upsf,
                                                           double* __restrict__ partial) {
    after_previous();
    extern __shared__ __align__(16) double psh[];
    constexpr int NW = PM_THREADS / 32;
    static_assert(NW % TE == 0 && (TS == 8 || TS == 4), "warps per energy, fragment rows");
    double* tile = psh;                       // [TS][TE][NDP]
    double* f0 = tile + TS * TE * NDP;        // [TS][TE] livetime factor / exposure
    double* f1 = f0 + TS * TE;                // [TS][TE] weighted factor / exposure
    double* part = f1 + TS * TE;              // [TE warps' shares][TS]: parts of the totals
    // livetime rows [2 TS][pitch] (weighted rows last, zeros past C), then the row tables
    double* sa = (double*)(((uintptr_t)(part + NW * TS) + 15) & ~(uintptr_t)15);
    double* st = sa;                          // [NDP] 2 pi sin(theta)
    double* hdt = st + NDP;                   // [NDP] half bin widths
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int s0 = blockIdx.y * TS, e0 = blockIdx.x * TE;
    const int ns = min(TS, S - s0), ne = min(TE, E - e0);
    const int KS = (C + 3) / 4, pitch = psf_row_pitch(C);
    double row_tab[(2 * NDP + PM_THREADS - 1) / PM_THREADS];
#pragma unroll
    for (int k = 0; k < (2 * NDP + PM_THREADS - 1) / PM_THREADS; ++k)
        if (t + k * PM_THREADS < 2 * NDP) row_tab[k] = __ldg(tab + t + k * PM_THREADS);
    for (int k = t; k < 2 * TS * pitch; k += PM_THREADS) {
        const int r = k / pitch, c = k - r * pitch, s = r % TS;
        sa[k] = s < ns && c < C ? (r < TS ? ecb : wecb)[(size_t)(s0 + s) * C + c] : 0.;
    }
    for (int k = t; k < TS * TE; k += PM_THREADS) {
        const int s = k / TE, e = k - s * TE;
        const bool ok = s < ns && e < ne;
        const double r = ok ? 1.0 / expo[(size_t)(s0 + s) * E + e0 + e] : 0.;
        f0[k] = ok ? ltf[e0 + e] * r : 0.;
        f1[k] = ok ? ltf[E + e0 + e] * r : 0.;
    }
    __syncthreads();
    {
        // fragments: lane holds A[lane / 4][lane % 4], B[lane % 4][lane / 4] and
        // C[lane / 4][2 (lane % 4) + {0, 1}]; M = 8 rows: 8 sources (livetime and weighted
        // livetime in two products) or 4 sources (both in one)
        constexpr int MT = TS == 8 ? 2 : 1, NT = (ND + 7) / 8;
        const int lr = lane >> 2, lk = lane & 3, el = warp % TE;  // a warp stays with one energy
        const char* pab = (const char*)pa;
        const double* arow = sa + lr * pitch + lk;
        unsigned off[PSF_KS];  // byte offsets of the lane's bins (past the end: the last, times zero)
        auto bins = [&](int k0) {
#pragma unroll
            for (int k = 0; k < PSF_KS; ++k) off[k] = (unsigned)min(4 * (k0 + k) + lk, C - 1) * (unsigned)(8 * E * NDP);
        };
        auto tile_off = [&](int i) { return 8u * (unsigned)((e0 + min(el, ne - 1)) * NDP + min(8 * i + lr, NDP - 1)); };
        const int q = (lr % TS) * TE + el, n = el < ne ? NT : 0;
        const double g0 = f0[q], g1 = f1[q];
        double b[PSF_KS], nb[PSF_KS], sum = 0.;
        bins(0);
        unsigned to = tile_off(warp / TE);
#pragma unroll
        for (int k = 0; k < PSF_KS; ++k) nb[k] = __ldg((const double*)(pab + (off[k] + to)));
        for (int i = warp / TE; i < n; i += NW / TE) {
            double acc[MT][2];
#pragma unroll
            for (int m = 0; m < MT; ++m) acc[m][0] = acc[m][1] = 0.;
            for (int k0 = 0; k0 < KS; k0 += PSF_KS) {
#pragma unroll
                for (int k = 0; k < PSF_KS; ++k) b[k] = nb[k];
                // the next k steps, or the next tile's first, in flight
                if (KS > PSF_KS) bins(k0 + PSF_KS < KS ? k0 + PSF_KS : 0);
                if (k0 + PSF_KS >= KS) to = tile_off(i + NW / TE);
#pragma unroll
                for (int k = 0; k < PSF_KS; ++k) nb[k] = __ldg((const double*)(pab + (off[k] + to)));
#pragma unroll
                for (int k = 0; k < PSF_KS; ++k)
#pragma unroll
                    for (int m = 0; m < MT; ++m) dmma(acc[m], arow[8 * m * pitch + 4 * (k0 + k)], b[k]);
            }
            const int d = 8 * i + 2 * lk;
            double w[2];
#pragma unroll
            for (int j = 0; j < 2; ++j)
                w[j] = MT == 2 ? acc[MT - 1][j] : __shfl_xor_sync(0xffffffffu, acc[0][j], 16);
            if (lr < TS && d < NDP) {
                const double2 h = __ldg((const double2*)(tab + 2 * NDP + d));
                const double2 u = make_double2(acc[0][0] * g0 + w[0] * g1, acc[0][1] * g0 + w[1] * g1);
                *(double2*)(tile + q * NDP + d) = u;
                sum = fma(h.x, u.x, sum);
                if (d + 1 < ND) sum = fma(h.y, u.y, sum);  // (rows from 401 on are padding, zeros)
            }
        }
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        if (lk == 0 && lr < TS) part[warp * TS + lr] = sum;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < (2 * NDP + PM_THREADS - 1) / PM_THREADS; ++k)
        if (t + k * PM_THREADS < 2 * NDP) st[t + k * PM_THREADS] = row_tab[k];
    if (t < TS * TE) {
        const int s = t / TE, el = t - s * TE;
        double tot = 0.;
        for (int w = el; w < NW; w += TE) tot += part[w * TS + s];
        f0[t] = tot;
        f1[t] = 1.0 / tot;  // +-inf when the total is 0: u / 0 as in the reference
    }
    __syncthreads();
    const int d0 = 1 + lane * PSCAN_ROWS, d1 = min(ND, d0 + PSCAN_ROWS);
    // write-out: a warp takes a third of a source's rows, a lane the energy lane % TE of
    // every RS-th row
    constexpr int RS = 32 / TE, PARTS = 3;
    const int wel = lane % TE, wd = lane / TE;
    auto write_out = [&](double* out, bool scaled) {
        for (int u = warp; u < TS * PARTS; u += NW) {
            const int s = u / PARTS, part = u - s * PARTS;
            if (s >= ns || wel >= ne) continue;
            const double* y = tile + (s * TE + wel) * NDP;
            const double f = scaled ? f1[s * TE + wel] : 1.0;
            double* o = out + ((size_t)(s0 + s) * ND) * E + e0 + wel;
#pragma unroll 4
            for (int d = wd + part * RS; d < ND; d += PARTS * RS) o[(size_t)d * E] = scaled ? y[d] * f : y[d];
        }
    };
    write_out(upsf, true);
    __syncthreads();
    for (int q = warp; q < TS * TE; q += NW) {
        const int s = q / TE, el = q - s * TE;
        if (s >= ns || el >= ne) continue;
        double* y = tile + q * NDP;
        double cum[PSCAN_ROWS];
        const double run = scan_run(y, st, hdt, d0, cum);
        double incl = run;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        const double before = incl - run, f = f0[q] != 0. ? f1[q] : 1.0;
        __syncwarp();  // every lane has read its run and the row before it
        if (lane == 0) y[0] = 0.0;
#pragma unroll
        for (int k = 0; k < PSCAN_ROWS; ++k)
            if (d0 + k < d1) y[d0 + k] = (before + cum[k]) * f;
    }
    __syncthreads();
    write_out(partial, false);
}

template <int TS, int TE>
static int launch_psf_mean(const PsfDev& a, const double* pa, const double* tab, cudaStream_t st) {
    const size_t smem = psf_mean_smem(TS, TE, a.C);
    if (smem > 48 * 1024)
        XTS_CUDA(cudaFuncSetAttribute(k_psf_mean<TS, TE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const dim3 g((a.E + TE - 1) / TE, (a.S + TS - 1) / TS);
    XTS_LAUNCH("k_psf_mean", st, launch_next(
                                     k_psf_mean<TS, TE>, g, PM_THREADS, smem, st, pa, tab, a.C, a.E, a.ecb, a.wecb, a.S,
                                     a.ltf, a.exposure, a.upsf, a.partial));
    return XTS_OK;
}

// The launches with caller-provided scratch: king holds both sides' King tables
// (401 * (Mc * Me front + Mc * Me back) doubles), pa the summed psf * aeff table
// (C * E * 404 doubles, 16-byte aligned), tab 3 * 404 doubles.  Nothing here allocates.
// With e, its exposure (the one that a.exposure points to) is formed beside the tables.
int launch_psf_scratch(const PsfDev& a, double* king, double* pa, double* tab, cudaStream_t st, const ExposureDev* e) {
    if (a.C > PSF_MAX_C) return set_error(XTS_ERR_ARG, "compute_psf_data: C=%d exceeds %d", a.C, PSF_MAX_C);
    if (a.E > PSF_MAX_E) return set_error(XTS_ERR_ARG, "compute_psf_data: E=%d exceeds %d", a.E, PSF_MAX_E);
    const int rc = launch_psf_tables(e, a, king, pa, tab, st);
    if (rc || a.S == 0) return rc;
    // 8 sources x 4 energies (most products per load of psf*aeff) where that fills the GPU
    // with two blocks per SM; 4 x 4 while two of three SMs get a block (50 sources x 37
    // energies: 130 blocks); below, one energy per block (7 x 21: 42 blocks instead of 12)
    int dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const long long e4 = (a.E + 3) / 4;
    if (e4 * ((a.S + 7) / 8) >= 2 * nsm) return launch_psf_mean<8, 4>(a, pa, tab, st);
    if (3 * e4 * ((a.S + 3) / 4) >= 2 * nsm) return launch_psf_mean<4, 4>(a, pa, tab, st);
    return launch_psf_mean<4, 1>(a, pa, tab, st);
}

int launch_psf(const PsfDev& a, cudaStream_t st, const ExposureDev* e) {
    double* king = (double*)workspace(W_KING, sizeof(double) * ND * ((size_t)a.pf.n_cos * a.pf.n_e +
                                                                     (size_t)a.pb.n_cos * a.pb.n_e));
    double* pa = (double*)workspace(W_PSFTAB, sizeof(double) * ((size_t)a.C * a.E + 4) * NDP);
    if (!king || !pa) return XTS_ERR_OOM;
    return launch_psf_scratch(a, king, pa + 4 * NDP, pa, st, e);
}

}  // namespace xts
