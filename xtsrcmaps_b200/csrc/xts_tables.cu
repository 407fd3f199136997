// xts_tables.cu -- steps (a) and (b) up to the mean PSF's contraction in two launches.
//
// The steps' tables are small (a few hundred thousand values) and form a chain of two
// links: the cos-theta bins, effective areas, livetime rows, King tables and integral row
// tables need only the inputs; the exposure contraction and psf*aeff need those.  Each link
// is one launch whose blocks are dealt out to its parts (six launches one after the other
// before: they cost the GPU about 10 us each in a small job, and the host 3).
#include "xts_tables.cuh"

namespace xts {

constexpr int TB = 128;  // threads per block

struct TablesArgs {
    ExposureDev e;
    xts_grid pf, pb;
    double *kf, *kb, *rows;
    int end[5];  // blocks up to and with: effective areas, livetime rows, King front, back, integral rows
};

__global__ void __launch_bounds__(TB) k_tables(const __grid_constant__ TablesArgs A) {
    const int b = blockIdx.x, t = threadIdx.x;
    let_next_start();
    if (b < A.end[0])
        exposure_table(b * TB + t, A.e.C, A.e.cosmin, A.e.thetabin, A.e.logEs, A.e.E, A.e.af, A.e.ab, A.e.exp_costhetas,
                       A.e.front_aeff, A.e.back_aeff);
    else if (b < A.end[1])
        src_cosbin((b - A.end[0]) * TB + t, A.e.src_sph, A.e.S, A.e.cube, A.e.wcube, A.e.nside, A.e.C, A.e.gathered,
                   A.e.ecb, A.e.wecb);
    else if (b < A.end[2]) king_entry((b - A.end[1]) * TB + t, A.pf, A.kf);
    else if (b < A.end[3]) king_entry((b - A.end[2]) * TB + t, A.pb, A.kb);
    else psf_row((b - A.end[3]) * TB + t, A.rows);
}

struct ContractArgs {
    const double *ecb, *wecb, *af, *ab, *ltf;
    double* exposure;
    int S, C, E, nb;  // nb: blocks of the exposure contraction, before those of psf*aeff
    xts_grid pf, pb;
    const double *kf, *kb, *costh, *logEs;
    double* pa;
};

__global__ void __launch_bounds__(TB) k_exposure_psf(const __grid_constant__ ContractArgs A) {
    const int b = blockIdx.x;
    after_previous();
    let_next_start();
    if (b < A.nb) exposure_value(b * TB + threadIdx.x, A.ecb, A.wecb, A.S, A.C, A.af, A.ab, A.ltf, A.E, A.exposure);
    else
        psf_aeff_block((b - A.nb) % A.E, (b - A.nb) / A.E, A.pf, A.pb, A.kf, A.kb, A.costh, A.C, A.logEs, A.E, A.af, A.ab,
                       A.pa);
}

static int blocks_of(long long n) { return (int)((n + TB - 1) / TB); }

// The first link: exposure's part (e) and mean PSF's (p), either may be missing.
static int launch_tables(const ExposureDev* e, const PsfDev* p, double* king, double* rows, cudaStream_t st) {
    TablesArgs A = {};
    int n = 0;
    if (e) A.e = *e;
    A.end[0] = n += e ? blocks_of((long long)e->C * e->E) : 0;
    A.end[1] = n += e ? blocks_of((long long)e->S * e->C) : 0;
    if (p) {
        const long long nf = (long long)ND * p->pf.n_cos * p->pf.n_e, nk = (long long)ND * p->pb.n_cos * p->pb.n_e;
        A.pf = p->pf;
        A.pb = p->pb;
        A.kf = king;
        A.kb = king + nf;
        A.rows = rows;
        A.end[2] = n += blocks_of(nf);
        A.end[3] = n += blocks_of(nk);
        A.end[4] = n += blocks_of(NDP);
    } else {
        A.end[2] = A.end[3] = A.end[4] = n;
    }
    if (n > 0) XTS_LAUNCH("k_tables", st, k_tables<<<n, TB, 0, st>>>(A));
    return XTS_OK;
}

static void exposure_args(ContractArgs& A, const double* ecb, const double* wecb, int S, int C, const double* af,
                          const double* ab, const double* ltf, int E, double* out) {
    A.ecb = ecb; A.wecb = wecb; A.S = S; A.C = C; A.af = af; A.ab = ab; A.ltf = ltf; A.E = E; A.exposure = out;
    A.nb = blocks_of((long long)S * E);
}

static void psf_args(ContractArgs& A, const PsfDev& p, const double* king, double* pa) {
    A.pf = p.pf; A.pb = p.pb;
    A.kf = king;
    A.kb = king + (size_t)ND * p.pf.n_cos * p.pf.n_e;
    A.costh = p.costh; A.logEs = p.logEs; A.af = p.af; A.ab = p.ab; A.C = p.C; A.E = p.E;
    A.pa = pa;
}

int launch_exposure_contract(const double* ecb, const double* wecb, int S, int C, const double* af, const double* ab,
                             const double* ltf, int E, double* out, cudaStream_t st) {
    if ((long long)S * E == 0) return XTS_OK;
    ContractArgs A = {};
    exposure_args(A, ecb, wecb, S, C, af, ab, ltf, E, out);
    XTS_LAUNCH("k_exposure_f64", st, launch_next(k_exposure_psf, A.nb, TB, 0, st, A));
    return XTS_OK;
}

int launch_exposure(const ExposureDev& a, cudaStream_t st) {
    const int rc = launch_tables(&a, nullptr, nullptr, nullptr, st);
    return rc ? rc : launch_exposure_contract(a.ecb, a.wecb, a.S, a.C, a.front_aeff, a.back_aeff, a.ltf, a.E, a.exposure, st);
}

// The King tables, the integral's row tables and psf*aeff of the mean PSF (xts_psf.cu), and
// with e the exposure that it divides by.
int launch_psf_tables(const ExposureDev* e, const PsfDev& p, double* king, double* pa, double* rows, cudaStream_t st) {
    const int rc = launch_tables(e, &p, king, rows, st);
    if (rc) return rc;
    ContractArgs A = {};
    psf_args(A, p, king, pa);
    if (e) exposure_args(A, e->ecb, e->wecb, e->S, e->C, e->front_aeff, e->back_aeff, e->ltf, e->E, e->exposure);
    XTS_LAUNCH("k_exposure_psf", st, launch_next(k_exposure_psf, A.nb + p.E * p.C, TB, 0, st, A));
    return XTS_OK;
}

}  // namespace xts
