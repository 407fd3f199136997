// xts_exposure_tc.cu -- the full-sky exposure contraction on tcgen05 tensor
// cores: for every HEALPix pixel p of the livetime cube,
//     expo[p][e] = L0[e] sum_c X[p][c] A[c][e] + L1[e] sum_c Wt[p][c] A[c][e]
// with X, Wt the livetime and weighted-livetime rows [12 nside^2, C], A the
// summed front and back effective area [C, E] (the back side uses the front
// livetime-efficiency factors, psf.psf_lookup_table_and_partial_integrals.cxx:151-156
// and exposure/exposure.cxx:159-263) and L0, L1 = front_LTF [2, E].  A source's
// exposure (Exposure::exposure) is the row of this map at the source's NESTED
// pixel (exposure/exposure.cxx:42-63).
//
// One GEMM: M = pixels, K = [X | Wt] (each half zero-padded from C to whole boxes of 32 by
// the TMA fill), N = E in groups of 64, B = [A L0 ; A L1] prepared once (K-major) as TF32
// hi and lo parts.  One persistent block per SM holds its group's B in shared memory and
// takes tiles of 128 pixels; the tile's halves go through a two-stage ring:
//   control warp   TMA of the next half's raw FP32 rows (128-byte swizzle) while this one
//                  is split and multiplied; tcgen05.mma.kind::tf32 for A_lo B_hi + A_hi
//                  B_lo + A_hi B_hi (3xTF32, small terms first) per 8 bins that hold any,
//                  into one of two FP32 accumulators in tensor memory;
//   split warps    each raw element in place into hi = tf32(x), lo = x - hi beside it
//                  (same byte positions, so the swizzle needs no handling; a lane takes
//                  the 16-byte units of its row in swizzled order, free of bank conflicts);
//   epilogue warps the previous tile's accumulator through an odd-pitch stage into FP64
//                  rows with coalesced stores.
// nside 256, C = 40, E = 50 (566 MB): 175 us = 0.50 of the measured copy bandwidth (with a
// block per 74 KB of shared memory running its K boxes one after the other and B loaded
// with each: 557 us).  The ring bounds it: without the products, the split or the write-out
// 152, 155 or 150 us; prefetching the rows into L2 changes nothing.  The products and their
// order are those of the earlier form, so the map's bits are too.
// Every mbarrier wait is bounded; a timeout sets the status word, lets in-flight
// copies and MMAs land (bounded), frees tensor memory and returns.
#include <cuda.h>

#include "xts_point.cuh"

namespace xts {

constexpr int XM = 128;  // pixels per tile == MMA M
constexpr int XK = 32;   // floats per K box (one 128-byte swizzle atom)
constexpr int XKP = 64;  // padded K of each half (livetime, weighted livetime)
constexpr int XN = 64;   // energies per group
constexpr int XBOX = XM * XK * 4, XBBOX = XN * XK * 4;  // bytes of an A and a B box
constexpr int X_SPLIT = 256;                            // threads of the split warps
constexpr int X_THREADS = 128 + X_SPLIT + 32;           // epilogue, split, control
constexpr int XPITCH = XN + 1;                          // floats per stage row

// Shared memory: two stages of [2 boxes hi][2 boxes lo], B [hi, lo][4 boxes], the epilogue
// stage [128][XPITCH], barriers.
constexpr size_t X_B = 2 * 4 * (size_t)XBOX;
constexpr size_t X_STAGE = X_B + 8 * (size_t)XBBOX;
constexpr size_t X_BARS = X_STAGE + sizeof(float) * XM * XPITCH;
constexpr size_t X_TOTAL = X_BARS + 128;

static __device__ __forceinline__ unsigned long long x_desc(unsigned addr) {
    // K-major, 128-byte swizzle: start >> 4, LBO 16 >> 4, SBO 1024 >> 4 (8-row groups), version 1
    return (unsigned long long)((addr >> 4) & 0x3FFF) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}

// D f32, A/B tf32, both K-major, M = 128, N.
static __host__ __device__ constexpr unsigned x_idesc(int N) {
    return (1u << 4) | (2u << 7) | (2u << 10) | ((unsigned)(N >> 3) << 17) | ((unsigned)(XM >> 4) << 24);
}

static __device__ __forceinline__ float tf32_hi(float v) {
    unsigned r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(v));
    return __uint_as_float(r);
}

static __device__ __forceinline__ void x_load(unsigned dst, const CUtensorMap* m, int x, int y, unsigned bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 :: "r"(dst), "l"((unsigned long long)m), "r"(x), "r"(y), "r"(bar) : "memory");
}
static __device__ __forceinline__ void x_expect(unsigned bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(bar), "r"(bytes) : "memory");
}
static __device__ __forceinline__ void x_arrive(unsigned bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(bar) : "memory");
}
static __device__ __forceinline__ void x_mma(unsigned d, unsigned long long a, unsigned long long b, unsigned idesc,
                                             unsigned acc) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}\n"
                 :: "r"(d), "l"(a), "l"(b), "r"(idesc), "r"(acc), "r"(0u));
}
static __device__ __forceinline__ void x_commit(unsigned bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(bar) : "memory");
}

__global__ void __launch_bounds__(X_THREADS, 1)
k_exposure_map_tc(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_w,
                  const __grid_constant__ CUtensorMap tm_bhi, const __grid_constant__ CUtensorMap tm_blo,
                  int npix, int C, int E, int groups, double* __restrict__ out, int* __restrict__ status) {
    after_previous();
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
    unsigned long long* bars = (unsigned long long*)(smem + X_BARS);
    unsigned* tmem_slot = (unsigned*)(smem + X_BARS + 96);
    volatile int* abort_flag = (volatile int*)(smem + X_BARS + 104);
    // per stage: rows landed, rows split, MMAs done; per accumulator: complete, read; B landed
    const unsigned full0 = smem_u32(bars), split0 = full0 + 16, done0 = full0 + 32, accf0 = full0 + 48,
                   acce0 = full0 + 64, bbar = full0 + 80;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    if (t == 0) {
        for (int k = 0; k < 2; ++k) {
            mbar_init(full0 + 8 * k, 1);
            mbar_init(split0 + 8 * k, X_SPLIT);
            mbar_init(done0 + 8 * k, 1);
            mbar_init(accf0 + 8 * k, 1);
            mbar_init(acce0 + 8 * k, 4);
        }
        mbar_init(bbar, 1);
        *abort_flag = 0;
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     :: "r"(smem_u32(tmem_slot)), "r"(2u * XN));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned tmem = *tmem_slot;

    const int group = blockIdx.x % groups, e0 = group * XN, ne = min(XN, E - e0);
    const int N = (ne + 15) / 16 * 16;
    const int ntiles = (npix + XM - 1) / XM, first = blockIdx.x / groups;
    const int step = ((int)gridDim.x - group + groups - 1) / groups;  // blocks of this group
    const int mine = first < ntiles ? (ntiles - first + step - 1) / step : 0;
    const int nbox = (C + XK - 1) / XK;                       // boxes per half that hold bins
    const int nks[2] = {(min(C, XK) + 7) / 8, nbox > 1 ? (C - XK + 7) / 8 : 0};  // their steps of 8 bins
    bool ok = true;
    auto wait = [&](unsigned bar, unsigned parity) {
        if (*abort_flag || !mbar_wait(bar, parity)) {
            *abort_flag = 1;
            ok = false;
        }
        return ok;
    };

    if (warp == X_THREADS / 32 - 1) {  // control
        if (lane == 0 && mine > 0) {
            const unsigned base = smem_u32(smem);
            x_expect(bbar, 8u * XBBOX);
            for (int k = 0; k < 4; ++k) {
                x_load(base + X_B + k * XBBOX, &tm_bhi, XK * k, e0, bbar);
                x_load(base + X_B + (4 + k) * XBBOX, &tm_blo, XK * k, e0, bbar);
            }
            const int n = 2 * mine;  // halves
            int loaded = 0;
            auto load = [&](int u) {
                const int st = u & 1, tile = first + (u >> 1) * step;
                if (u >= 2 && !wait(done0 + 8 * st, ((u >> 1) - 1) & 1)) return;
                x_expect(full0 + 8 * st, (unsigned)(nbox * XBOX));
                for (int b = 0; b < nbox; ++b)
                    x_load(base + (4 * st + b) * XBOX, (u & 1) ? &tm_w : &tm_x, XK * b, tile * XM, full0 + 8 * st);
                loaded = u + 1;
            };
            load(0);
            wait(bbar, 0);
            int issued = 0;
            for (int u = 0; u < n && ok; ++u) {
                const int st = u & 1, i = u >> 1, ab = i & 1, half = u & 1;
                if (u + 1 < n) load(u + 1);
                if (!ok || !wait(split0 + 8 * st, i & 1)) break;
                if (half == 0 && i >= 2 && !wait(acce0 + 8 * ab, ((i >> 1) - 1) & 1)) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const unsigned idesc = x_idesc(N), d = tmem + (unsigned)(ab * XN);
                for (int b = 0; b < nbox; ++b) {
                    const unsigned a_hi = base + (4 * st + b) * XBOX, a_lo = a_hi + 2 * XBOX;
                    const unsigned b_hi = base + X_B + (2 * half + b) * XBBOX, b_lo = b_hi + 4 * XBBOX;
                    // a step of 8 bins is 32 bytes on: 2 in the descriptors' start address
                    unsigned long long ah = x_desc(a_hi), al = x_desc(a_lo), bh = x_desc(b_hi), bl = x_desc(b_lo);
#pragma unroll
                    for (int ks = 0; ks < XK / 8; ++ks, ah += 2, al += 2, bh += 2, bl += 2) {
                        if (ks >= nks[b]) break;
                        x_mma(d, al, bh, idesc, (half > 0 || b > 0 || ks > 0) ? 1u : 0u);
                        x_mma(d, ah, bl, idesc, 1u);
                        x_mma(d, ah, bh, idesc, 1u);
                    }
                }
                x_commit(done0 + 8 * st);
                if (half == 1) x_commit(accf0 + 8 * ab);
                issued = u + 1;
            }
            if (!ok) {  // bounded: let the copies and MMAs in flight land before the block exits
                mbar_wait(bbar, 0);
                if (loaded > 0) mbar_wait(full0 + 8 * ((loaded - 1) & 1), ((loaded - 1) >> 1) & 1);
                if (loaded > 1) mbar_wait(full0 + 8 * ((loaded - 2) & 1), ((loaded - 2) >> 1) & 1);
                if (issued > 0) mbar_wait(done0 + 8 * ((issued - 1) & 1), ((issued - 1) >> 1) & 1);
            }
        }
        __syncwarp();
    } else if (warp >= 4) {  // split: two threads per pixel row, alternate 16-byte units
        const int row = (t - 128) & (XM - 1), part = (t - 128) >> 7;
        for (int u = 0; u < 2 * mine && ok; ++u) {
            const int st = u & 1;
            if (!wait(full0 + 8 * st, (u >> 1) & 1)) break;
            for (int b = 0; b < nbox; ++b) {
                float4* ah = (float4*)(smem + (4 * st + b) * XBOX + row * 128);
                float4* al = (float4*)((unsigned char*)ah + 2 * XBOX);
#pragma unroll 4
                for (int j = part; j < 2 * nks[b]; j += 2) {
                    const int k = j ^ (row & 7);
                    const float4 v = ah[k];
                    const float4 h = make_float4(tf32_hi(v.x), tf32_hi(v.y), tf32_hi(v.z), tf32_hi(v.w));
                    ah[k] = h;
                    al[k] = make_float4(v.x - h.x, v.y - h.y, v.z - h.z, v.w - h.w);
                }
            }
            fence_async_shared();
            x_arrive(split0 + 8 * st);
        }
    } else {  // epilogue: warp w the pixels 32 w .. of each tile
        float* stage = (float*)(smem + X_STAGE) + warp * 32 * XPITCH;
        for (int i = 0; i < mine && ok; ++i) {
            const int ab = i & 1, p0 = (first + i * step) * XM + warp * 32;
            const bool got = wait(accf0 + 8 * ab, (i >> 1) & 1);
            if (!__all_sync(0xffffffffu, got)) { ok = false; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            for (int c0 = 0; c0 < N; c0 += 16) {
                unsigned v[16];
                const unsigned taddr = tmem + ((unsigned)(warp * 32) << 16) + (unsigned)(ab * XN + c0);
                asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                             : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                               "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                             : "r"(taddr));
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int j = 0; j < 16; ++j) stage[lane * XPITCH + c0 + j] = __uint_as_float(v[j]);
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) x_arrive(acce0 + 8 * ab);
            const int rows = min(32, npix - p0);
            double* dst = out + (long long)p0 * E + e0;
#pragma unroll 4
            for (int r = 0; r < rows; ++r) {
                if (lane < ne) dst[(long long)r * E + lane] = (double)stage[r * XPITCH + lane];
                if (lane + 32 < ne) dst[(long long)r * E + lane + 32] = (double)stage[r * XPITCH + lane + 32];
            }
            __syncwarp();
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (t == 0 && *abort_flag) atomicExch(status, 1);
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(2u * XN));
}

// B = [A L0 ; A L1] as TF32 hi and lo, [N][2 * XKP] (K contiguous); rows past E,
// and the padding columns of each half, are zero.
__global__ void k_exposure_b(const double* af, const double* ab, const double* ltf, int C, int E, int N,
                             float* bhi, float* blo) {
    after_previous();
    let_next_start();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= N * 2 * XKP) return;
    const int e = k / (2 * XKP), kk = k - e * (2 * XKP);
    const int half = kk / XKP, c = kk - half * XKP;
    double v = 0.;
    if (e < E && c < C) v = (af[(size_t)c * E + e] + ab[(size_t)c * E + e]) * ltf[(size_t)half * E + e];
    const float f = (float)v;
    const float h = tf32_hi(f);
    bhi[k] = h;
    blo[k] = f - h;
}

typedef CUresult (*XEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                              const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                              CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static XEncodeFn x_encode() {
    static XEncodeFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (XEncodeFn)p;
        else
            cudaGetLastError();
    }
    return fn;
}

// 2-D FP32 map [rows][cols], boxes of 32 columns x box_rows rows, 128-byte swizzle;
// columns past `cols` and rows past `rows` read as zeros.
static int x_map(CUtensorMap* m, const float* base, long long rows, int cols, int box_rows) {
    XEncodeFn fn = x_encode();
    if (!fn) return set_error(XTS_ERR_CUDA, "cuTensorMapEncodeTiled is not available");
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)cols * 4};
    cuuint32_t box[2] = {(cuuint32_t)XK, (cuuint32_t)box_rows};
    cuuint32_t es[2] = {1, 1};
    CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, (void*)base, dims, strides, box, es,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return set_error(XTS_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
    return XTS_OK;
}

bool exposure_map_supported(int C, int E) { return C >= 1 && C <= XKP && (C * 4) % 16 == 0 && E >= 1 && E <= 256; }

int launch_exposure_map_tc(const float* cube, const float* wcube, long long npix, int C, const double* front_aeff,
                           const double* back_aeff, const double* ltf, int E, double* out, int* status,
                           cudaStream_t st) {
    if (!exposure_map_supported(C, E))
        return set_error(XTS_ERR_ARG, "exposure map: needs C <= 64 with 16-byte rows (C %% 4 == 0) and E <= 256");
    if (npix > 0x7fffffffLL) return set_error(XTS_ERR_ARG, "exposure map: too many pixels");
    const int N = (E + 15) / 16 * 16;
    float* b = (float*)workspace(W_MISC2, sizeof(float) * 2 * (size_t)N * 2 * XKP + 64);
    if (!b) return XTS_ERR_OOM;
    float* bhi = b;
    float* blo = b + (size_t)N * 2 * XKP;
    const int nb = N * 2 * XKP;
    XTS_LAUNCH("k_exposure_b", st, launch_next(k_exposure_b, (nb + 255) / 256, 256, 0, st, front_aeff, back_aeff, ltf,
                                               C, E, N, bhi, blo));
    CUtensorMap mx, mw, mbh, mbl;
    int rc;
    if ((rc = x_map(&mx, cube, npix, C, XM))) return rc;
    if ((rc = x_map(&mw, wcube, npix, C, XM))) return rc;
    if ((rc = x_map(&mbh, bhi, N, 2 * XKP, XN))) return rc;
    if ((rc = x_map(&mbl, blo, N, 2 * XKP, XN))) return rc;
    const size_t smem = X_TOTAL + 1024;
    XTS_CUDA(cudaFuncSetAttribute(k_exposure_map_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const int groups = (E + XN - 1) / XN;  // at most 4, fewer than SMs
    const long long items = (npix + XM - 1) / XM * groups;
    const int G = (int)(items < nsm ? items : nsm);
    XTS_LAUNCH("k_exposure_map_tc", st, launch_next(k_exposure_map_tc, G, X_THREADS, smem, st, mx, mw, mbh, mbl, (int)npix,
                                                    C, E, groups, out, status));
    return XTS_OK;
}

}  // namespace xts
