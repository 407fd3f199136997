// xts_mlp.cu -- the surrogate network of the pixel cubature: a 5 -> 128 -> 128 ->
// 128 -> 1 perceptron with tanh-form GELU (Hendrycks & Gimpel, "Gaussian Error
// Linear Units", 2016: gelu(z) = z/2 (1 + tanh(sqrt(2/pi) (z + 0.044715 z^3)))),
// its forward pass, its gradient and an Adam update (Kingma & Ba, 2015).
//
// The three hidden layers run on tcgen05 tensor cores: BF16 operands in shared
// memory (K-major, 128-byte swizzle: a [128 rows][64] BF16 atom is 16 KB, rows
// of 128 bytes whose 16-byte chunks are permuted by row & 7, 8-row groups 1024
// bytes apart), one thread issuing tcgen05.mma.kind::f16 (M = N = 128, K = 16)
// into an FP32 accumulator of 128 tensor-memory columns, the four warps reading
// it back with tcgen05.ld (warp w owns lanes 32w..32w+31 = rows of the tile).
//
//   * k_mlp_forward: one tile of 128 rows per step of a persistent loop, two
//     blocks of two warpgroups per SM (each row's 128 columns split between two
//     threads).  Layer 1 (K = 5) is one K = 16 MMA over the features split into
//     three BF16 terms; the GELUs run on CUDA cores; each hidden layer's BF16
//     activations are written by their row's threads straight into the swizzled
//     A operand of the next MMA; the output layer is a per-row dot product.
//   * k_mlp_gradient: forward and backward pass of a training batch in one kernel, the
//     hidden weights' gradients accumulated in tensor memory.
//   * k_gemm_bf16: C = A B^T, with either operand given transposed (gathered into the
//     swizzled layout by the loading threads), a two-stage shared-memory ring and
//     split-K whose partial tiles are summed in a fixed order (k_sum_splits).
//   * k_mlp_grad_sum: k_mlp_gradient's partials summed in a fixed order, so training is
//     reproducible.
//   * k_mlp_adam: the update of the FP32 master parameters and the BF16 copies.
//
// Every mbarrier wait is bounded (WAIT_LIMIT polls); a timeout sets the status
// word, stops issuing work, lets issued MMAs complete (bounded) and frees the
// tensor memory.
#include <cuda_bf16.h>

#include "xts_point.cuh"

namespace xts {

constexpr int MH = XTS_MLP_HID;  // hidden width == MMA N
constexpr int MI = XTS_MLP_IN;
constexpr int MT = 128;          // rows per tile == MMA M == threads per block
constexpr int ATOM = 16384;      // bytes of a [128][64] BF16 swizzled atom

static_assert(MH == 128 && MT == 128, "the MMA shapes below assume 128 x 128 tiles");

struct MlpNorm {
    float mu[MI], sd[MI], out_mu, out_sd;
};

static MlpNorm mlp_norm(const xts_mlp* net) {
    MlpNorm m;
    for (int k = 0; k < MI; ++k) { m.mu[k] = net->in_mu[k]; m.sd[k] = net->in_sd[k]; }
    m.out_mu = net->out_mu;
    m.out_sd = net->out_sd;
    return m;
}

__device__ __forceinline__ float tanh_fast(float x) {
    float r;
    asm("tanh.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
constexpr float GK0 = 0.7978845608028654f;   // sqrt(2 / pi)
constexpr float GK1 = 0.035677408136300125f; // sqrt(2 / pi) * 0.044715
// the tanh argument sqrt(2/pi) (z + 0.044715 z^3) as z (GK0 + GK1 z^2): two multiplies and
// one FMA
__device__ __forceinline__ float gelu_arg(float z) { return z * fmaf(z * z, GK1, GK0); }
__device__ __forceinline__ float gelu(float z) {
    return 0.5f * z * (1.f + tanh_fast(gelu_arg(z)));
}
__device__ __forceinline__ float2 gelu_arg2(float2 z) {
    return __fmul2_rn(z, __ffma2_rn(__fmul2_rn(z, z), make_float2(GK1, GK1), make_float2(GK0, GK0)));
}
// two GELUs with packed FP32 arithmetic (same formula as gelu, rounding order differs)
__device__ __forceinline__ float2 gelu2(float2 z) {
    const float2 u = gelu_arg2(z);
    const float2 hz = __fmul2_rn(make_float2(0.5f, 0.5f), z);
    return __ffma2_rn(hz, make_float2(tanh_fast(u.x), tanh_fast(u.y)), hz);
}
// 2 gelu(z) for two values: the same rounding as gelu2 scaled by 2 (exact), one
// multiply fewer; the inference kernel halves the next layer's weights to match
__device__ __forceinline__ float2 gelu2x(float2 z) {
    const float2 u = gelu_arg2(z);
    return __ffma2_rn(z, make_float2(tanh_fast(u.x), tanh_fast(u.y)), z);
}
__device__ __forceinline__ float gelu_grad(float z) {
    const float z2 = z * z, th = tanh_fast(z * fmaf(z2, GK1, GK0));
    return 0.5f * (1.f + th) + 0.5f * z * (1.f - th * th) * fmaf(3.f * GK1, z2, GK0);
}

// byte offset of element (r, k) of a [128][K] BF16 operand made of [128][64] atoms
__device__ __forceinline__ unsigned sw_off(int r, int k) {
    return (unsigned)((k >> 6) * ATOM + r * 128 + ((((k & 63) >> 3) ^ (r & 7)) << 4) + (k & 7) * 2);
}

static __device__ __forceinline__ unsigned long long m_desc(unsigned addr) {
    // K-major, 128-byte swizzle: start >> 4, LBO 16 >> 4, SBO 1024 >> 4 (8-row groups), version 1
    return (unsigned long long)((addr >> 4) & 0x3FFF) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}

// D f32, A and B bf16, both K-major, M = 128, N = 128.
constexpr unsigned M_IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(MH >> 3) << 17) |
                             ((unsigned)(MT >> 4) << 24);

// K = 16 * nk of one MMA chain; a, b: shared addresses of the operands (atoms
// 16 KB apart); acc0: accumulate onto D from the first step.
__device__ __forceinline__ void mma_chain(unsigned tmem, unsigned a, unsigned b, int nk, bool acc0) {
    for (int ks = 0; ks < nk; ++ks) {
        const unsigned off = (unsigned)((ks >> 2) * ATOM + (ks & 3) * 32);
        const unsigned long long da = m_desc(a + off), db = m_desc(b + off);
        const unsigned acc = (acc0 || ks > 0) ? 1u : 0u;
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                     "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}\n"
                     :: "r"(tmem), "l"(da), "l"(db), "r"(M_IDESC), "r"(acc), "r"(0u));
    }
}

// K-major without swizzle (layer 1's W1 operand, K = 16): core matrices of 8 rows x 16
// bytes, the two along K (leading byte offset) 128 bytes apart, 8-row groups (stride
// byte offset) 256 bytes apart; version 1, layout type 0
static __device__ __forceinline__ unsigned long long m_desc_ns(unsigned addr) {
    return (unsigned long long)((addr >> 4) & 0x3FFF) | ((unsigned long long)(128 >> 4) << 16) |
           ((unsigned long long)(256 >> 4) << 32) | (1ull << 46);
}
// byte offset of element (r, k) of that [128][16] BF16 operand
__device__ __forceinline__ unsigned ns_off(int r, int k) {
    return (unsigned)((r >> 3) * 256 + (k >> 3) * 128 + (r & 7) * 16 + (k & 7) * 2);
}
constexpr int W1OP = MH * 16 * 2;  // bytes of the W1 operand

// Layer 1 on the tensor cores.  A row of A holds the standardised features split into
// three BF16 terms, x = hi + mid + lo (each difference exact in FP32, so the sum
// equals x to 2^-27 relative), at K = 0..4, 5..9, 10..14; B holds W1 (already BF16)
// three times over, so one K = 16 MMA forms W1 x with every product exact.
__device__ __forceinline__ void fill_w1_operand(unsigned char* dst, const float* params, int t, int nt) {
    for (int e = t; e < MH * 16; e += nt) {
        const int j = e >> 4, k = e & 15;
        const __nv_bfloat16 w = k < 3 * MI ? __float2bfloat16_rn(params[XTS_MLP_W1 + j * MI + k % MI])
                                           : __float2bfloat16_rn(0.f);
        *reinterpret_cast<__nv_bfloat16*>(dst + ns_off(j, k)) = w;
    }
}
__device__ __forceinline__ void split_x(const float* x, uint4* q) {
    unsigned short e[16];
#pragma unroll
    for (int k = 0; k < MI; ++k) {
        const __nv_bfloat16 hi = __float2bfloat16_rn(x[k]);
        const float r1 = x[k] - __bfloat162float(hi);
        const __nv_bfloat16 mid = __float2bfloat16_rn(r1);
        const __nv_bfloat16 lo = __float2bfloat16_rn(r1 - __bfloat162float(mid));
        e[k] = __bfloat16_as_ushort(hi);
        e[MI + k] = __bfloat16_as_ushort(mid);
        e[2 * MI + k] = __bfloat16_as_ushort(lo);
    }
    e[15] = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        reinterpret_cast<unsigned*>(q)[i] = (unsigned)e[2 * i] | ((unsigned)e[2 * i + 1] << 16);
    }
}
__device__ __forceinline__ void store_x_split(unsigned char* act, int r, const float* x) {
    uint4 q[2];
    split_x(x, q);
    *reinterpret_cast<uint4*>(act + sw_off(r, 0)) = q[0];
    *reinterpret_cast<uint4*>(act + sw_off(r, 8)) = q[1];
}
__device__ __forceinline__ void store_x_split_ns(unsigned char* op, int r, const float* x) {
    uint4 q[2];
    split_x(x, q);
    *reinterpret_cast<uint4*>(op + ns_off(r, 0)) = q[0];
    *reinterpret_cast<uint4*>(op + ns_off(r, 8)) = q[1];
}
// the layer-1 MMA: A = K columns 0..15 of the swizzled activation operand, B = W1
__device__ __forceinline__ void mma_layer1(unsigned tmem, unsigned a, unsigned w1op) {
    const unsigned long long da = m_desc(a), db = m_desc_ns(w1op);
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}\n"
                 :: "r"(tmem), "l"(da), "l"(db), "r"(M_IDESC), "r"(0u), "r"(0u));
}

__device__ __forceinline__ void mma_commit(unsigned bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(bar) : "memory");
}

// 16 accumulator columns c0..c0+15 of this thread's row
__device__ __forceinline__ void tmem_ld16(unsigned taddr, float* v) {
    unsigned r[16];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
}

// the same load without its wait, for a load kept in flight while other columns are
// worked on; tmem_ld_done waits for every load issued so far and ties r to that wait
__device__ __forceinline__ void tmem_ld16_issue(unsigned taddr, unsigned* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_done(unsigned* r) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    // no use of r may be moved above the wait
    asm volatile("" : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                      "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]));
}

__device__ __forceinline__ unsigned pack_bf16(float a, float b) {
    const __nv_bfloat162 p = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const unsigned*>(&p);
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ unsigned tmem_alloc(unsigned slot_addr, unsigned ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(slot_addr), "r"(ncols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    return 0;
}
__device__ __forceinline__ void tmem_free(unsigned tmem, unsigned ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(ncols));
}

// ====================================================================== forward
constexpr int FT = 2 * MT;  // forward threads: two warpgroups, each row's 128 columns split in halves

struct FwdLayout {
    static constexpr size_t w2 = 0, w3 = 2 * ATOM, act = 4 * ATOM, w1 = 6 * ATOM;
    // b1, b2, b3, w4 [128 each], b4 (+3), partial y [128]
    static constexpr size_t f32 = w1 + W1OP;
    static constexpr size_t bars = f32 + 4 * (4 * MH + 4 + MT);
    static constexpr size_t total = bars + 64;
};
constexpr size_t FWD_SMEM = FwdLayout::total + 1024;

// Thread t works on row r = t & 127 of the tile and hidden columns [64 hf, 64 hf + 64),
// hf = t >> 7: warp w reads tensor-memory lanes 32 (w & 3).. and, in the A operand,
// writes the [128][64] atom hf of its rows.  All three layers run on the tensor cores
// (layer 1 as one K = 16 MMA over the split features); the GELUs on CUDA cores.
__global__ void __launch_bounds__(FT, 2)
k_mlp_forward(const float* __restrict__ params, const __nv_bfloat16* __restrict__ wbf, MlpNorm nm,
              const float* __restrict__ X, long long n, const unsigned long long* __restrict__ n_dev,
              long long ldx, float* __restrict__ y, int* __restrict__ status) {
    if (n_dev) n = min(n, (long long)*n_dev);  // rows counted on the device (at most n)
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
    const int t = threadIdx.x, warp = t >> 5, r = t & (MT - 1), hf = t >> 7, cb = 64 * hf;
    float* b1 = (float*)(smem + FwdLayout::f32);
    float* b2 = b1 + MH;
    float* b3 = b2 + MH;
    float* w4 = b3 + MH;
    float* b4 = w4 + MH;
    float* ypart = b4 + 4;
    unsigned long long* bars = (unsigned long long*)(smem + FwdLayout::bars);
    unsigned* tmem_slot = (unsigned*)(smem + FwdLayout::bars + 32);
    const unsigned bar = smem_u32(&bars[0]);
    const unsigned s_w2 = smem_u32(smem + FwdLayout::w2), s_w3 = smem_u32(smem + FwdLayout::w3);
    const unsigned s_w1 = smem_u32(smem + FwdLayout::w1);
    const unsigned s_act = smem_u32(smem + FwdLayout::act);

    // weights: W2, W3 [out][in] BF16 -> swizzled B operands (row = out, K = in)
    for (int idx = t; idx < 2 * MH * (MH / 8); idx += FT) {
        const int l = idx / (MH * (MH / 8)), rem = idx - l * (MH * (MH / 8));
        const int row = rem >> 4, ch = rem & 15;
        const uint4 v = *reinterpret_cast<const uint4*>(wbf + (size_t)l * MH * MH + row * MH + ch * 8);
        *reinterpret_cast<uint4*>(smem + (l ? FwdLayout::w3 : FwdLayout::w2) + sw_off(row, ch * 8)) = v;
    }
    fill_w1_operand(smem + FwdLayout::w1, params, t, FT);
    for (int k = t; k < MH; k += FT) {
        b1[k] = params[XTS_MLP_B1 + k];
        b2[k] = params[XTS_MLP_B2 + k];
        b3[k] = params[XTS_MLP_B3 + k];
        w4[k] = __bfloat162float(__float2bfloat16_rn(params[XTS_MLP_W4 + k]));
    }
    if (t == 0) {
        b4[0] = params[XTS_MLP_B4];
        mbar_init(bar, 1);
    }
    if (warp == 0) tmem_alloc(smem_u32(tmem_slot), 128);
    fence_async_shared();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = *tmem_slot;
    const unsigned trow = tmem + ((unsigned)((warp & 3) * 32) << 16) + (unsigned)cb;
    unsigned ph = 0;
    bool ok = true;
    const long long ntiles = (n + MT - 1) / MT;
    for (long long tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x) {
        const long long row = tile * MT + r;
        const bool live = row < n;
        // layer 1's A operand (the accumulator's last reader, the previous tile's
        // epilogue, has finished: the barrier below orders it before the MMA)
        if (!hf) {
            float x[MI];
#pragma unroll
            for (int k = 0; k < MI; ++k)
                x[k] = live ? (X[ldx ? k * ldx + row : row * MI + k] - nm.mu[k]) / nm.sd[k] : 0.f;
            store_x_split(smem + FwdLayout::act, r, x);
        }
        float yacc = 0.f;
        for (int layer = 1; layer <= 3 && ok; ++layer) {
            fence_async_shared();
            tc_fence_before();
            __syncthreads();
            if (t == 0) {
                tc_fence_after();
                if (layer == 1) mma_layer1(tmem, s_act, s_w1);
                else mma_chain(tmem, s_act, layer == 2 ? s_w2 : s_w3, MH / 16, false);
                mma_commit(bar);
            }
            const bool got = mbar_wait(bar, ph);
            if (!__syncthreads_and(got)) { ok = false; break; }  // ph stays: the exit path waits on it
            ph ^= 1;
            tc_fence_after();
            const float* bias = layer == 1 ? b1 : layer == 2 ? b2 : b3;
            for (int c0 = 0; c0 < 64; c0 += 16) {
                float v[16], bv[16];
                tmem_ld16(trow + (unsigned)c0, v);
                const int cc = cb + c0;
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float4 b = reinterpret_cast<const float4*>(bias + cc)[q];
                    bv[4 * q] = b.x; bv[4 * q + 1] = b.y; bv[4 * q + 2] = b.z; bv[4 * q + 3] = b.w;
                }
#pragma unroll
                for (int j = 0; j < 16; j += 2) {
                    const float2 z = __fadd2_rn(make_float2(v[j], v[j + 1]), make_float2(bv[j], bv[j + 1]));
                    const float2 g2 = gelu2(z);
                    v[j] = g2.x;
                    v[j + 1] = g2.y;
                }
                if (layer < 3) {
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        const float* u = v + 8 * q;
                        uint4 pk = make_uint4(pack_bf16(u[0], u[1]), pack_bf16(u[2], u[3]), pack_bf16(u[4], u[5]),
                                              pack_bf16(u[6], u[7]));
                        *reinterpret_cast<uint4*>(smem + FwdLayout::act + sw_off(r, cc + 8 * q)) = pk;
                    }
                } else {
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const float4 wv = reinterpret_cast<const float4*>(w4 + cc)[q];
                        yacc = fmaf(v[4 * q], wv.x, fmaf(v[4 * q + 1], wv.y, fmaf(v[4 * q + 2], wv.z,
                                                                                   fmaf(v[4 * q + 3], wv.w, yacc))));
                    }
                }
            }
        }
        if (!ok) break;
        if (hf) ypart[r] = yacc;
        tc_fence_before();  // the next tile's MMA overwrites the accumulator read above
        __syncthreads();
        if (!hf && live) {
            const float yn = (yacc + ypart[r]) + b4[0];
            y[row] = fmaf(yn, nm.out_sd, nm.out_mu);
        }
    }
    if (!ok && t == 0) {
        atomicExch(status, 1);
        mbar_wait(bar, ph);  // bounded: let an issued MMA land
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) tmem_free(tmem, 128);
}

// ====================================================================== inference
// k_mlp_infer: the same forward arithmetic as k_mlp_forward, with four tiles in
// flight per SM.  One block per SM of four warpgroups; warpgroup g owns tile slot g
// (its BF16 activation operand and accumulator columns [128 g, 128 g + 128) of tensor
// memory) and runs its own tiles, thread = row, all 128 columns per thread; the three
// weight operands are shared.  A warpgroup synchronises only with itself (named
// barrier 1 + g, its own mbarrier), so while one waits for its MMAs the other three
// run their GELUs: the tensor pipe, the FMA pipe and the tanh unit overlap across
// the four tiles.  The hidden activations are kept as 2 gelu(z) (gelu2x, one multiply
// fewer per value) and the weights that read them (W2, W3, w4) are halved on loading;
// both scalings are exact, so the outputs are those of k_mlp_forward bit for bit.
constexpr int IG = 4;                    // warpgroups (tile slots) per block
constexpr int IT = IG * MT;              // threads per block
struct InfLayout {
    static constexpr size_t w2 = 0, w3 = 2 * ATOM, act = 4 * ATOM;  // act: IG slots of 2 atoms
    static constexpr size_t w1 = act + (size_t)IG * 2 * ATOM;       // layer 1's B operand
    static constexpr size_t f32 = w1 + W1OP;                        // b1, b2, b3, w4, b4
    static constexpr size_t bars = f32 + 4 * (4 * MH + 4);
    static constexpr size_t total = bars + 64;
};
constexpr size_t INF_SMEM = InfLayout::total + 1024;

__device__ __forceinline__ void group_sync(int g) {
    asm volatile("bar.sync %0, %1;" :: "r"(1 + g), "r"(MT) : "memory");
}
__device__ __forceinline__ bool group_and(int g, bool v) {
    int r;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %1, 0;\n\tbar.red.and.pred q, %2, %3, p;\n\t"
                 "selp.s32 %0, 1, 0, q;\n\t}\n" : "=r"(r) : "r"((int)v), "r"(1 + g), "r"(MT) : "memory");
    return r != 0;
}

__global__ void __launch_bounds__(IT, 1)
k_mlp_infer(const float* __restrict__ params, const __nv_bfloat16* __restrict__ wbf, MlpNorm nm,
            const float* __restrict__ X, long long n, const unsigned long long* __restrict__ n_dev,
            long long ldx, float* __restrict__ y, int* __restrict__ status) {
    if (n_dev) n = min(n, (long long)*n_dev);  // rows counted on the device (at most n)
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
    const int t = threadIdx.x, warp = t >> 5, g = t >> 7, r = t & (MT - 1);
    float* b1 = (float*)(smem + InfLayout::f32);
    float* b2 = b1 + MH;
    float* b3 = b2 + MH;
    float* w4 = b3 + MH;
    float* b4 = w4 + MH;
    unsigned long long* bars = (unsigned long long*)(smem + InfLayout::bars);
    unsigned* tmem_slot = (unsigned*)(smem + InfLayout::bars + 8 * IG);
    const unsigned bar = smem_u32(&bars[g]);
    const unsigned s_w2 = smem_u32(smem + InfLayout::w2), s_w3 = smem_u32(smem + InfLayout::w3);
    const unsigned s_w1 = smem_u32(smem + InfLayout::w1);
    unsigned char* act = smem + InfLayout::act + (size_t)g * 2 * ATOM;
    const unsigned s_act = smem_u32(act);

    for (int idx = t; idx < 2 * MH * (MH / 8); idx += IT) {
        const int l = idx / (MH * (MH / 8)), rem = idx - l * (MH * (MH / 8));
        const int row = rem >> 4, ch = rem & 15;
        uint4 v = *reinterpret_cast<const uint4*>(wbf + (size_t)l * MH * MH + row * MH + ch * 8);
        __nv_bfloat162* h2 = reinterpret_cast<__nv_bfloat162*>(&v);
#pragma unroll
        for (int q = 0; q < 4; ++q) h2[q] = __hmul2(h2[q], __float2bfloat162_rn(0.5f));  // exact: a power of 2
        *reinterpret_cast<uint4*>(smem + (l ? InfLayout::w3 : InfLayout::w2) + sw_off(row, ch * 8)) = v;
    }
    fill_w1_operand(smem + InfLayout::w1, params, t, IT);
    for (int k = t; k < MH; k += IT) {
        b1[k] = params[XTS_MLP_B1 + k];
        b2[k] = params[XTS_MLP_B2 + k];
        b3[k] = params[XTS_MLP_B3 + k];
        w4[k] = 0.5f * __bfloat162float(__float2bfloat16_rn(params[XTS_MLP_W4 + k]));
    }
    if (t < IG) mbar_init(smem_u32(&bars[t]), 1);
    if (t == 0) b4[0] = params[XTS_MLP_B4];
    if (warp == 0) tmem_alloc(smem_u32(tmem_slot), 128 * IG);
    fence_async_shared();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = *tmem_slot + (unsigned)(MH * g);  // this slot's accumulator columns
    const unsigned trow = tmem + ((unsigned)((warp & 3) * 32) << 16);
    unsigned ph = 0;
    bool ok = true;
    const long long ntiles = (n + MT - 1) / MT;
    const long long stride = (long long)gridDim.x * IG;
    // the features of this slot's next row, loaded one tile ahead
    float xn[MI];
    auto load_x = [&](long long tl) {
        const long long rw = tl * MT + r;
#pragma unroll
        for (int k = 0; k < MI; ++k) xn[k] = tl < ntiles && rw < n ? X[ldx ? k * ldx + rw : rw * MI + k] : 0.f;
    };
    load_x((long long)blockIdx.x * IG + g);
    for (long long tile = (long long)blockIdx.x * IG + g; tile < ntiles && ok; tile += stride) {
        const long long row = tile * MT + r;
        const bool live = row < n;
        // layer 1's A operand: the row's split features (the slot's last MMA, which read
        // the operand, has completed)
        {
            float x[MI];
#pragma unroll
            for (int k = 0; k < MI; ++k) x[k] = live ? (xn[k] - nm.mu[k]) / nm.sd[k] : 0.f;
            load_x(tile + stride);
            store_x_split(act, r, x);
        }
        float ylo = 0.f, yhi = 0.f;  // the output layer over columns 0..63 and 64..127
        for (int layer = 1; layer <= 3 && ok; ++layer) {
            fence_async_shared();
            tc_fence_before();
            group_sync(g);
            if (r == 0) {
                tc_fence_after();
                if (layer == 1) mma_layer1(tmem, s_act, s_w1);
                else mma_chain(tmem, s_act, layer == 2 ? s_w2 : s_w3, MH / 16, false);
                mma_commit(bar);
            }
            // one warp of the group polls the MMA's mbarrier; the other three sleep in the
            // group's barrier instead of spinning (their issue slots go to the other groups)
            bool got = true;
            if ((warp & 3) == 0) got = mbar_wait(bar, ph);
            if (!group_and(g, got)) { ok = false; break; }  // ph stays: the exit path waits on it
            ph ^= 1;
            tc_fence_after();
            const float* bias = layer == 1 ? b1 : layer == 2 ? b2 : b3;
            // the accumulator read 16 columns at a time, the next 16 in flight while
            // these are worked on
            unsigned ra[16], rb[16];
            tmem_ld16_issue(trow, ra);
            tmem_ld_done(ra);
#pragma unroll
            for (int c0 = 0; c0 < MH; c0 += 16) {
                if (c0 + 16 < MH) tmem_ld16_issue(trow + (unsigned)(c0 + 16), rb);
                float v[16], bv[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(ra[j]);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float4 b = reinterpret_cast<const float4*>(bias + c0)[q];
                    bv[4 * q] = b.x; bv[4 * q + 1] = b.y; bv[4 * q + 2] = b.z; bv[4 * q + 3] = b.w;
                }
#pragma unroll
                for (int j = 0; j < 16; j += 2) {
                    const float2 z = __fadd2_rn(make_float2(v[j], v[j + 1]), make_float2(bv[j], bv[j + 1]));
                    const float2 g2 = gelu2x(z);
                    v[j] = g2.x;
                    v[j + 1] = g2.y;
                }
                if (layer < 3) {
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        const float* u = v + 8 * q;
                        *reinterpret_cast<uint4*>(act + sw_off(r, c0 + 8 * q)) =
                            make_uint4(pack_bf16(u[0], u[1]), pack_bf16(u[2], u[3]), pack_bf16(u[4], u[5]),
                                       pack_bf16(u[6], u[7]));
                    }
                } else {
                    float ya = c0 < 64 ? ylo : yhi;
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const float4 wv = reinterpret_cast<const float4*>(w4 + c0)[q];
                        ya = fmaf(v[4 * q], wv.x, fmaf(v[4 * q + 1], wv.y, fmaf(v[4 * q + 2], wv.z,
                                                                                fmaf(v[4 * q + 3], wv.w, ya))));
                    }
                    if (c0 < 64) ylo = ya; else yhi = ya;
                }
                if (c0 + 16 < MH) {
                    tmem_ld_done(rb);
#pragma unroll
                    for (int j = 0; j < 16; ++j) ra[j] = rb[j];
                }
            }
            tc_fence_before();  // the next MMA overwrites the accumulator read above
        }
        if (!ok) break;
        if (live) y[row] = fmaf((ylo + yhi) + b4[0], nm.out_sd, nm.out_mu);
    }
    if (!ok && r == 0) {
        atomicExch(status, 1);
        mbar_wait(bar, ph);  // bounded: let this slot's issued MMA land
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) tmem_free(*tmem_slot, 128 * IG);
}

// ====================================================================== GEMM
constexpr size_t GEMM_SMEM = 4 * ATOM / 2 * 2 + 64 + 1024;  // two stages of A and B chunks ([128][64] each)

// Stage the [128 rows][64] chunk (rows r0.., K columns k0..) of an operand into
// one swizzled atom.  trans: the operand is stored [K][ld] (row index fastest).
__device__ __forceinline__ void load_chunk(unsigned char* dst, const __nv_bfloat16* src, int trans, long long ld,
                                           long long r0, long long k0, int t) {
    if (!trans) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int idx = t + MT * i, r = idx >> 3, ch = idx & 7;
            const uint4 v = *reinterpret_cast<const uint4*>(src + (r0 + r) * ld + k0 + ch * 8);
            *reinterpret_cast<uint4*>(dst + sw_off(r, ch * 8)) = v;
        }
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int idx = t + MT * i, kk = idx >> 4, rg = idx & 15;
            const uint4 v = *reinterpret_cast<const uint4*>(src + (k0 + kk) * ld + r0 + rg * 8);
            const unsigned short* e = reinterpret_cast<const unsigned short*>(&v);
#pragma unroll
            for (int j = 0; j < 8; ++j) *reinterpret_cast<unsigned short*>(dst + sw_off(rg * 8 + j, kk)) = e[j];
        }
    }
}

__global__ void __launch_bounds__(MT, 1)
k_gemm_bf16(const __nv_bfloat16* __restrict__ A, int a_trans, const __nv_bfloat16* __restrict__ B, int b_trans,
            int M, int K, int cps, float* __restrict__ C, int c_trans, int atomic, int* __restrict__ status) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
    const int t = threadIdx.x, warp = t >> 5;
    const int nkc = K / 64;
    const int kc0 = blockIdx.y * cps, kc1 = min(kc0 + cps, nkc);
    if (kc0 >= kc1) return;  // uniform over the block, before any tensor memory is held
    const long long m0 = (long long)blockIdx.x * MT;
    unsigned long long* bars = (unsigned long long*)(smem + 4 * ATOM);
    unsigned* tmem_slot = (unsigned*)(smem + 4 * ATOM + 32);
    if (t == 0) {
        mbar_init(smem_u32(&bars[0]), 1);
        mbar_init(smem_u32(&bars[1]), 1);
    }
    if (warp == 0) tmem_alloc(smem_u32(tmem_slot), 128);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = *tmem_slot;
    unsigned ph[2] = {0, 0};
    int pending[2] = {0, 0};
    bool ok = true;
    for (int c = kc0; c < kc1; ++c) {
        const int st = (c - kc0) & 1;
        unsigned char* sa = smem + st * 2 * ATOM;
        unsigned char* sb = sa + ATOM;
        if (pending[st]) {  // the MMAs issued two chunks ago read this stage
            const bool got = mbar_wait(smem_u32(&bars[st]), ph[st]);
            if (!__syncthreads_and(got)) { ok = false; break; }  // still pending: the exit path waits
            ph[st] ^= 1;
            pending[st] = 0;
        }
        load_chunk(sa, A, a_trans, a_trans ? (long long)M : (long long)K, m0, (long long)c * 64, t);
        load_chunk(sb, B, b_trans, b_trans ? (long long)MH : (long long)K, 0, (long long)c * 64, t);
        fence_async_shared();
        tc_fence_before();
        __syncthreads();
        if (t == 0) {
            tc_fence_after();
            mma_chain(tmem, smem_u32(sa), smem_u32(sb), 4, c > kc0);
            mma_commit(smem_u32(&bars[st]));
        }
        pending[st] = 1;
    }
    // the last commit covers every MMA issued before it
    const int last = (kc1 - 1 - kc0) & 1;
    if (ok) {
        const bool got = mbar_wait(smem_u32(&bars[last]), ph[last]);
        ok = __syncthreads_and(got);
        if (ok) {
            ph[last] ^= 1;
            pending[last] = 0;
        }
    }
    if (ok) {
        tc_fence_after();
        const long long m = m0 + t;
        const unsigned trow = tmem + ((unsigned)(warp * 32) << 16);
        for (int c0 = 0; c0 < MH; c0 += 16) {
            float v[16];
            tmem_ld16(trow + (unsigned)c0, v);
            float* Cs = atomic ? C + (size_t)blockIdx.y * M * MH : C;  // split-K: this split's partial tile
#pragma unroll
            for (int j = 0; j < 16; ++j)
                *(c_trans ? Cs + (size_t)(c0 + j) * M + m : Cs + (size_t)m * MH + c0 + j) = v[j];
        }
    } else if (t == 0) {
        atomicExch(status, 1);
        for (int s = 0; s < 2; ++s)
            if (pending[s]) mbar_wait(smem_u32(&bars[s]), ph[s]);  // bounded
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) tmem_free(tmem, 128);
}

// ====================================================================== training
// One kernel from the batch to all partial sums of the gradient.  A block takes tiles of
// 128 rows; thread = row r and 32 of the 128 units (four warpgroups).  Per tile:
//   z1 = W1 x -> accumulator A, h1 to shared memory;  z2 = W2 h1 -> B, h2;  z3 = W3 h2 -> A;
//   dz3 = dy w4 gelu'(z3), to shared memory as BF16;  dh2 = dz3 W3 -> A,  dW3 += dz3^T h2;
//   dz2 = dh2 gelu'(z2);  dh1 = dz2 W2 -> B,  dW2 += dz2^T h1,  z1 once more -> A;
//   dz1 = dh1 gelu'(z1).
// No pre-activation, activation or dh leaves the SM: A, B, dW3 and dW2 fill the 512
// columns of tensor memory, the two weight gradients staying there over the block's tiles.
// Each operand is stored once: W, dz and h are read as K-major in the one product and,
// with the transpose bits of the instruction, along the other axis in the next.  A weight
// product is waited for only before its operands are written again.  Sums over rows
// (biases, W1, w4): each warp turns 32 rows x 16 units through its own shared memory and a
// lane adds eight rows of a pair of units (a shuffle butterfly took four instructions per
// value and sum, this takes one and a half).  Each block writes its sums once;
// k_mlp_grad_sum adds the blocks' in a fixed order, so trainings repeat bit for bit.
// 37,888 rows (two tiles per block): 43 us and 9 us for the sums, where a forward, a
// backward and a weight-product kernel that pass z, h and dz through memory took 37, 48 and
// 42 us.  A further tile per block takes 12.5 us, about half of it issuing (the GELUs, their
// derivatives and the sums), the rest the five waits for products that need the whole tile.
enum { BQ_B3 = 0, BQ_W4 = 1, BQ_B2 = 2, BQ_B1 = 3, BQ_W1 = 4, BQ_LOSS = 9, BQ_B4 = 10, BQ_N = 11 };
constexpr int GT = 4 * MT;  // threads
struct GradLayout {
    static constexpr size_t w2 = 0, w3 = 2 * ATOM, h1 = 4 * ATOM, h2 = 6 * ATOM, dz = 8 * ATOM;
    static constexpr size_t w1 = 10 * ATOM, xop = w1 + W1OP;     // layer 1's operands, no swizzle
    static constexpr size_t turn = xop + W1OP;                   // [16 warps][32 rows][8] pairs
    static constexpr size_t xs = turn + 16 * 32 * 8 * 8;         // [MT][8]: x, then y's parts 1..3
    static constexpr size_t tot = xs + MT * 8 * 4;               // [9][4 row warps][MH]
    static constexpr size_t f32 = tot + 9 * 4 * MH * 4;          // b1, b2, b3, w4, y's part 0 [MT], b4 (+3)
    static constexpr size_t sred = f32 + 4 * (5 * MH + 4);       // [4][2]: loss, dy
    static constexpr size_t bars = sred + 4 * 8;
    static constexpr size_t total = bars + 64;
};
constexpr size_t GRAD_SMEM = GradLayout::total + 1024;
static_assert(GRAD_SMEM <= 232448, "shared memory of one block");

// An operand of [128][64] atoms read along its other axis (M or N = the atom's 64
// contiguous elements, K = its rows): 128-byte swizzle, next 64 elements ATOM bytes on
// (leading offset), next 8 rows 1024 bytes on (stride offset); 16 rows per MMA step.
static __device__ __forceinline__ unsigned long long m_desc_mn(unsigned addr) {
    return (unsigned long long)((addr >> 4) & 0x3FFF) | ((unsigned long long)(ATOM >> 4) << 16) | (64ull << 32) |
           (1ull << 46) | (2ull << 61);
}
constexpr unsigned A_MN = 1u << 15, B_MN = 1u << 16;

// D = A B over K = 128; A K-major (adv 0) or along its other axis, B along its other axis
template <bool AT>
__device__ __forceinline__ void mma_chain_t(unsigned tmem, unsigned a, unsigned b, bool acc0) {
    for (int ks = 0; ks < 8; ++ks) {
        const unsigned long long da = AT ? m_desc_mn(a + (unsigned)(ks * 2048))
                                         : m_desc(a + (unsigned)((ks >> 2) * ATOM + (ks & 3) * 32));
        const unsigned long long db = m_desc_mn(b + (unsigned)(ks * 2048));
        const unsigned acc = (acc0 || ks > 0) ? 1u : 0u;
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                     "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}\n"
                     :: "r"(tmem), "l"(da), "l"(db), "r"(M_IDESC | B_MN | (AT ? A_MN : 0u)), "r"(acc), "r"(0u));
    }
}

__device__ __forceinline__ void store_bf16x16(unsigned char* op, int r, int c, const float* u) {
#pragma unroll
    for (int q = 0; q < 2; ++q)
        *reinterpret_cast<uint4*>(op + sw_off(r, c + 8 * q)) =
            make_uint4(pack_bf16(u[8 * q], u[8 * q + 1]), pack_bf16(u[8 * q + 2], u[8 * q + 3]),
                       pack_bf16(u[8 * q + 4], u[8 * q + 5]), pack_bf16(u[8 * q + 6], u[8 * q + 7]));
}

// Sums over the warp's 32 rows (lane = row) of 16 units, added to tot[unit], and with XW
// the five sums weighted by the rows' features, to tot[(1 + q) * 4 * MH + unit].  Pair p of
// row r at word pair 8 r + (p ^ (r / 2 & 7)): writes (a row per lane) and reads (eight pairs
// of four rows) each touch all banks once per half warp.  The lane that adds to a slot of
// tot is always the same.
template <bool XW>
__device__ __forceinline__ void row_sums(float2* turn, const float* v, const float* xs, float* tot) {
    const int lane = threadIdx.x & 31, pair = lane & 7, rg = lane >> 3;
    __syncwarp();
#pragma unroll
    for (int p = 0; p < 8; ++p) turn[lane * 8 + (p ^ ((lane >> 1) & 7))] = make_float2(v[2 * p], v[2 * p + 1]);
    __syncwarp();
    constexpr int NS = XW ? 1 + MI : 1;
    float2 s[NS];
#pragma unroll
    for (int k = 0; k < NS; ++k) s[k] = make_float2(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int row = rg + 4 * i;
        const float2 u = turn[row * 8 + (pair ^ ((row >> 1) & 7))];
        s[0] = __fadd2_rn(s[0], u);
        if (XW) {
            const float4 x = *reinterpret_cast<const float4*>(xs + row * 8);
            const float x4 = xs[row * 8 + 4];
            s[1 % NS] = __ffma2_rn(u, make_float2(x.x, x.x), s[1 % NS]);
            s[2 % NS] = __ffma2_rn(u, make_float2(x.y, x.y), s[2 % NS]);
            s[3 % NS] = __ffma2_rn(u, make_float2(x.z, x.z), s[3 % NS]);
            s[4 % NS] = __ffma2_rn(u, make_float2(x.w, x.w), s[4 % NS]);
            s[5 % NS] = __ffma2_rn(u, make_float2(x4, x4), s[5 % NS]);
        }
    }
#pragma unroll
    for (int k = 0; k < NS; ++k) {
#pragma unroll
        for (int o = 8; o <= 16; o <<= 1) {
            s[k].x += __shfl_xor_sync(0xffffffffu, s[k].x, o);
            s[k].y += __shfl_xor_sync(0xffffffffu, s[k].y, o);
        }
        if (rg == 0) {
            float2* d = reinterpret_cast<float2*>(tot + k * 4 * MH + 2 * pair);
            *d = __fadd2_rn(*d, s[k]);
        }
    }
}

__global__ void __launch_bounds__(GT, 1)
k_mlp_gradient(const float* __restrict__ params, const __nv_bfloat16* __restrict__ wbf, MlpNorm nm,
               const float* __restrict__ X, const float* __restrict__ Y, long long n, float* __restrict__ part,
               float* __restrict__ wpart, int* __restrict__ status) {
    let_next_start();
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31, r = t & (MT - 1), qd = t >> 7, cb = 32 * qd, rw = warp & 3;
    unsigned char* h1 = smem + GradLayout::h1;
    unsigned char* h2 = smem + GradLayout::h2;
    unsigned char* dz = smem + GradLayout::dz;
    unsigned char* xop = smem + GradLayout::xop;
    float2* turn = (float2*)(smem + GradLayout::turn) + warp * 256;
    float* xs = (float*)(smem + GradLayout::xs);
    float* tot = (float*)(smem + GradLayout::tot);
    float* b1 = (float*)(smem + GradLayout::f32);
    float* b2 = b1 + MH;
    float* b3 = b2 + MH;
    float* w4 = b3 + MH;
    float* y0 = w4 + MH;
    float* b4 = y0 + MT;
    float* sred = (float*)(smem + GradLayout::sred);
    unsigned long long* bars = (unsigned long long*)(smem + GradLayout::bars);
    unsigned* tmem_slot = (unsigned*)(smem + GradLayout::bars + 32);
    const unsigned bar = smem_u32(&bars[0]), wbar = smem_u32(&bars[1]);
    const unsigned s_w1 = smem_u32(smem + GradLayout::w1), s_w2 = smem_u32(smem + GradLayout::w2);
    const unsigned s_w3 = smem_u32(smem + GradLayout::w3), s_x = smem_u32(xop);
    const unsigned s_h1 = smem_u32(h1), s_h2 = smem_u32(h2), s_dz = smem_u32(dz);

    for (int idx = t; idx < 2 * MH * (MH / 8); idx += GT) {
        const int l = idx / (MH * (MH / 8)), rem = idx - l * (MH * (MH / 8));
        const int row = rem >> 4, ch = rem & 15;
        const uint4 v = *reinterpret_cast<const uint4*>(wbf + (size_t)l * MH * MH + row * MH + ch * 8);
        *reinterpret_cast<uint4*>(smem + (l ? GradLayout::w3 : GradLayout::w2) + sw_off(row, ch * 8)) = v;
    }
    fill_w1_operand(smem + GradLayout::w1, params, t, GT);
    for (int k = t; k < 9 * 4 * MH; k += GT) tot[k] = 0.f;
    if (t < MH) {
        b1[t] = params[XTS_MLP_B1 + t];
        b2[t] = params[XTS_MLP_B2 + t];
        b3[t] = params[XTS_MLP_B3 + t];
        w4[t] = __bfloat162float(__float2bfloat16_rn(params[XTS_MLP_W4 + t]));
    }
    if (t == 0) {
        b4[0] = params[XTS_MLP_B4];
        mbar_init(bar, 1);
        mbar_init(wbar, 1);
    }
    if (warp == 0) tmem_alloc(smem_u32(tmem_slot), 512);
    fence_async_shared();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tm = *tmem_slot, t_a = tm, t_b = tm + 128, t_w3 = tm + 256, t_w2 = tm + 384;
    const unsigned lane0 = (unsigned)(rw * 32) << 16;
    const float inv_n = 1.f / (float)n;
    float sum_d2 = 0.f, sum_dy = 0.f;
    unsigned ph = 0, wph = 0;
    bool ok = true, got = true, wpend = false;  // wpend: a weight product not yet waited for
    // mma_issue: operands in shared memory and the accumulators' last readers, then the
    // MMAs of issue; mma_wait: their end.  Work between the two overlaps them.  A wait that
    // timed out in any thread ends the loop at the next mma_issue.
    bool pend = false;
    auto mma_issue = [&](auto issue) {
        fence_async_shared();
        tc_fence_before();
        if (!__syncthreads_and(got)) return false;
        if (t == 0) {
            tc_fence_after();
            issue();
        }
        pend = true;
        return true;
    };
    auto mma_wait = [&]() {
        if (mbar_wait(bar, ph)) {
            ph ^= 1;
            pend = false;
        }
        got = got && !pend;
        __syncwarp();
        tc_fence_after();
    };
    // each thread sees the weight product complete; a timeout ends the loop
    auto weights_done = [&]() {
        if (wpend && mbar_wait(wbar, wph)) {
            wph ^= 1;
            wpend = false;
        }
        got = got && !wpend;
        __syncwarp();
    };
    auto layer1 = [&](unsigned d) {  // as mma_layer1, the A operand without swizzle
        const unsigned long long da = m_desc_ns(s_x), db = m_desc_ns(s_w1);
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                     "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}\n"
                     :: "r"(d), "l"(da), "l"(db), "r"(M_IDESC), "r"(0u), "r"(0u));
    };
    // 16 pre-activations of this thread's row: accumulator plus bias
    auto load_z = [&](unsigned acc, const float* bias, int c, float* z) {
        tmem_ld16(acc + lane0 + (unsigned)c, z);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float4 b = reinterpret_cast<const float4*>(bias + c)[q];
            z[4 * q] += b.x; z[4 * q + 1] += b.y; z[4 * q + 2] += b.z; z[4 * q + 3] += b.w;
        }
    };
    // the same and 16 values of dh, one wait for both
    auto load_z_dh = [&](unsigned acc, const float* bias, unsigned dacc, int c, float* z, float* dh) {
        unsigned ra[16], rb[16];
        tmem_ld16_issue(acc + lane0 + (unsigned)c, ra);
        tmem_ld16_issue(dacc + lane0 + (unsigned)c, rb);
        tmem_ld_done(ra);
        tmem_ld_done(rb);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float4 b = reinterpret_cast<const float4*>(bias + c)[q];
            z[4 * q] = __uint_as_float(ra[4 * q]) + b.x;
            z[4 * q + 1] = __uint_as_float(ra[4 * q + 1]) + b.y;
            z[4 * q + 2] = __uint_as_float(ra[4 * q + 2]) + b.z;
            z[4 * q + 3] = __uint_as_float(ra[4 * q + 3]) + b.w;
        }
#pragma unroll
        for (int j = 0; j < 16; ++j) dh[j] = __uint_as_float(rb[j]);
    };
    auto act16 = [&](float* z) {
#pragma unroll
        for (int j = 0; j < 16; j += 2) {
            const float2 g = gelu2(make_float2(z[j], z[j + 1]));
            z[j] = g.x;
            z[j + 1] = g.y;
        }
    };
    const long long ntiles = n / MT;
    float xn[MI], tn;  // the next tile's features and target of this row
    auto load_row = [&](long long tile) {
        const long long row = (tile < ntiles ? tile : (long long)blockIdx.x) * MT + r;
        if (qd == 0)
#pragma unroll
            for (int k = 0; k < MI; ++k) xn[k] = X[row * MI + k];
        tn = Y[row];
    };
    load_row(blockIdx.x);
    for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        if (qd == 0) {
            float x[MI];
#pragma unroll
            for (int k = 0; k < MI; ++k) xs[r * 8 + k] = x[k] = (xn[k] - nm.mu[k]) / nm.sd[k];
            store_x_split_ns(xop, r, x);
        }
        const float target = (tn - nm.out_mu) / nm.out_sd;
        if (!(ok = mma_issue([&] { layer1(t_a); mma_commit(bar); }))) break;
        mma_wait();
        weights_done();  // the previous tile's dW2 has read h1 and dz
        float v[32], u[32];
#pragma unroll 1
        for (int c = cb; c < cb + 32; c += 16) {
            load_z(t_a, b1, c, v);
            act16(v);
            store_bf16x16(h1, r, c, v);
        }
        if (!(ok = mma_issue([&] { mma_chain(t_b, s_h1, s_w2, 8, false); mma_commit(bar); }))) break;
        mma_wait();
#pragma unroll 1
        for (int c = cb; c < cb + 32; c += 16) {
            load_z(t_b, b2, c, v);
            act16(v);
            store_bf16x16(h2, r, c, v);
        }
        if (!(ok = mma_issue([&] { mma_chain(t_a, s_h2, s_w3, 8, false); mma_commit(bar); }))) break;
        mma_wait();
        float yp = 0.f;
#pragma unroll 1
        for (int c = cb; c < cb + 32; c += 16) {
            load_z(t_a, b3, c, v);
            act16(v);
#pragma unroll
            for (int j = 0; j < 16; ++j) yp = fmaf(v[j], w4[c + j], yp);
        }
        *(qd ? xs + r * 8 + MI - 1 + qd : y0 + r) = yp;
        __syncthreads();
        const float yn = ((y0[r] + xs[r * 8 + MI]) + (xs[r * 8 + MI + 1] + xs[r * 8 + MI + 2])) + b4[0];
        const float d = yn - target, dy = 2.f * d * inv_n;
        if (qd == 0) {
            sum_d2 = fmaf(d, d, sum_d2);
            sum_dy += dy;
        }
#pragma unroll
        for (int g = 0; g < 32; g += 16) {
            load_z(t_a, b3, cb + g, v + g);
#pragma unroll
            for (int j = g; j < g + 16; ++j) {
                u[j] = dy * gelu(v[j]);
                v[j] = dy * w4[cb + j] * gelu_grad(v[j]);
            }
            store_bf16x16(dz, r, cb + g, v + g);
        }
        const bool first = tile == blockIdx.x;
        if (!(ok = mma_issue([&] {
                  mma_chain_t<false>(t_a, s_dz, s_w3, false);
                  mma_commit(bar);
                  mma_chain_t<true>(t_w3, s_dz, s_h2, !first);
                  mma_commit(wbar);
              })))
            break;
        wpend = true;
#pragma unroll
        for (int g = 0; g < 32; g += 16) {
            row_sums<false>(turn, v + g, nullptr, tot + (BQ_B3 * 4 + rw) * MH + cb + g);
            row_sums<false>(turn, u + g, nullptr, tot + (BQ_W4 * 4 + rw) * MH + cb + g);
        }
        mma_wait();
#pragma unroll
        for (int g = 0; g < 32; g += 16) {
            load_z_dh(t_b, b2, t_a, cb + g, v + g, u);
#pragma unroll
            for (int j = 0; j < 16; ++j) v[g + j] = u[j] * gelu_grad(v[g + j]);
        }
        weights_done();  // dW3 has read dz
        store_bf16x16(dz, r, cb, v);
        store_bf16x16(dz, r, cb + 16, v + 16);
        if (!(ok = mma_issue([&] {
                  mma_chain_t<false>(t_b, s_dz, s_w2, false);
                  layer1(t_a);
                  mma_commit(bar);
                  mma_chain_t<true>(t_w2, s_dz, s_h1, !first);
                  mma_commit(wbar);
              })))
            break;
        wpend = true;
#pragma unroll
        for (int g = 0; g < 32; g += 16)
            row_sums<false>(turn, v + g, nullptr, tot + (BQ_B2 * 4 + rw) * MH + cb + g);
        load_row(tile + gridDim.x);
        mma_wait();
#pragma unroll 1
        for (int c = cb; c < cb + 32; c += 16) {
            load_z_dh(t_a, b1, t_b, c, v, u);
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = u[j] * gelu_grad(v[j]);
            row_sums<true>(turn, v, xs + rw * 32 * 8, tot + (BQ_B1 * 4 + rw) * MH + c);
        }
        __syncthreads();  // xs is read before the next tile's is written
    }
    if (ok) {
        weights_done();
        ok = __syncthreads_and(got);
    }
    if (ok) {
        tc_fence_after();
        const int l = qd >> 1, hc = 64 * (qd & 1);
        float4* dst = reinterpret_cast<float4*>(wpart) + ((size_t)l * gridDim.x + blockIdx.x) * (MH * MH / 4) + r;
#pragma unroll 1
        for (int c = 0; c < 64; c += 16) {
            float w[16];
            tmem_ld16((l ? t_w2 : t_w3) + lane0 + (unsigned)(hc + c), w);
#pragma unroll
            for (int q = 0; q < 4; ++q)
                dst[((hc + c) / 4 + q) * MH] = make_float4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
        }
        for (int o = 16; o > 0; o >>= 1) {
            sum_d2 += __shfl_xor_sync(0xffffffffu, sum_d2, o);
            sum_dy += __shfl_xor_sync(0xffffffffu, sum_dy, o);
        }
        if (qd == 0 && lane == 0) { sred[2 * rw] = sum_d2; sred[2 * rw + 1] = sum_dy; }
    } else if (t == 0) {
        atomicExch(status, 1);
        if (pend) mbar_wait(bar, ph);  // bounded: let issued MMAs land
        if (wpend) mbar_wait(wbar, wph);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (ok) {
        for (int k = t; k < 9 * MH; k += GT) {
            const float* a = tot + (size_t)(k / MH) * 4 * MH + k % MH;
            part[(size_t)k * gridDim.x + blockIdx.x] = ((a[0] + a[MH]) + a[2 * MH]) + a[3 * MH];
        }
        if (t < 2)
            part[(size_t)(BQ_LOSS + t) * MH * gridDim.x + blockIdx.x] =
                ((sred[t] + sred[2 + t]) + sred[4 + t]) + sred[6 + t];
    }
    if (warp == 0) tmem_free(tm, 512);
}

// The gradients from their parts, written to (add 0) or added to grads; the loss likewise.
// Blocks 0 .. 255: 128 elements each of the hidden weights' tiles (wpart
// [2][nb][column / 4][row][4]: W3, W2), warp w the tiles k = w mod 8, the warps' sums in order;
// further blocks: one warp per (quantity, unit) of k_mlp_gradient's nb blocks.
constexpr int GS_WB = 2 * MH * MH / 128;
__global__ void __launch_bounds__(256) k_mlp_grad_sum(const float* __restrict__ part, const float* __restrict__ wpart,
                                                      int nb, float inv_n, int add, float* __restrict__ grads,
                                                      float* __restrict__ loss) {
    after_previous();
    __shared__ float4 red[8][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if ((int)blockIdx.x < GS_WB) {
        const int l = blockIdx.x / (GS_WB / 2), e0 = (blockIdx.x - l * (GS_WB / 2)) * 128;
        const float* w = wpart + (size_t)l * nb * MH * MH + e0 + 4 * lane;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
        for (int k = warp; k < nb; k += 8) {
            const float4 u = *reinterpret_cast<const float4*>(w + (size_t)k * MH * MH);
            v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
        }
        red[warp][lane] = v;
        __syncthreads();
        if (threadIdx.x < 128) {
            const float* f = reinterpret_cast<const float*>(red) + threadIdx.x;
            float s = 0.f;
#pragma unroll
            for (int k = 0; k < 8; ++k) s += f[128 * k];
            const int e = (e0 + (int)threadIdx.x) >> 2, col = (e / MH) * 4 + (threadIdx.x & 3), row = e & (MH - 1);
            float* g = grads + (l ? XTS_MLP_W2 : XTS_MLP_W3) + row * MH + col;
            *g = add ? *g + s : s;
        }
        return;
    }
    const int i = ((int)blockIdx.x - GS_WB) * 8 + warp, q = i / MH, j = i - q * MH;
    if (q >= BQ_N || (q >= BQ_LOSS && j > 0)) return;
    const float* p = part + (size_t)i * nb;
    float v = 0.f;
    for (int b = lane; b < nb; b += 32) v += p[b];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane) return;
    if (q == BQ_LOSS) {
        if (loss) *loss = add ? *loss + v * inv_n : v * inv_n;
        return;
    }
    const int at = q == BQ_B3 ? XTS_MLP_B3 + j : q == BQ_W4 ? XTS_MLP_W4 + j : q == BQ_B2 ? XTS_MLP_B2 + j
                 : q == BQ_B1 ? XTS_MLP_B1 + j : q == BQ_B4 ? XTS_MLP_B4 : XTS_MLP_W1 + j * MI + (q - BQ_W1);
    grads[at] = add ? grads[at] + v : v;
}

// C[i] += sum over the splits s (in order) of part[s][i]
__global__ void k_sum_splits(const float* __restrict__ part, int nsplit, long long n, float* __restrict__ C) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float v = 0.f;
    for (int s = 0; s < nsplit; ++s) v += part[(size_t)s * n + i];
    C[i] += v;
}

// Adam on the FP32 master parameters; the BF16 copies of W2 and W3 follow.
__global__ void k_mlp_adam(float* __restrict__ p, float* __restrict__ g, float* __restrict__ m,
                           float* __restrict__ v, __nv_bfloat16* __restrict__ wbf, float lr, float c1, float c2) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= XTS_MLP_NPARAM) return;
    const float gi = g[i];
    const float mi = fmaf(0.9f, m[i], 0.1f * gi);
    const float vi = fmaf(0.999f, v[i], 0.001f * gi * gi);
    m[i] = mi;
    v[i] = vi;
    g[i] = 0.f;
    const float pi = p[i] - lr * (mi * c1) / (sqrtf(vi * c2) + 1e-8f);
    p[i] = pi;
    if (i >= XTS_MLP_W2 && i < XTS_MLP_B2) wbf[i - XTS_MLP_W2] = __float2bfloat16_rn(pi);
    if (i >= XTS_MLP_W3 && i < XTS_MLP_B3) wbf[MH * MH + (i - XTS_MLP_W3)] = __float2bfloat16_rn(pi);
}

// ====================================================================== launchers
static int sm_count() {
    int dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    return nsm;
}

static int mlp_status(int* status, cudaStream_t st) {
    int v = 0;
    XTS_CUDA(cudaMemcpyAsync(&v, status, sizeof(int), cudaMemcpyDeviceToHost, st));
    XTS_CUDA(cudaStreamSynchronize(st));
    if (v) {
        cudaMemsetAsync(status, 0, sizeof(int), st);
        return set_error(XTS_ERR_TIMEOUT, "a bounded tensor-core wait gave up (surrogate network)");
    }
    return XTS_OK;
}

int launch_gemm_bf16(const void* A, int a_trans, const void* B, int b_trans, int M, int K, float* C, int c_trans,
                     int accumulate, int* status, cudaStream_t st) {
    if (M <= 0 || K <= 0 || M % MT || K % 64)
        return set_error(XTS_ERR_ARG, "gemm_bf16: M (%d) must be a multiple of 128 and K (%d) of 64", M, K);
    XTS_CUDA(cudaFuncSetAttribute(k_gemm_bf16, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GEMM_SMEM));
    const int mt = M / MT, nkc = K / 64;
    int nsplit = 1;
    if (accumulate) {  // spread the K chunks over about one wave of blocks
        nsplit = (sm_count() + mt - 1) / mt;
        nsplit = nsplit < 1 ? 1 : (nsplit > nkc ? nkc : nsplit);
    }
    const int cps = (nkc + nsplit - 1) / nsplit;
    nsplit = (nkc + cps - 1) / cps;
    if (!accumulate && nsplit != 1) return set_error(XTS_ERR_ARG, "gemm_bf16: internal split");
    float* dst = C;
    const long long nc = (long long)M * MH;
    if (accumulate) {  // partial tiles per split, summed in a fixed order below
        dst = (float*)workspace(W_MLP_PART, sizeof(float) * (size_t)nsplit * nc);
        if (!dst) return XTS_ERR_OOM;
    }
    XTS_LAUNCH("k_gemm_bf16", st, k_gemm_bf16<<<dim3(mt, nsplit), MT, GEMM_SMEM, st>>>(
                                      (const __nv_bfloat16*)A, a_trans, (const __nv_bfloat16*)B, b_trans, M, K, cps,
                                      dst, c_trans, accumulate, status));
    if (accumulate)
        XTS_LAUNCH("k_sum_splits", st, k_sum_splits<<<(unsigned)((nc + 255) / 256), 256, 0, st>>>(dst, nsplit, nc, C));
    return XTS_OK;
}

// X: row-major [n][5] (ldx 0) or feature-major [5][ldx] (ldx >= n)
static int forward(const xts_mlp* net, const float* X, long long n, const unsigned long long* n_dev, float* y,
                   int* status, cudaStream_t st, long long ldx = 0) {
    // per call: the attribute belongs to the current device's context
    XTS_CUDA(cudaFuncSetAttribute(k_mlp_forward, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FWD_SMEM));
    if (!y) return set_error(XTS_ERR_ARG, "mlp forward: output");
    const long long ntiles = (n + MT - 1) / MT;
    const int bps = g_tuning.mlp_blocks_per_sm > 0 ? g_tuning.mlp_blocks_per_sm : 2;  // blocks per SM (two fit)
    const long long g = ntiles < bps * sm_count() ? ntiles : bps * sm_count();
    if (g_tuning.mlp_blocks_per_sm == 0) {
        // inference: four tiles in flight per SM, one block per SM
        XTS_CUDA(cudaFuncSetAttribute(k_mlp_infer, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)INF_SMEM));
        const long long gi = (ntiles + IG - 1) / IG < sm_count() ? (ntiles + IG - 1) / IG : sm_count();
        XTS_LAUNCH("k_mlp_infer", st, k_mlp_infer<<<(unsigned)gi, IT, INF_SMEM, st>>>(
                                            net->params, (const __nv_bfloat16*)net->wbf16, mlp_norm(net), X, n, n_dev,
                                            ldx, y, status));
    } else {
        XTS_LAUNCH("k_mlp_forward", st, k_mlp_forward<<<(unsigned)g, FT, FWD_SMEM, st>>>(
                                            net->params, (const __nv_bfloat16*)net->wbf16, mlp_norm(net), X, n, n_dev,
                                            ldx, y, status));
    }
    return XTS_OK;
}

int launch_mlp_forward(const xts_mlp* net, const float* X, long long n, float* y, int* status, cudaStream_t st) {
    if (n <= 0) return XTS_OK;
    return forward(net, X, n, nullptr, y, status, st);
}

int launch_mlp_forward_dev(const xts_mlp* net, const float* X, const unsigned long long* n_dev, long long n_max,
                           float* y, int* status, cudaStream_t st, long long ldx) {
    if (n_max <= 0) return XTS_OK;
    if (ldx && ldx < n_max) return set_error(XTS_ERR_ARG, "mlp forward: feature stride below the row count");
    return forward(net, X, n_max, n_dev, y, status, st, ldx);
}

// the gradient written (add 0) or added to grads, the loss likewise
static int mlp_backprop(const xts_mlp* net, const float* X, const float* Y, long long n, int add, float* grads,
                        float* loss, int* status, cudaStream_t st) {
    if (n <= 0 || n % MT) return set_error(XTS_ERR_ARG, "surrogate training: n (%lld) must be a positive multiple of 128", n);
    if (n > (1ll << 24)) return set_error(XTS_ERR_ARG, "surrogate training: n (%lld) above 2^24 rows per batch", n);
    const int nb = (int)(n / MT < sm_count() ? n / MT : sm_count());
    float* part = (float*)workspace(W_MLP_PART2, sizeof(float) * (size_t)BQ_N * MH * nb);
    float* wpart = (float*)workspace(W_MLP_PART, sizeof(float) * 2 * (size_t)nb * MH * MH);
    if (!part || !wpart) return XTS_ERR_OOM;
    XTS_CUDA(cudaFuncSetAttribute(k_mlp_gradient, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GRAD_SMEM));
    XTS_LAUNCH("k_mlp_gradient", st, k_mlp_gradient<<<nb, GT, GRAD_SMEM, st>>>(
                                         net->params, (const __nv_bfloat16*)net->wbf16, mlp_norm(net), X, Y, n, part,
                                         wpart, status));
    XTS_LAUNCH("k_mlp_grad_sum", st, launch_next(
                                         k_mlp_grad_sum, GS_WB + (BQ_N * MH + 7) / 8, 256, 0, st, part, wpart, nb,
                                         1.f / (float)n, add, grads, loss));
    return XTS_OK;
}

int launch_mlp_grads(const xts_mlp* net, const float* X, const float* Y, long long n, float* grads, float* loss,
                     int* status, cudaStream_t st) {
    int rc = mlp_backprop(net, X, Y, n, 0, grads, loss, status, st);
    if (rc) return rc;
    return mlp_status(status, st);
}

int launch_mlp_train_step(const xts_mlp* net, const float* X, const float* Y, long long n, float* grads,
                          float* m, float* v, int step, float lr, float* loss, int* status, cudaStream_t st) {
    if (step < 1) return set_error(XTS_ERR_ARG, "surrogate training: step must be >= 1");
    int rc = mlp_backprop(net, X, Y, n, 1, grads, loss, status, st);
    if (rc) return rc;
    const float c1 = (float)(1.0 / (1.0 - pow(0.9, step))), c2 = (float)(1.0 / (1.0 - pow(0.999, step)));
    XTS_LAUNCH("k_mlp_adam", st, k_mlp_adam<<<(XTS_MLP_NPARAM + 255) / 256, 256, 0, st>>>(
                                     net->params, grads, m, v, (__nv_bfloat16*)net->wbf16, lr, c1, c2));
    return XTS_OK;
}

int mlp_check_status(int* status, cudaStream_t st) { return mlp_status(status, st); }

}  // namespace xts
