// The kernels either side of the MoE path: the hyper-connection residual mixer
// that feeds every layer and the teacher's head (mda_qwen_res_rec,
// src/qwen.c:641-663; mda_qwen_head, src/qwen.c:1080-1099), and the dense fp16
// product both use (mda_qwen_mm, src/qwen.c:541-570).
//   moe_cuda_norm    shader/qwen_norm.comp op 0 / op 1 (grouped RMSNorm)
//   moe_cuda_hc      shader/qwen_hc.comp ops 0, 1, 2
//   moe_cuda_dense   C[rows x n] fp32 = A16[rows x k] * W[n x k]^T / scale(sa):
//                    the weight-stationary tcgen05 kernel of moe_mm_ws.cu over
//                    all rows (one "expert")
// Elementwise kernels are HBM bound: 128-bit accesses, coalesced along the row.
#include "moe_common.cuh"

#define NR_THREADS 256

__device__ __forceinline__ float dn_sigmoid(float v) { return 1.0f / (1.0f + expf(-v)); }  // qwen_hc.comp:16-18

__device__ __forceinline__ void dn_store(float *p, float v) {
    asm volatile("st.global.L1::no_allocate.f32 [%0], %1;" ::"l"(p), "f"(v) : "memory");
}

// One block per (row, group), as the shader (:64-67).  op 0: y = x * rsqrt(mean(x^2) + eps) * (1 + w);
// op 1: y = x * scale * rsqrt(sum(x^2) + 1e-6), no weight (:45-61).
// General form: the second read of the group is meant to hit L1, so the stores pass it by (3001 rows of 4 x 2050: 38.9 us
// without that, 37.8 us).
template <int U>
__global__ void __launch_bounds__(NR_THREADS)
moe_norm_kernel(const float *x, const float *w, float *y, struct mda_pc_qwen_norm_t pc) {
    moe_pdl_begin();
    __shared__ float red[NR_THREADS / 32];
    const uint32_t r = blockIdx.x / pc.groups, g = blockIdx.x % pc.groups;
    const float *xi = x + (size_t)r * pc.in_stride + pc.in_off + (size_t)g * pc.in_gstride;
    float *yi = y + (size_t)r * pc.out_stride + pc.out_off + (size_t)g * pc.out_gstride;
    const float *wi = w != NULL ? w + pc.w_off + (size_t)g * pc.wstride : NULL;
    const bool weighted = pc.op == 0u && w != NULL;  // :45-53
    float acc = 0.0f;
    for (uint32_t c0 = threadIdx.x; c0 < pc.gsize; c0 += U * NR_THREADS) {  // :71-73
        float v[U];
#pragma unroll
        for (int i = 0; i < U; i += 1) v[i] = c0 + i * NR_THREADS < pc.gsize ? xi[c0 + i * NR_THREADS] : 0.0f;
#pragma unroll
        for (int i = 0; i < U; i += 1) acc += v[i] * v[i];
    }
#pragma unroll
    for (uint32_t o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31u) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    float ss = 0.0f;
#pragma unroll
    for (uint32_t q = 0; q < NR_THREADS / 32; q += 1) ss += red[q];
    const float f = pc.op == 1u ? pc.scale * rsqrtf(ss + 1e-6f) : rsqrtf(ss / (float)pc.gsize + pc.eps);  // :55-61
    for (uint32_t c0 = threadIdx.x; c0 < pc.gsize; c0 += U * NR_THREADS) {
        float v[U], wt[U];
#pragma unroll
        for (int i = 0; i < U; i += 1) {
            const uint32_t c = c0 + i * NR_THREADS;
            v[i] = c < pc.gsize ? xi[c] : 0.0f;
            wt[i] = c < pc.gsize && weighted ? wi[c] : 0.0f;
        }
#pragma unroll
        for (int i = 0; i < U; i += 1) {
            const uint32_t c = c0 + i * NR_THREADS;
            if (c < pc.gsize) dn_store(yi + c, v[i] * f * (1.0f + wt[i]));  // :78,90
        }
    }
}

// The same with groups of at most NR_THREADS * 4 * NV columns, all on 16 bytes: the group is read once and kept in
// registers.  Bound by HBM; 3001 rows of 4 x 2048: 36.6 us read twice in single values, 34.0 us this way; of 8192: 37.5
// and 34.3 us.
template <int NV>
__global__ void __launch_bounds__(NR_THREADS)
moe_norm4_kernel(const float *x, const float *w, float *y, struct mda_pc_qwen_norm_t pc) {
    moe_pdl_begin();
    __shared__ float red[NR_THREADS / 32];
    const uint32_t r = blockIdx.x / pc.groups, g = blockIdx.x % pc.groups, n4 = pc.gsize / 4u;
    const float4 *xi = reinterpret_cast<const float4 *>(x + (size_t)r * pc.in_stride + pc.in_off + (size_t)g * pc.in_gstride);
    float4 *yi = reinterpret_cast<float4 *>(y + (size_t)r * pc.out_stride + pc.out_off + (size_t)g * pc.out_gstride);
    const bool weighted = pc.op == 0u && w != NULL;
    const float4 *wi = weighted ? reinterpret_cast<const float4 *>(w + pc.w_off + (size_t)g * pc.wstride) : NULL;
    float4 v[NV], wv[NV];
    float acc = 0.0f;
#pragma unroll
    for (int i = 0; i < NV; i += 1) {
        const uint32_t c = i * NR_THREADS + threadIdx.x;
        v[i] = c < n4 ? xi[c] : make_float4(0.f, 0.f, 0.f, 0.f);
        wv[i] = weighted && c < n4 ? wi[c] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int i = 0; i < NV; i += 1) acc += v[i].x * v[i].x + v[i].y * v[i].y + v[i].z * v[i].z + v[i].w * v[i].w;
#pragma unroll
    for (uint32_t o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31u) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    float ss = 0.0f;
#pragma unroll
    for (uint32_t q = 0; q < NR_THREADS / 32; q += 1) ss += red[q];
    const float f = pc.op == 1u ? pc.scale * rsqrtf(ss + 1e-6f) : rsqrtf(ss / (float)pc.gsize + pc.eps);
#pragma unroll
    for (int i = 0; i < NV; i += 1) {
        const uint32_t c = i * NR_THREADS + threadIdx.x;
        if (c < n4) yi[c] = make_float4(v[i].x * f * (1.0f + wv[i].x), v[i].y * f * (1.0f + wv[i].y),
                                        v[i].z * f * (1.0f + wv[i].z), v[i].w * f * (1.0f + wv[i].w));
    }
}

extern "C" void moe_cuda_norm(moe_cuda_ctx_t *c, const float *x, const float *w, float *y, const float *z,
                              struct mda_pc_qwen_norm_t pc) {
    (void)z;  // binding 3 of the shader: only its op 2 reads it
    if (!MOE_LIVE(c)) return;
    MOE_REQUIRE(c, pc.op <= 1u, "norm: only op 0 (weighted RMSNorm) and op 1 (scaled L2 norm) are part of this path");
    MOE_REQUIRE(c, x != NULL && y != NULL && (w != NULL || pc.op == 1u), "norm: null buffer");
    MOE_REQUIRE(c, pc.groups >= 1 && pc.gsize >= 1, "norm: empty group");
    if (pc.rows == 0) return;
    const uint32_t wlay = pc.op == 0u ? pc.w_off | pc.wstride : 0u;
    if ((pc.gsize | pc.in_stride | pc.in_off | pc.in_gstride | pc.out_stride | pc.out_off | pc.out_gstride | wlay) % 4u == 0 &&
        (((uintptr_t)x | (uintptr_t)y | (pc.op == 0u ? (uintptr_t)w : 0u)) & 15) == 0 && pc.gsize <= NR_THREADS * 4u * 8u) {
        if (pc.gsize <= NR_THREADS * 4u * 2u) moe_run(c, moe_norm4_kernel<2>, pc.rows * pc.groups, NR_THREADS, 0, x, w, y, pc);
        else if (pc.gsize <= NR_THREADS * 4u * 4u) moe_run(c, moe_norm4_kernel<4>, pc.rows * pc.groups, NR_THREADS, 0, x, w, y, pc);
        else moe_run(c, moe_norm4_kernel<8>, pc.rows * pc.groups, NR_THREADS, 0, x, w, y, pc);
        MOE_LAUNCHED(c);
        return;
    }
    // A chip that is not full (8 blocks per SM) waits for loads, so eight columns per thread are in flight; on a full one
    // issue slots count (12,004 groups of 2050: 37.6 us one by one, 46.4 by four).
    const uint32_t grid = pc.rows * pc.groups;
    if (grid < 8u * (uint32_t)c->sm_count) moe_run(c, moe_norm_kernel<8>, grid, NR_THREADS, 0, x, w, y, pc);
    else moe_run(c, moe_norm_kernel<1>, grid, NR_THREADS, 0, x, w, y, pc);
    MOE_LAUNCHED(c);
}

// shader/qwen_hc.comp.  op 0: h[r,c] = mean_s sigmoid(a[r,s,c]) * b[r,s,c]  (the mixer's read-out, :24-30);
// op 1: h[r,s,c] += a[r,c] * 2*sigmoid(b[r*inj_stride + inj_off + s] / hc)  (:31-35);
// op 2: h[i] += a[i] + b[i]  (:36-38).
template <uint32_t OP>
__global__ void __launch_bounds__(256, 8)
moe_hc_kernel(const float *a, const float *b, float *h, struct mda_pc_qwen_hc_t pc) {
    moe_pdl_begin();
    const size_t n = (size_t)pc.rows * pc.d * (OP == 2u ? pc.hc : 1u);
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        if (OP == 2u) {
            h[i] += a[i] + b[i];
            continue;
        }
        const size_t r = i / pc.d;
        const uint32_t col = (uint32_t)(i - r * pc.d);
        if (OP == 0u) {
            float acc = 0.0f;
            for (uint32_t s = 0; s < pc.hc; s += 1) {
                const size_t j = (r * pc.hc + s) * pc.d + col;
                acc += dn_sigmoid(a[j]) * b[j];
            }
            h[i] = acc / (float)pc.hc;
        } else {
            const float av = a[i];
            // four streams' loads in front of their stores (3001 rows of 4 x 2048: 73.8 us one by one, 64.9 us this way)
            for (uint32_t s0 = 0; s0 < pc.hc; s0 += 4u) {
                float g[4], hv[4];
#pragma unroll
                for (uint32_t q = 0; q < 4; q += 1) {
                    if (s0 + q >= pc.hc) break;
                    g[q] = b[r * pc.inj_stride + pc.inj_off + s0 + q];
                    hv[q] = h[(r * pc.hc + s0 + q) * pc.d + col];
                }
#pragma unroll
                for (uint32_t q = 0; q < 4; q += 1) {
                    if (s0 + q >= pc.hc) break;
                    h[(r * pc.hc + s0 + q) * pc.d + col] = hv[q] + av * (2.0f * dn_sigmoid(g[q] / (float)pc.hc));
                }
            }
        }
    }
}

// The read-out with four columns per thread (d % 4 == 0, 16-byte aligned): all 2 * HC loads of a thread are in flight
// together.  Bound by HBM; 3001 rows of 4 x 2048: 76 us one column at a time, 35 us this way.
template <uint32_t HC>
__global__ void __launch_bounds__(NR_THREADS)
moe_hc_read4_kernel(const float4 *a, const float4 *b, float4 *h, uint32_t total4, uint32_t d4) {
    moe_pdl_begin();
    const uint32_t i = blockIdx.x * NR_THREADS + threadIdx.x;
    if (i >= total4) return;
    const uint32_t r = i / d4;
    const size_t j0 = (size_t)r * HC * d4 + (i - r * d4);
    float4 av[HC], bv[HC];
#pragma unroll
    for (uint32_t s = 0; s < HC; s += 1) {
        av[s] = a[j0 + (size_t)s * d4];
        bv[s] = b[j0 + (size_t)s * d4];
    }
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (uint32_t s = 0; s < HC; s += 1) {
        acc.x += dn_sigmoid(av[s].x) * bv[s].x;
        acc.y += dn_sigmoid(av[s].y) * bv[s].y;
        acc.z += dn_sigmoid(av[s].z) * bv[s].z;
        acc.w += dn_sigmoid(av[s].w) * bv[s].w;
    }
    h[i] = make_float4(acc.x / (float)HC, acc.y / (float)HC, acc.z / (float)HC, acc.w / (float)HC);
}

extern "C" void moe_cuda_hc(moe_cuda_ctx_t *c, const float *a, const float *b, float *h, struct mda_pc_qwen_hc_t pc) {
    if (!MOE_LIVE(c)) return;
    MOE_REQUIRE(c, pc.op <= 2u && pc.hc >= 1 && pc.d >= 1, "hc: bad op or shape");
    MOE_REQUIRE(c, a != NULL && b != NULL && h != NULL, "hc: null buffer");
    const size_t n = (size_t)pc.rows * pc.d * (pc.op == 2u ? pc.hc : 1u);
    if (n == 0) return;
    // the teacher's four streams; other counts and ragged or unaligned rows take the general form below
    if (pc.op == 0u && pc.hc == 4u && pc.d % 4u == 0 && ((uintptr_t)a | (uintptr_t)b | (uintptr_t)h) % 16 == 0 && n / 4 < (1ull << 31)) {
        const uint32_t total4 = (uint32_t)(n / 4);
        moe_run(c, moe_hc_read4_kernel<4>, (total4 + NR_THREADS - 1u) / NR_THREADS, NR_THREADS, 0,
                (const float4 *)a, (const float4 *)b, (float4 *)h, total4, pc.d / 4u);
        MOE_LAUNCHED(c);
        return;
    }
    size_t blocks = (n + 255) / 256;
    if (blocks > (size_t)c->sm_count * 16) blocks = (size_t)c->sm_count * 16;
    if (pc.op == 0u) moe_run(c, moe_hc_kernel<0>, (unsigned)blocks, 256, 0, a, b, h, pc);
    else if (pc.op == 1u) moe_run(c, moe_hc_kernel<1>, (unsigned)blocks, 256, 0, a, b, h, pc);
    else moe_run(c, moe_hc_kernel<2>, (unsigned)blocks, 256, 0, a, b, h, pc);
    MOE_LAUNCHED(c);
}

// mda_qwen_mm (src/qwen.c:541-570): the reference picks matmul_f16_wide.comp or the small-tile kernel by the
// number of 128 x 128 tiles; here one tcgen05 kernel serves both.  rows need not be a multiple of 128: rows of A
// beyond `rows` read as zero and rows of C beyond `rows` are not written.
extern "C" void moe_cuda_dense(moe_cuda_ctx_t *c, const void *A16, const void *W, float *C, const uint32_t *amax,
                               struct moe_pc_dense_t pc) {
    if (!MOE_LIVE(c)) return;
    MOE_REQUIRE(c, A16 != NULL && W != NULL && C != NULL, "dense: null buffer");
    MOE_REQUIRE(c, pc.rows >= 1 && pc.n % 128u == 0 && pc.n >= 128u && pc.k % 8u == 0 && pc.k >= 8u,
                "dense: rows %u n %u k %u (n must be a multiple of 128, k of 8)", pc.rows, pc.n, pc.k);
    moe_launch_mm_dense(c, A16, W, C, amax, NULL, pc.rows, pc.n, pc.k, pc.sa, MDA_PC_NO_SLOT, 1);
}
