// Weighted gather-sum back to token order, and the three elementwise glue
// kernels that sit between the two grouped products in the unfused sequence.
// CUDA for sm_100a; all HBM access is 128-bit and coalesced along the row.
#include "moe_common.cuh"

#define CB_THREADS 256
#define CB_KEEP 32  // values per thread kept for the fused norm: d <= 8192
#define CB_TERMS 8  // expert rows whose loads a thread has in flight together

__device__ __forceinline__ float moe_sigmoid(float v) {  // shader/moe_combine.comp:22-24
    return 1.0f / (1.0f + expf(-v));
}

// V neighbouring values of a row, 8 to 16 bytes, as fetched and as floats.
template <typename YT, int V> struct moe_vec;
template <> struct moe_vec<float, 4> { typedef float4 raw; };
template <> struct moe_vec<__half, 4> { typedef uint2 raw; };
template <> struct moe_vec<__half, 8> { typedef uint4 raw; };
template <typename YT, int V>
__device__ __forceinline__ typename moe_vec<YT, V>::raw moe_fetch(const YT *p) {
    return *reinterpret_cast<const typename moe_vec<YT, V>::raw *>(p);
}
__device__ __forceinline__ void moe_floats(float4 r, float (&f)[4]) {
    f[0] = r.x; f[1] = r.y; f[2] = r.z; f[3] = r.w;
}
__device__ __forceinline__ void moe_floats2(uint32_t r, float *f) {
    const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&r));
    f[0] = a.x; f[1] = a.y;
}
__device__ __forceinline__ void moe_floats(uint2 r, float (&f)[4]) {
    moe_floats2(r.x, f); moe_floats2(r.y, f + 2);
}
__device__ __forceinline__ void moe_floats(uint4 r, float (&f)[8]) {
    moe_floats2(r.x, f); moe_floats2(r.y, f + 2); moe_floats2(r.z, f + 4); moe_floats2(r.w, f + 6);
}
// acc += w * v, multiply and add rounded separately
template <int V>
__device__ __forceinline__ void moe_axpy(float (&acc)[V], float w, const float (&v)[V]) {
#pragma unroll
    for (int i = 0; i < V; i += 1) acc[i] = __fadd_rn(acc[i], __fmul_rn(w, v[i]));
}

// One block per row (shader/moe_combine.comp:26-40 uses one thread per element).
// acc = sum_j wt[r,j] * y[slot[r,j], c] in j order with separately rounded
// multiply and add, as the expression is written in the shader (:32-34).
// Bound by HBM for many rows and by the chain of loads for few: a thread takes V values of 16 bytes where the row
// allows it, and the loads of up to CB_TERMS expert rows are issued before the first is used (one at a time, 16 rows
// of 2048 with the norm took 11.2 us); the values kept for the norm are indexed statically, so that they stay in
// registers (2048 rows: 37 us before, 23 us now; 16 rows 4.5 us).
// NORM: 0, or the fused norm's passes of CB_THREADS * V columns over the row.
template <typename YT, int NORM, bool PEER, int V>
__global__ void __launch_bounds__(CB_THREADS)
moe_combine_kernel(moe_combine_args a) {
    moe_pdl_begin();
    __shared__ uint32_t s_slot[MOE_MAX_TOPK];
    __shared__ float s_wt[MOE_MAX_TOPK];
    __shared__ float s_f[8];
    __shared__ float s_red[CB_THREADS / 32];
    __shared__ const YT *s_y[PEER ? MOE_MAX_TOPK : 1];
    __shared__ uint32_t s_mask, s_terms;
    const YT *y = reinterpret_cast<const YT *>(a.y);
    // One row per block and pass (rows blockIdx.x, blockIdx.x + gridDim.x, ...).
    for (uint32_t r = blockIdx.x; r < a.rows; r += gridDim.x) {
        if (PEER && a.per_gpu) {
            // Expert-parallel, one row per owning GPU: every GPU that owns some of the token's experts has
            // already summed wt * row over those experts (moe_ep_partial_kernel); one such partial row per
            // GPU comes over NVLink and the partial rows are added in ascending GPU order.
            if (threadIdx.x == 0) s_mask = 0;
            __syncthreads();
            if (threadIdx.x < a.topk) {
                uint32_t g = a.idx[(size_t)r * a.topk + threadIdx.x] / a.experts_per_rank;
                if (g < a.world) atomicOr(&s_mask, 1u << g);  // a row the router refused carries ~0: no term
            }
            __syncthreads();
            if (threadIdx.x == 0) {
                uint32_t n = 0;
                for (uint32_t mk = s_mask; mk != 0; mk &= mk - 1u, n += 1) {
                    s_y[n] = reinterpret_cast<const YT *>(a.y_peers[__ffs((int)mk) - 1]);
                    s_slot[n] = a.src_base + r;
                    s_wt[n] = 1.0f;
                }
                s_terms = n;
            }
        } else if (threadIdx.x < a.topk) {
            uint32_t sl = a.slot[(size_t)r * a.topk + threadIdx.x];
            if (PEER) {  // expert-parallel, one row per pair: read from the GPU that owns the expert, over NVLink
                const uint32_t g = a.idx[(size_t)r * a.topk + threadIdx.x] / a.experts_per_rank;
                s_y[threadIdx.x] = reinterpret_cast<const YT *>(a.y_peers[g < a.world ? g : 0u]);
                if (g >= a.world) sl = ~0u;
            }
            s_slot[threadIdx.x] = sl;  // ~0: a pair the router refused, contributes nothing
            s_wt[threadIdx.x] = a.wt[(size_t)r * a.topk + threadIdx.x];
        }
        if (threadIdx.x >= 32 && threadIdx.x < 32 + a.hc && a.hc <= 7) {
            uint32_t s = threadIdx.x - 32;
            float iv = a.inj != NULL ? a.inj[(size_t)r * a.inj_stride + a.inj_off + s] : 0.0f;
            s_f[s] = moe_sigmoid(iv / (float)a.hc);  // :37
        }
        if (threadIdx.x == 64) {
            s_f[7] = a.sh != NULL ? moe_sigmoid(a.proj[(size_t)r * a.pstride + a.sg_off]) : 0.0f;  // :35
        }
        __syncthreads();
        const uint32_t terms = (PEER && a.per_gpu) ? s_terms : a.topk;
        float sg = s_f[7];
        constexpr uint32_t TERMS = sizeof(YT) == 4 ? CB_TERMS / 2 : CB_TERMS;
        constexpr int ITS = NORM ? NORM : 1;  // unrolled where their values are kept
        float keep[ITS][V];
        float ss = 0.0f;
        for (uint32_t c0 = 0; c0 < a.d; c0 += CB_THREADS * V * ITS) {
#pragma unroll
            for (int it = 0; it < ITS; it += 1) {
                const uint32_t c = c0 + (it * CB_THREADS + threadIdx.x) * V;
                if (c >= a.d) break;
                float acc[V], f[V];
#pragma unroll
                for (int i = 0; i < V; i += 1) acc[i] = 0.0f;
                for (uint32_t j0 = 0; j0 < terms; j0 += TERMS) {
                    typename moe_vec<YT, V>::raw v[TERMS];
#pragma unroll
                    for (uint32_t j = 0; j < TERMS; j += 1) {
                        if (j0 + j < terms && s_slot[j0 + j] != ~0u)
                            v[j] = moe_fetch<YT, V>((PEER ? s_y[j0 + j] : y) + (size_t)s_slot[j0 + j] * a.d + c);
                    }
#pragma unroll
                    for (uint32_t j = 0; j < TERMS; j += 1) {
                        if (j0 + j >= terms || s_slot[j0 + j] == ~0u) continue;
                        moe_floats(v[j], f);
                        moe_axpy<V>(acc, s_wt[j0 + j], f);
                    }
                }
                if (a.sh != NULL) {
#pragma unroll
                    for (int i = 0; i < V; i += 4) {
                        const float4 v = *reinterpret_cast<const float4 *>(a.sh + (size_t)r * a.d + c + i);
                        acc[i] = __fadd_rn(acc[i], __fmul_rn(sg, v.x));
                        acc[i + 1] = __fadd_rn(acc[i + 1], __fmul_rn(sg, v.y));
                        acc[i + 2] = __fadd_rn(acc[i + 2], __fmul_rn(sg, v.z));
                        acc[i + 3] = __fadd_rn(acc[i + 3], __fmul_rn(sg, v.w));
                    }
                }
                if (NORM) {
                    moe_floats(moe_fetch<__half, V>(a.x16 + (size_t)r * a.d + c), f);
#pragma unroll
                    for (int i = 0; i < V; i += 1) {
                        keep[it][i] = __fadd_rn(f[i], __fmul_rn(__fmul_rn(acc[i], 2.0f), s_f[0]));
                        ss += keep[it][i] * keep[it][i];
                    }
                }
                if (a.h != NULL) {
#pragma unroll 2
                    for (uint32_t s = 0; s < a.hc; s += 1) {  // :36-38
                        const float g = a.hc <= 7 ? s_f[s]
                                                  : moe_sigmoid((a.inj != NULL ? a.inj[(size_t)r * a.inj_stride + a.inj_off + s] : 0.0f) / (float)a.hc);
                        float4 *hp = reinterpret_cast<float4 *>(a.h + ((size_t)r * a.hc + s) * a.d + c);
                        float4 hv[V / 4];
#pragma unroll
                        for (int i = 0; i < V / 4; i += 1) hv[i] = hp[i];
#pragma unroll
                        for (int i = 0; i < V / 4; i += 1) {
                            hv[i].x = __fadd_rn(hv[i].x, __fmul_rn(__fmul_rn(acc[4 * i], 2.0f), g));
                            hv[i].y = __fadd_rn(hv[i].y, __fmul_rn(__fmul_rn(acc[4 * i + 1], 2.0f), g));
                            hv[i].z = __fadd_rn(hv[i].z, __fmul_rn(__fmul_rn(acc[4 * i + 2], 2.0f), g));
                            hv[i].w = __fadd_rn(hv[i].w, __fmul_rn(__fmul_rn(acc[4 * i + 3], 2.0f), g));
                            hp[i] = hv[i];
                        }
                    }
                }
            }
        }
        if (NORM) {
            // residual + RMSNorm with unit weight (shader/qwen_norm.comp:55-61,79 op 0)
#pragma unroll
            for (uint32_t o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
            if ((threadIdx.x & 31u) == 0) s_red[threadIdx.x >> 5] = ss;
            __syncthreads();
            float tot = 0.0f;
#pragma unroll
            for (uint32_t w = 0; w < CB_THREADS / 32; w += 1) tot += s_red[w];
            float inv = 1.0f / sqrtf(tot / (float)a.d + a.eps);
#pragma unroll
            for (int it = 0; it < ITS; it += 1) {
                const uint32_t c = (it * CB_THREADS + threadIdx.x) * V;
                if (c >= a.d) break;
                __align__(16) __half2 o[V / 2];
#pragma unroll
                for (int i = 0; i < V / 2; i += 1) o[i] = __floats2half2_rn(keep[it][2 * i] * inv, keep[it][2 * i + 1] * inv);
                *reinterpret_cast<typename moe_vec<__half, V>::raw *>(a.y16 + (size_t)r * a.d + c) =
                    *reinterpret_cast<const typename moe_vec<__half, V>::raw *>(o);
            }
        }
        __syncthreads();  // the row's tables are rewritten by the next pass
    }
}

// Lets the kernels that move rows over NVLink share an SM with a resident grouped-product CTA: a
// kernel can only join an SM whose shared-memory carve-out matches its own, and the products run
// with the maximum carve-out.
void moe_overlap_prepare_combine(moe_cuda_ctx *c) {
    MOE_CUDA_TRY(c, cudaFuncSetAttribute(moe_combine_kernel<__half, 0, true, 8>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                         cudaSharedmemCarveoutMaxShared));
    MOE_CUDA_TRY(c, cudaFuncSetAttribute(moe_combine_kernel<__half, CB_KEEP / 8, true, 8>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                         cudaSharedmemCarveoutMaxShared));
}

void moe_launch_combine(moe_cuda_ctx *c, const moe_combine_args &a) {
    if (!MOE_LIVE(c)) return;
    MOE_REQUIRE(c, (a.y_peers != NULL && a.per_gpu) || (a.wt != NULL && a.slot != NULL && (a.y != NULL || a.y_peers != NULL)),
                "combine: null buffer");
    MOE_REQUIRE(c, a.y_peers == NULL || (a.idx != NULL && a.experts_per_rank >= 1 && a.world >= 1 && a.world <= 16),
                "combine: peer rows need idx and the world size");
    MOE_REQUIRE(c, a.h != NULL || a.y16 != NULL, "combine: no output");
    MOE_REQUIRE(c, a.sh == NULL || a.proj != NULL, "combine: shared term needs proj");
    MOE_REQUIRE(c, a.topk >= 1 && a.topk <= MOE_MAX_TOPK, "combine: topk %u outside 1..16", a.topk);
    MOE_REQUIRE(c, a.d % 4 == 0 && a.d >= 4, "combine: d %u not a multiple of 4", a.d);
    MOE_REQUIRE(c, a.hc >= 1, "combine: hc 0");
    MOE_REQUIRE(c, ((uintptr_t)a.y & 15) == 0 && ((uintptr_t)a.h & 15) == 0 && ((uintptr_t)a.sh & 15) == 0,
                "combine: buffers not 16-byte aligned");
    if (a.y16 != NULL) {
        MOE_REQUIRE(c, a.x16 != NULL && a.hc == 1 && a.d <= CB_THREADS * CB_KEEP, "combine: fused norm needs x16, hc 1, d <= 8192");
    }
    if (a.rows == 0) return;
    const bool peer = a.y_peers != NULL;
    MOE_REQUIRE(c, !peer || a.y_is_f16, "combine: peer rows are fp16");
    // One block per row: the peer loads want every row in flight.  (A grid bounded to two blocks per SM, meant to
    // leave room for another token slice's product CTAs, measured 115 us against 47 us for the return over 2 GPUs
    // and 0.686 ms against 0.670 ms per layer over 8.)
    const uint32_t grid = a.rows;
    // 16 bytes of fp16 at a time; rows of 4 values more than a multiple of 8, or a caller's buffer on 8 bytes, take 8 bytes
    const bool wide = a.y_is_f16 && a.d % 8u == 0 && (((uintptr_t)a.x16 | (uintptr_t)a.y16) & 15) == 0;
#define CB_RUN(YT, NORM, PEER, V) moe_run(c, moe_combine_kernel<YT, NORM, PEER, V>, grid, CB_THREADS, 0, a)
    if (a.y16 != NULL) {
        if (peer && wide) CB_RUN(__half, CB_KEEP / 8, true, 8);
        else if (peer) CB_RUN(__half, CB_KEEP / 4, true, 4);
        else if (wide && a.d <= CB_THREADS * 8) CB_RUN(__half, 1, false, 8);  // a third fewer registers: more rows in flight
        else if (wide) CB_RUN(__half, CB_KEEP / 8, false, 8);
        else if (a.y_is_f16) CB_RUN(__half, CB_KEEP / 4, false, 4);
        else CB_RUN(float, CB_KEEP / 4, false, 4);
    } else {
        if (peer && wide) CB_RUN(__half, 0, true, 8);
        else if (peer) CB_RUN(__half, 0, true, 4);
        else if (wide) CB_RUN(__half, 0, false, 8);
        else if (a.y_is_f16) CB_RUN(__half, 0, false, 4);
        else CB_RUN(float, 0, false, 4);
    }
#undef CB_RUN
    MOE_LAUNCHED(c);
}

extern "C" void moe_cuda_combine(moe_cuda_ctx_t *c, const float *wt, const uint32_t *slot, const float *y,
                                 const float *proj, const float *sh, const float *inj, float *h,
                                 struct mda_pc_moe_combine_t pc) {
    moe_combine_args a = {};
    a.wt = wt;
    a.slot = slot;
    a.y = y;
    a.proj = proj;
    a.sh = sh;
    a.inj = inj;
    a.h = h;
    a.rows = pc.rows;
    a.d = pc.d;
    a.topk = pc.topk;
    a.pstride = pc.pstride;
    a.sg_off = pc.sg_off;
    a.inj_stride = pc.inj_stride;
    a.inj_off = pc.inj_off;
    a.hc = pc.hc;
    a.y_is_f16 = false;
    moe_launch_combine(c, a);
}

// ---- glue: shader/qwen_elem.comp op 0, shader/absmax.comp, shader/cast_f16.comp ----
__device__ __forceinline__ float moe_silu(float v) { return v / (1.0f + expf(-v)); }  // qwen_elem.comp:16-18

// These kernels are bound by HBM.  Four values per load and several independent loads per thread keep enough bytes in
// flight; the scalar forms (one 4-byte load per thread and iteration, a 64-bit division per value in the SwiGLU) reached
// 2.5 to 4 TB/s.  Measured for 24,320 x 768 SwiGLU outputs, absmax and cast of them: 90, 33 and 26 us scalar against
// 37, 14 and 11 us; absmax and cast of 3001 x 8192: 48 and 42 against 19 and 19 us.
#define EL_THREADS 256u
#define EL_VECS 4u  // 16-byte loads per thread

__device__ __forceinline__ float moe_elem(float g, float u, uint32_t op, float scale) {
    return op == 0u ? __fmul_rn(moe_silu(g), u)    // qwen_elem.comp:27
                    : moe_silu(__fmul_rn(g, scale));  // :29 (the mixer's gate, src/qwen.c:648-657)
}

// General form: any n, stride, offset and alignment.
__global__ void moe_swiglu_kernel(const float *a, float *y, uint32_t rows, uint32_t n,
                                  uint32_t astride, uint32_t ao, uint32_t bo, uint32_t op, float scale) {
    moe_pdl_begin();
    size_t total = (size_t)rows * n;
    size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
        size_t r = i / n;
        uint32_t cidx = (uint32_t)(i - r * n);
        y[i] = moe_elem(a[r * astride + ao + cidx], op == 0u ? a[r * astride + bo + cidx] : 0.0f, op, scale);
    }
}

// Rows, offsets and strides in whole float4: total4 = rows * n4 values of four, below 2^31.
template <uint32_t OP>
__global__ void __launch_bounds__(EL_THREADS)
moe_swiglu4_kernel(const float4 *a, float4 *y, uint32_t total4, uint32_t n4, uint32_t astride4,
                   uint32_t ao4, uint32_t bo4, float scale) {
    moe_pdl_begin();
    constexpr uint32_t U = 2;  // two operands: four loads in flight
    const uint32_t i0 = blockIdx.x * (EL_THREADS * U) + threadIdx.x;
    float4 g[U], u[U];
#pragma unroll
    for (uint32_t j = 0; j < U; j += 1) {
        const uint32_t i = i0 + j * EL_THREADS;
        if (i >= total4) break;
        const uint32_t r = i / n4;
        const float4 *row = a + (size_t)r * astride4 + (i - r * n4);
        g[j] = row[ao4];
        u[j] = OP == 0u ? row[bo4] : g[j];
    }
#pragma unroll
    for (uint32_t j = 0; j < U; j += 1) {
        const uint32_t i = i0 + j * EL_THREADS;
        if (i >= total4) break;
        y[i] = make_float4(moe_elem(g[j].x, u[j].x, OP, scale), moe_elem(g[j].y, u[j].y, OP, scale),
                           moe_elem(g[j].z, u[j].z, OP, scale), moe_elem(g[j].w, u[j].w, OP, scale));
    }
}

extern "C" void moe_cuda_swiglu(moe_cuda_ctx_t *c, const float *a, float *y, struct mda_pc_qwen_elem_t pc) {
    if (!MOE_LIVE(c)) return;
    MOE_REQUIRE(c, pc.op <= 1u, "swiglu: op %u (the shader has 0: silu(gate)*up and 1: silu(scale*a))", pc.op);
    MOE_REQUIRE(c, a != NULL && y != NULL, "swiglu: null buffer");
    size_t total = (size_t)pc.rows * pc.n;
    if (total == 0) return;
    // four values at a time where every row starts on 16 bytes; index arithmetic of 32 bits up to 2^33 values
    if (((uintptr_t)a | (uintptr_t)y) % 16 == 0 && (pc.n | pc.astride | pc.ao | (pc.op == 0u ? pc.bo : 0u)) % 4u == 0 &&
        total / 4 < (1ull << 31)) {
        const uint32_t total4 = (uint32_t)(total / 4), blocks = (total4 + 2u * EL_THREADS - 1u) / (2u * EL_THREADS);
        if (pc.op == 0u)
            moe_run(c, moe_swiglu4_kernel<0>, blocks, EL_THREADS, 0, (const float4 *)a, (float4 *)y, total4, pc.n / 4u,
                    pc.astride / 4u, pc.ao / 4u, pc.bo / 4u, pc.scale);
        else
            moe_run(c, moe_swiglu4_kernel<1>, blocks, EL_THREADS, 0, (const float4 *)a, (float4 *)y, total4, pc.n / 4u,
                    pc.astride / 4u, pc.ao / 4u, 0, pc.scale);
        MOE_LAUNCHED(c);
        return;
    }
    size_t blocks = (total + 255) / 256;
    if (blocks > (size_t)c->sm_count * 16) blocks = (size_t)c->sm_count * 16;
    moe_run(c, moe_swiglu_kernel, (unsigned)blocks, 256, 0, a, y, pc.rows, pc.n, pc.astride, pc.ao, pc.bo, pc.op, pc.scale);
    MOE_LAUNCHED(c);
}

// n4 float4 from the first 16-byte boundary of x on; the few values before and behind them go to the first threads.
__global__ void __launch_bounds__(EL_THREADS)
moe_absmax_kernel(const float *x, uint32_t *amax, uint32_t n, uint32_t head, uint32_t slot) {
    moe_pdl_begin();
    __shared__ float red[EL_THREADS / 32];
    const uint32_t n4 = (n - head) / 4u, stride = gridDim.x * EL_THREADS;
    const float4 *x4 = reinterpret_cast<const float4 *>(x + head);
    const uint32_t first = blockIdx.x * EL_THREADS + threadIdx.x;
    float m = 0.0f;
    for (uint32_t base = first; base < n4; base += EL_VECS * stride) {
        float4 v[EL_VECS];
#pragma unroll
        for (uint32_t j = 0; j < EL_VECS; j += 1) {
            v[j] = base + j * stride < n4 ? x4[base + j * stride] : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (uint32_t j = 0; j < EL_VECS; j += 1) {
            m = fmaxf(m, fmaxf(fmaxf(fabsf(v[j].x), fabsf(v[j].y)), fmaxf(fabsf(v[j].z), fabsf(v[j].w))));
        }
    }
    if (first < head) m = fmaxf(m, fabsf(x[first]));
    const uint32_t tail = head + 4u * n4 + first;
    if (first < 4u && tail < n) m = fmaxf(m, fabsf(x[tail]));
#pragma unroll
    for (uint32_t o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31u) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (uint32_t w = 1; w < EL_THREADS / 32; w += 1) m = fmaxf(m, red[w]);
        atomicMax(&amax[slot], __float_as_uint(m));  // absmax.comp:29; valid for non-negative floats
    }
}

extern "C" void moe_cuda_absmax(moe_cuda_ctx_t *c, const float *x, uint32_t *amax, struct mda_pc_absmax_t pc) {
    if (!MOE_LIVE(c)) return;
    MOE_REQUIRE(c, x != NULL && amax != NULL && pc.slot != MDA_PC_NO_SLOT, "absmax: null buffer or no slot");
    if (pc.n == 0) return;
    uint32_t head = (uint32_t)((16u - (uintptr_t)x % 16u) % 16u / 4u);
    if (head > pc.n) head = pc.n;
    uint32_t blocks = (uint32_t)(((uint64_t)pc.n + 4u * EL_VECS * EL_THREADS - 1u) / (4u * EL_VECS * EL_THREADS));
    if (blocks > (uint32_t)c->sm_count * 8u) blocks = (uint32_t)c->sm_count * 8u;
    moe_run(c, moe_absmax_kernel, blocks, EL_THREADS, 0, x, amax, pc.n, head, pc.slot);
    MOE_LAUNCHED(c);
}

__device__ __forceinline__ uint2 moe_pack4(float4 v, float s) {
    __half2 lo = __floats2half2_rn(v.x * s, v.y * s), hi = __floats2half2_rn(v.z * s, v.w * s);  // cast_f16.comp:33
    return make_uint2(*reinterpret_cast<uint32_t *>(&lo), *reinterpret_cast<uint32_t *>(&hi));
}

// General form: any alignment, four single values in flight per thread.
__global__ void __launch_bounds__(EL_THREADS)
moe_cast_f16_kernel(const float *src, __half *dst, size_t n, const uint32_t *amax, uint32_t slot) {
    moe_pdl_begin();
    const size_t i0 = (size_t)blockIdx.x * (EL_THREADS * EL_VECS) + threadIdx.x;
    float v[EL_VECS];
#pragma unroll
    for (uint32_t j = 0; j < EL_VECS; j += 1) {
        if (i0 + j * EL_THREADS < n) v[j] = src[i0 + j * EL_THREADS];
    }
    const float s = moe_slot_scale(amax, slot);
#pragma unroll
    for (uint32_t j = 0; j < EL_VECS; j += 1) {
        if (i0 + j * EL_THREADS < n) dst[i0 + j * EL_THREADS] = __float2half_rn(v[j] * s);  // cast_f16.comp:33
    }
}

// src on 16 bytes, dst on 8.
__global__ void __launch_bounds__(EL_THREADS)
moe_cast4_f16_kernel(const float4 *src, uint2 *dst, uint32_t n, const uint32_t *amax,
                     uint32_t slot) {
    moe_pdl_begin();
    const uint32_t n4 = n / 4u, i0 = blockIdx.x * (EL_THREADS * EL_VECS) + threadIdx.x;
    float4 v[EL_VECS];
#pragma unroll
    for (uint32_t j = 0; j < EL_VECS; j += 1) {
        if (i0 + j * EL_THREADS < n4) v[j] = src[i0 + j * EL_THREADS];
    }
    const float s = moe_slot_scale(amax, slot);
#pragma unroll
    for (uint32_t j = 0; j < EL_VECS; j += 1) {
        if (i0 + j * EL_THREADS < n4) dst[i0 + j * EL_THREADS] = moe_pack4(v[j], s);
    }
    const uint32_t tail = 4u * n4 + i0;
    if (i0 < 4u && tail < n) reinterpret_cast<__half *>(dst)[tail] = __float2half_rn(reinterpret_cast<const float *>(src)[tail] * s);
}

extern "C" void moe_cuda_cast_f16(moe_cuda_ctx_t *c, const float *src, void *dst, const uint32_t *amax,
                                  struct mda_pc_cast_t pc) {
    if (!MOE_LIVE(c)) return;
    MOE_REQUIRE(c, src != NULL && dst != NULL && (amax != NULL || pc.slot == MDA_PC_NO_SLOT), "cast: null buffer");
    if (pc.n == 0) return;
    if ((uintptr_t)src % 16 == 0 && (uintptr_t)dst % 8 == 0) {
        const uint32_t per = 4u * EL_VECS * EL_THREADS, blocks = (uint32_t)(((uint64_t)pc.n + per - 1u) / per);
        moe_run(c, moe_cast4_f16_kernel, blocks, EL_THREADS, 0, (const float4 *)src, (uint2 *)dst, pc.n, amax, pc.slot);
        MOE_LAUNCHED(c);
        return;
    }
    const uint32_t per = EL_VECS * EL_THREADS, blocks = (uint32_t)(((uint64_t)pc.n + per - 1u) / per);
    moe_run(c, moe_cast_f16_kernel, blocks, EL_THREADS, 0, src, (__half *)dst, pc.n, amax, pc.slot);
    MOE_LAUNCHED(c);
}

// ---- weight upload step: shader/qwen_bf16.comp (call src/qwen.c:365-378) ----
// The reference uploads a layer's bf16 weights and rewrites them in place as fp16 on the
// device.  HBM bound (2 bytes read + 2 bytes written per value): 128-bit accesses, grid-stride.
__device__ __forceinline__ uint32_t moe_bf16x2_to_f16x2(uint32_t u) {
    __half2 h = __floats2half2_rn(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u));  // qwen_bf16.comp:13
    return *reinterpret_cast<uint32_t *>(&h);
}

__global__ void moe_bf16_to_f16_kernel(uint32_t *__restrict__ w, size_t n) {
    size_t n4 = n / 4;
    size_t stride = (size_t)gridDim.x * blockDim.x;
    uint4 *w4 = reinterpret_cast<uint4 *>(w);
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += stride) {
        uint4 v = w4[i];
        v.x = moe_bf16x2_to_f16x2(v.x);
        v.y = moe_bf16x2_to_f16x2(v.y);
        v.z = moe_bf16x2_to_f16x2(v.z);
        v.w = moe_bf16x2_to_f16x2(v.w);
        w4[i] = v;
    }
    size_t tail = n4 * 4 + (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (tail < n) w[tail] = moe_bf16x2_to_f16x2(w[tail]);
}

extern "C" void moe_cuda_bf16_to_f16(moe_cuda_ctx_t *c, void *w, struct mda_pc_qwen_bf16_t pc) {
    if (!MOE_LIVE(c)) return;
    MOE_REQUIRE(c, w != NULL && ((uintptr_t)w & 15) == 0, "bf16_to_f16: null or unaligned buffer");
    if (pc.n == 0) return;
    size_t blocks = ((size_t)pc.n / 4 + 255) / 256;
    if (blocks > (size_t)c->sm_count * 16) blocks = (size_t)c->sm_count * 16;
    if (blocks == 0) blocks = 1;
    moe_bf16_to_f16_kernel<<<(unsigned)blocks, 256, 0, c->stream>>>((uint32_t *)w, pc.n);
    MOE_LAUNCHED(c);
}
