// Context, status and buffer calls of libmoe_cuda: the part of the reference's
// Vulkan harness (src/vkc.c) that the MoE call sites use, restated over the CUDA
// runtime.  One context = one device + one in-order stream + a sticky status.
#include <stdlib.h>
#include <string.h>

#include "moe_common.cuh"

void moe_fail(moe_cuda_ctx *c, int code, const char *fmt, ...) {
    if (c == NULL || c->status != MOE_OK) return;  // first failure wins (src/vkc.c:15-20)
    c->status = code;
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(c->err, sizeof(c->err), fmt, ap);
    va_end(ap);
    fprintf(stderr, "moe_cuda: %s\n", c->err);
}

// Folds refusals recorded by kernels into the sticky status.  Returns true if
// the context is still live.
bool moe_poll_device_status(moe_cuda_ctx *c) {
    if (c == NULL) return false;
    if (c->status == MOE_OK && c->dev_status_host != NULL) {
        uint32_t w = *(volatile uint32_t *)c->dev_status_host;
        if (w != 0) {
            int code = (int)(w & 0xffu);
            if (code == MOE_ERR_ROUTE) {
                moe_fail(c, code, "route: row %u has fewer selectable logits than topk", w >> 8);
            } else if (code == MOE_ERR_TIMEOUT) {
                moe_fail(c, code, "device wait gave up (site %u)", w >> 8);
            } else {
                moe_fail(c, code, "device reported status 0x%x", w);
            }
        }
    }
    return c->status == MOE_OK;
}

extern "C" moe_cuda_ctx_t *moe_cuda_create(int device, void *stream) {
    moe_cuda_ctx *c = (moe_cuda_ctx *)calloc(1, sizeof(moe_cuda_ctx));
    if (c == NULL) return NULL;
    c->device = device;
    c->status = MOE_OK;
    c->wait_ns = 2000000000ull;
    cudaError_t e = cudaSetDevice(device);
    if (e != cudaSuccess) {
        moe_fail(c, MOE_ERR_CUDA, "no usable CUDA device %d: %s", device, cudaGetErrorString(e));
        return c;
    }
    // attributes one by one: cudaGetDeviceProperties takes 2.7 ms, more than all else here
    int major = 0, minor = 0;
    e = cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&c->sm_count, cudaDevAttrMultiProcessorCount, device);
    if (e != cudaSuccess) {
        moe_fail(c, MOE_ERR_CUDA, "device attributes: %s", cudaGetErrorString(e));
        return c;
    }
    if (major != 10) {  // the kernels are built for sm_100a only (cf. src/vkc.c:49-64 feature checks)
        moe_fail(c, MOE_ERR_UNSUPPORTED, "device %d is sm_%d%d, need sm_100", device, major, minor);
        return c;
    }
    if (stream != NULL) {
        c->stream = (cudaStream_t)stream;
    } else {
        e = cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking);
        if (e != cudaSuccess) {
            moe_fail(c, MOE_ERR_CUDA, "stream: %s", cudaGetErrorString(e));
            return c;
        }
        c->own_stream = true;
    }
    e = cudaHostAlloc((void **)&c->dev_status_host, 64, cudaHostAllocMapped);
    if (e == cudaSuccess) {
        memset(c->dev_status_host, 0, 64);
        e = cudaHostGetDevicePointer((void **)&c->dev_status_dev, c->dev_status_host, 0);
    }
    if (e != cudaSuccess) {
        moe_fail(c, MOE_ERR_CUDA, "status word: %s", cudaGetErrorString(e));
        return c;
    }
    c->work_bytes = (size_t)c->sm_count * MOE_WORK_PER_SM;
    if (cudaMalloc(&c->work, c->work_bytes) != cudaSuccess) {
        (void)cudaGetLastError();
        c->work = NULL;
        c->work_bytes = 0;
    }
    cudaDriverEntryPointQueryResult q;
    e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &c->encode_tiled, cudaEnableDefault, &q);
    if (e != cudaSuccess || q != cudaDriverEntryPointSuccess || c->encode_tiled == NULL) {
        moe_fail(c, MOE_ERR_CUDA, "cuTensorMapEncodeTiled not available from this driver");
        return c;
    }
    return c;
}

extern "C" void moe_cuda_destroy(moe_cuda_ctx_t *c) {
    if (c == NULL) return;
    moe_ep_teardown(c);
    if (c->stream != NULL) cudaStreamSynchronize(c->stream);
    for (int i = 0; i < MOE_SCR_COUNT; i += 1) {
        if (c->scratch[i] != NULL) cudaFree(c->scratch[i]);
    }
    if (c->work != NULL) cudaFree(c->work);
    if (c->ev_made) {
        for (int i = 0; i <= MOE_PROF_STAGES; i += 1) cudaEventDestroy(c->ev[i]);
    }
    for (int m = 0; m < c->ev_mb_made; m += 1) {
        for (int i = 0; i <= MOE_PROF_STAGES; i += 1) cudaEventDestroy(c->ev_mb[m][i]);
    }
    if (c->ticket != NULL) cudaFree(c->ticket);
    if (c->dev_status_host != NULL) cudaFreeHost(c->dev_status_host);
    if (c->own_stream) cudaStreamDestroy(c->stream);
    free(c);
}

extern "C" int moe_cuda_status(moe_cuda_ctx_t *c) {
    if (c == NULL) return MOE_ERR_ARG;
    moe_poll_device_status(c);
    return c->status;
}

extern "C" const char *moe_cuda_last_error(moe_cuda_ctx_t *c) {
    return c == NULL ? "no context" : c->err;
}

extern "C" void *moe_cuda_stream(moe_cuda_ctx_t *c) { return c == NULL ? NULL : (void *)c->stream; }

extern "C" void moe_cuda_fail_alloc_after(moe_cuda_ctx_t *c, int n) {
    if (c != NULL) c->fail_alloc_countdown = n;
}

extern "C" void moe_cuda_set_wait_ns(moe_cuda_ctx_t *c, uint64_t ns) {
    if (c != NULL && ns != 0) c->wait_ns = ns;
}

extern "C" uint64_t moe_cuda_launches(moe_cuda_ctx_t *c) { return c == NULL ? 0 : c->launches; }

static bool moe_alloc_refused(moe_cuda_ctx *c) {
    if (c->fail_alloc_countdown > 0) {
        c->fail_alloc_countdown -= 1;
        if (c->fail_alloc_countdown == 0) return true;
    }
    return false;
}

extern "C" void *moe_cuda_alloc(moe_cuda_ctx_t *c, size_t bytes) {
    if (!MOE_LIVE(c)) return NULL;
    void *p = NULL;
    if (moe_alloc_refused(c)) {
        moe_fail(c, MOE_ERR_NOMEM, "alloc of %zu bytes refused (injected)", bytes);
        return NULL;
    }
    cudaError_t e = cudaMalloc(&p, bytes == 0 ? 1 : bytes);
    if (e != cudaSuccess) {
        moe_fail(c, MOE_ERR_NOMEM, "alloc of %zu bytes: %s", bytes, cudaGetErrorString(e));
        return NULL;
    }
    return p;
}

extern "C" void *moe_cuda_alloc_pinned(moe_cuda_ctx_t *c, size_t bytes) {
    if (!MOE_LIVE(c)) return NULL;
    void *p = NULL;
    if (moe_alloc_refused(c)) {
        moe_fail(c, MOE_ERR_NOMEM, "pinned alloc of %zu bytes refused (injected)", bytes);
        return NULL;
    }
    cudaError_t e = cudaHostAlloc(&p, bytes == 0 ? 1 : bytes, cudaHostAllocDefault);
    if (e != cudaSuccess) {
        moe_fail(c, MOE_ERR_NOMEM, "pinned alloc of %zu bytes: %s", bytes, cudaGetErrorString(e));
        return NULL;
    }
    return p;
}

extern "C" void moe_cuda_free(moe_cuda_ctx_t *c, void *p) {
    if (c == NULL || p == NULL) return;
    cudaStreamSynchronize(c->stream);
    cudaFree(p);
}

extern "C" void moe_cuda_free_pinned(moe_cuda_ctx_t *c, void *p) {
    if (c == NULL || p == NULL) return;
    cudaStreamSynchronize(c->stream);
    cudaFreeHost(p);
}

void *moe_scratch(moe_cuda_ctx *c, int area, size_t bytes) {
    if (!MOE_LIVE(c)) return NULL;
    if (c->scratch_bytes[area] >= bytes && c->scratch[area] != NULL) return c->scratch[area];
    if (c->scratch[area] != NULL) {
        cudaStreamSynchronize(c->stream);
        cudaFree(c->scratch[area]);
        c->scratch[area] = NULL;
        c->scratch_bytes[area] = 0;
    }
    size_t want = (bytes + 0xfffffu) & ~(size_t)0xfffffu;
    void *p = moe_cuda_alloc(c, want);
    if (p == NULL) return NULL;
    c->scratch[area] = p;
    c->scratch_bytes[area] = want;
    return p;
}

__global__ void moe_fill_kernel(uint4 *dst4, size_t n16, uint32_t *tail, uint32_t ntail, uint32_t word) {
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    size_t stride = (size_t)gridDim.x * blockDim.x;
    uint4 v = make_uint4(word, word, word, word);
    for (; i < n16; i += stride) dst4[i] = v;
    if (blockIdx.x == 0 && threadIdx.x < ntail) tail[threadIdx.x] = word;
}

// mda_vkc_fill (src/vkc.c:803-815): whole 32-bit words.
extern "C" void moe_cuda_fill(moe_cuda_ctx_t *c, void *dst, size_t bytes, uint32_t word) {
    if (!MOE_LIVE(c)) return;
    MOE_REQUIRE(c, dst != NULL && bytes % 4 == 0 && ((uintptr_t)dst & 3) == 0, "fill: dst/bytes not word aligned");
    if (bytes == 0) return;
    uint32_t b = word & 0xffu;
    if (((word >> 8) & 0xffu) == b && ((word >> 16) & 0xffu) == b && (word >> 24) == b) {
        MOE_CUDA_TRY(c, cudaMemsetAsync(dst, (int)b, bytes, c->stream));
        return;
    }
    uintptr_t a = (uintptr_t)dst;
    size_t head = ((16 - (a & 15)) & 15);
    if (head > bytes) head = bytes;
    if (head != 0) {  // leading words up to 16-byte alignment
        moe_fill_kernel<<<1, 32, 0, c->stream>>>(NULL, 0, (uint32_t *)dst, (uint32_t)(head / 4), word);
        MOE_LAUNCHED(c);
    }
    size_t rest = bytes - head;
    size_t n16 = rest / 16;
    uint32_t ntail = (uint32_t)((rest % 16) / 4);
    uint8_t *body = (uint8_t *)dst + head;
    if (n16 != 0 || ntail != 0) {
        size_t blocks = (n16 + 255) / 256;
        if (blocks > (size_t)c->sm_count * 8) blocks = (size_t)c->sm_count * 8;
        if (blocks == 0) blocks = 1;
        moe_fill_kernel<<<(unsigned)blocks, 256, 0, c->stream>>>((uint4 *)body, n16, (uint32_t *)(body + n16 * 16), ntail, word);
        MOE_LAUNCHED(c);
    }
}

extern "C" void moe_cuda_copy(moe_cuda_ctx_t *c, void *dst, const void *src, size_t bytes) {
    if (!MOE_LIVE(c)) return;
    MOE_CUDA_TRY(c, cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToDevice, c->stream));
}

extern "C" void moe_cuda_write(moe_cuda_ctx_t *c, void *dst, const void *host_src, size_t bytes) {
    if (!MOE_LIVE(c)) return;
    MOE_CUDA_TRY(c, cudaMemcpyAsync(dst, host_src, bytes, cudaMemcpyHostToDevice, c->stream));
}

extern "C" void moe_cuda_read(moe_cuda_ctx_t *c, void *host_dst, const void *src, size_t bytes) {
    if (!MOE_LIVE(c)) return;
    MOE_CUDA_TRY(c, cudaMemcpyAsync(host_dst, src, bytes, cudaMemcpyDeviceToHost, c->stream));
    MOE_CUDA_TRY(c, cudaStreamSynchronize(c->stream));
    moe_poll_device_status(c);
}

// Enqueued device-to-host copy; the data is on the host after the next moe_cuda_flush.
extern "C" void moe_cuda_read_async(moe_cuda_ctx_t *c, void *host_dst, const void *src, size_t bytes) {
    if (!MOE_LIVE(c)) return;
    MOE_CUDA_TRY(c, cudaMemcpyAsync(host_dst, src, bytes, cudaMemcpyDeviceToHost, c->stream));
}

extern "C" void moe_cuda_flush(moe_cuda_ctx_t *c) {
    if (c == NULL || c->stream == NULL) return;
    if (c->status == MOE_OK) {
        MOE_CUDA_TRY(c, cudaStreamSynchronize(c->stream));
        moe_poll_device_status(c);
    }
}

extern "C" void moe_cuda_prof(moe_cuda_ctx_t *c, int on) {
    if (!MOE_LIVE(c)) return;
    if (on && !c->ev_made) {
        for (int i = 0; i <= MOE_PROF_STAGES; i += 1) MOE_CUDA_TRY(c, cudaEventCreate(&c->ev[i]));
        c->ev_made = true;
    }
    c->prof = on != 0;
    c->ev_valid = false;
}

extern "C" void moe_cuda_prof_read(moe_cuda_ctx_t *c, float ms[MOE_PROF_STAGES]) {
    for (int i = 0; i < MOE_PROF_STAGES; i += 1) ms[i] = 0.0f;
    if (!MOE_LIVE(c) || !c->ev_valid) return;
    MOE_CUDA_TRY(c, cudaStreamSynchronize(c->stream));  // the slices' streams have joined the context's stream
    for (int m = 0; m < (c->ev_slices > 1 ? c->ev_slices : 1); m += 1) {
        cudaEvent_t *ev = m == 0 ? c->ev : c->ev_mb[m - 1];
        for (int i = 0; i < MOE_PROF_STAGES; i += 1) {
            float t = 0.0f;
            MOE_CUDA_TRY(c, cudaEventElapsedTime(&t, ev[i], ev[i + 1]));
            ms[i] += t;
        }
    }
}

// Tensor maps: row-major fp16, boxes of 64 columns with a 128-byte swizzle, zero fill outside the tensor; never multicast.
typedef CUresult (*moe_encode_fn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);

static bool moe_encode(moe_cuda_ctx *c, CUtensorMap *out, uint32_t rank, const void *ptr, const cuuint64_t *dims,
                       const cuuint64_t *strides, const cuuint32_t *box) {
    static const cuuint32_t ones[4] = {1, 1, 1, 1};
    CUresult r = ((moe_encode_fn)c->encode_tiled)(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, rank, (void *)ptr, dims, strides, box, ones,
                                                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) moe_fail(c, MOE_ERR_CUDA, "cuTensorMapEncodeTiled failed: %d", (int)r);
    return r == CUDA_SUCCESS;
}

static uint32_t moe_tmap_hash(const void *ptr, uint64_t rows, uint64_t cols, uint32_t box_rows) {
    uint64_t h = ((uint64_t)(uintptr_t)ptr >> 4) ^ (rows << 24) ^ (cols << 40) ^ ((uint64_t)box_rows << 56);
    return (uint32_t)((h * 0x9e3779b97f4a7c15ull) >> 40);
}

static bool moe_tmap_encode_2d(moe_cuda_ctx *c, CUtensorMap *out, const void *ptr, uint64_t rows, uint64_t cols, uint32_t box_rows) {
    if (((uintptr_t)ptr & 15) != 0 || ptr == NULL || (cols * 2) % 16 != 0 || box_rows > 256 || rows == 0) {
        moe_fail(c, MOE_ERR_ARG, "tensor map: base %p rows %llu cols %llu not TMA-addressable", ptr,
                 (unsigned long long)rows, (unsigned long long)cols);
        return false;
    }
    const cuuint64_t dims[2] = {cols, rows}, strides[1] = {cols * 2};
    const cuuint32_t box[2] = {64, box_rows};
    return moe_encode(c, out, 2, ptr, dims, strides, box);
}

// One entry of `kind`: the cached one, or a new one in its place.
static bool moe_tmap_get(moe_cuda_ctx *c, CUtensorMap *out, const void *ptr, uint64_t rows, uint64_t cols, uint32_t box_rows, uint32_t kind) {
    if (!MOE_LIVE(c)) return false;
    const uint32_t set = moe_tmap_hash(ptr, rows, cols, box_rows + kind) % MOE_TMAP_SETS;
    for (uint32_t i = 0; i < MOE_TMAP_WAYS; i += 1) {
        moe_tmap_entry *t = &c->tmaps[set][i];
        if (t->ptr == ptr && t->rows == rows && t->cols == cols && t->box_rows == box_rows && t->kind == kind && ptr != NULL) {
            memcpy(out, &t->map, sizeof(*out));
            return true;
        }
    }
    if (kind == 0) {
        if (!moe_tmap_encode_2d(c, out, ptr, rows, cols, box_rows)) return false;
    } else {  // gate/up bank: rows = experts, box_rows = inter
        const cuuint64_t inter = box_rows;
        const cuuint64_t dims[4] = {cols, 2, inter, rows};
        const cuuint64_t strides[3] = {inter * cols * 2, cols * 2, 2 * inter * cols * 2};
        const cuuint32_t box[4] = {64, 2, 64, 1};
        if (!moe_encode(c, out, 4, ptr, dims, strides, box)) return false;
    }
    moe_tmap_entry *t = &c->tmaps[set][c->next_tmap[set]++ % MOE_TMAP_WAYS];
    t->ptr = ptr;
    t->rows = rows;
    t->cols = cols;
    t->box_rows = box_rows;
    t->kind = kind;
    memcpy(&t->map, out, sizeof(*out));
    return true;
}

bool moe_tmap_2d_f16(moe_cuda_ctx *c, CUtensorMap *out, const void *ptr, uint64_t rows, uint64_t cols, uint32_t box_rows) {
    return moe_tmap_get(c, out, ptr, rows, cols, box_rows, 0);
}

bool moe_tmap_gate_up_f16(moe_cuda_ctx *c, CUtensorMap *out, const void *ptr, uint32_t experts, uint32_t inter, uint32_t k) {
    if (!MOE_LIVE(c)) return false;
    if (((uintptr_t)ptr & 15) != 0 || ptr == NULL || k % 8u != 0 || inter % 64u != 0 || experts == 0) {
        moe_fail(c, MOE_ERR_ARG, "tensor map: gate/up bank %p experts %u inter %u k %u not TMA-addressable", ptr, experts, inter, k);
        return false;
    }
    return moe_tmap_get(c, out, ptr, experts, k, inter, 1);
}

bool moe_tmap_tokens_f16(moe_cuda_ctx *c, moe_xmaps *out, const void *ptr, uint64_t rows, uint64_t cols) {
    if (!MOE_LIVE(c)) return false;
    const uint32_t set = moe_tmap_hash(ptr, rows, cols, 0) % MOE_XMAP_SETS;
    for (uint32_t i = 0; i < MOE_TMAP_WAYS; i += 1) {
        moe_xmap_entry *t = &c->xmaps[set][i];
        if (t->ptr == ptr && t->rows == rows && t->cols == cols && ptr != NULL) {
            memcpy(out, &t->maps, sizeof(*out));
            return true;
        }
    }
    for (uint32_t i = 0; i < MOE_XMAP_BOXES; i += 1) {
        if (!moe_tmap_encode_2d(c, &out->m[i], ptr, rows, cols, 16u * (i + 1u))) return false;
    }
    moe_xmap_entry *t = &c->xmaps[set][c->next_xmap[set]++ % MOE_TMAP_WAYS];
    t->ptr = ptr;
    t->rows = rows;
    t->cols = cols;
    memcpy(&t->maps, out, sizeof(*out));
    return true;
}
