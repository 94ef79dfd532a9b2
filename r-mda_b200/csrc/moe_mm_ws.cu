// Grouped expert products, weight-stationary form, for the fused layer: the
// MMA's M dimension runs over weight rows (output features), its N dimension
// over the tokens of one expert.  Compared with the token-major kernel in
// moe_mm.cu (the reference's 128-row tile schedule, shader/matmul_f16_moe.comp):
//   * an expert's rows are cut into chunks of at most 256 tokens whose MMA width
//     is rounded to 16, not 128, so ragged expert sizes waste almost no tensor
//     work (the reference pads every expert to 128 rows);
//   * with PAIR = 2 two CTAs of a cluster issue one tcgen05.mma.cta_group::2
//     (M 256) over a shared token tile: each CTA loads its own 128 weight rows
//     and only half of the token tile, i.e. 32 KB instead of 48 KB of operands
//     per 64-wide K step and SM.  The loads are plain per-CTA TMA tile loads.
// D lands transposed in tensor memory (lane = feature, column = token); the
// epilogue warps turn it round through a small shared-memory tile so that global
// stores are 16 bytes wide and row-contiguous.
// SWIGLU mode: a 4-D tensor map over [expert][gate|up][inter][d] lets TMA fetch 64
// gate rows and the matching 64 up rows interleaved (row 2i = gate i, row 2i+1 =
// up i), so the two values of an output sit in neighbouring lanes of one warp and
// meet with one shuffle; silu(gate)*up (shader/qwen_elem.comp:20-31 op 0) and the
// fp16 store are the epilogue.
// Every spin on an mbarrier is bounded; on timeout the kernel records
// MOE_ERR_TIMEOUT in the context's status word and unwinds.
#include "moe_tc.cuh"

namespace {

using namespace moe_tc;

constexpr uint32_t BK = 64;
constexpr uint32_t W_BYTES = 128 * BK * 2;   // 16 KB: this CTA's 128 weight rows
constexpr uint32_t MAX_TOK = 256;            // tokens per chunk = MMA N
constexpr uint32_t WS_THREADS = 352;        // warps: 0 weight loads, 1 MMA issue, 2..5 epilogue, 6 token loads, 7..10 more loads
constexpr uint32_t NPROD = 3;               // issuing threads per operand, taking K steps in turn
constexpr uint32_t TMEM_COLS = 512;
constexpr uint32_t ET = 32;                  // tokens per epilogue step (one tcgen05.ld of 32 columns)
constexpr uint32_t PITCH_SW = 160;           // bytes per token row of the turn-round tile, SwiGLU (64 fp16 + pad)
constexpr uint32_t PITCH_F16 = 256;          // pitch of the two turn-round buffers
constexpr uint32_t PITCH_T = 80;             // bytes per token row of a warp's own tile of 32 fp16 features: eight rows meet eight bank groups
constexpr uint32_t TURN_BYTES = 2 * ET * PITCH_F16;  // two buffers

template <int PAIR>
struct Geo {
    static constexpr uint32_t X_BYTES = MAX_TOK / PAIR * BK * 2;  // this CTA's share of the token tile
    static constexpr uint32_t STAGE_BYTES = W_BYTES + X_BYTES;
    static constexpr uint32_t STAGES = PAIR == 2 ? 6 : 4;         // 192 KB of operands either way (3 stages measured only 9 % slower)
};

struct __align__(8) WsBarriers {
    uint64_t full[8];
    uint64_t empty[8];
    uint64_t tmem_full[2];
    uint64_t tmem_empty[2];
    uint32_t tmem_base;
    uint32_t abort;
};

template <int PAIR>
constexpr uint32_t ws_smem() {
    return Geo<PAIR>::STAGES * Geo<PAIR>::STAGE_BYTES + TURN_BYTES + sizeof(WsBarriers) + 1024;
}

struct WsArgs {
    void *C;
    const uint4 *chunks;       // (expert, first row, MMA width, valid rows)
    const uint32_t *n_chunks;
    uint32_t n;                // weight rows per expert (2*inter, or d)
    uint32_t k;
    uint32_t ldc;              // row stride of C in elements
    uint32_t *status;
    uint64_t wait_ns;
    // dense form (MM_DENSE): no chunk list, rows are cut into chunks of `per` (a multiple of 16)
    uint32_t rows, per;
    uint32_t splits, ksplit;   // K split `splits` ways, ksplit K steps each; the first one's sums go to C,
    float *part;               // split p's to part + (p - 1) * rows * ldc
    const uint32_t *tiles;     // or NULL: expert of each 128-row tile, >= experts: the tile is skipped (per divides 128)
    uint32_t experts;
    const uint32_t *amax;      // scale slots (power of two) of both operands
    uint32_t sa, sb;
};
// C fp32 = X * W^T over all rows, for moe_cuda_dense and small moe_cuda_mm calls
constexpr int MM_DENSE = 3;

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t map_to_cta(uint32_t saddr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
    return r;
}
// Relaxed: a release at cluster scope waits until the warp's global stores have been performed (3100 cycles per item of
// the down product).  What the barrier hands over is the accumulator, whose reads are complete (tcgen05.wait::ld) and
// ordered by tcgen05.fence::before_thread_sync.
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// TMA tile loads issued by either CTA of a pair; the completion bytes are counted
// on the barrier at cluster address `bar` (the leader's).  Not multicast.
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap *map, uint32_t bar, int32_t c0, int32_t c1) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        :
        : "r"(dst), "l"((uint64_t)map), "r"(bar), "r"(c0), "r"(c1)
        : "memory");
}
__device__ __forceinline__ void tma_load_4d_pair(uint32_t dst, const CUtensorMap *map, uint32_t bar, int32_t c0, int32_t c1,
                                                 int32_t c2, int32_t c3) {
    asm volatile(
        "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
        :
        : "r"(dst), "l"((uint64_t)map), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
        : "memory");
}
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap *map, uint32_t bar, int32_t c0, int32_t c1, int32_t c2,
                                            int32_t c3) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
        :
        : "r"(dst), "l"((uint64_t)map), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
        : "memory");
}
template <int PAIR>
__device__ __forceinline__ void tma_2d(uint32_t dst, const CUtensorMap *map, uint32_t bar, int32_t c0, int32_t c1) {
    if (PAIR == 2) tma_load_2d_pair(dst, map, bar, c0, c1);
    else tma_load_2d(dst, map, bar, c0, c1);
}
template <int PAIR>
__device__ __forceinline__ void tma_4d(uint32_t dst, const CUtensorMap *map, uint32_t bar, int32_t c0, int32_t c1, int32_t c2,
                                       int32_t c3) {
    if (PAIR == 2) tma_load_4d_pair(dst, map, bar, c0, c1, c2, c3);
    else tma_load_4d(dst, map, bar, c0, c1, c2, c3);
}
__device__ __forceinline__ void umma_f16_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accum) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
        :
        : "r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accum)
        : "memory");
}
// One commit that arrives on the barrier at the same shared-memory offset in both CTAs of the pair.
__device__ __forceinline__ void umma_commit_both(uint32_t local_bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(local_bar),
                 "h"((uint16_t)3)
                 : "memory");
}
// All 128 epilogue threads agree on whether to go on (named barrier 1).
__device__ __forceinline__ bool epi_all(bool ok) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "bar.red.and.pred q, 1, 128, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}\n"
        : "=r"(r)
        : "r"(ok ? 1u : 0u)
        : "memory");
    return r != 0;
}
__device__ __forceinline__ void epi_sync() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

// Token rows per TMA box: the smallest multiple of 16 up to 128 that covers what is left.
__device__ __forceinline__ uint32_t x_box_rows(uint32_t left) { return left > 112u ? 128u : (left + 15u) & ~15u; }
__device__ __forceinline__ uint32_t x_rows_loaded(uint32_t half) {
    uint32_t rows = 0;
    for (uint32_t done = 0; done < half; done += x_box_rows(half - done)) rows += x_box_rows(half - done);
    return rows;
}
struct WsItem {
    uint32_t e, row0, ntok, nvalid, ft, kb0, kb1, split;
};

// False: nothing to do for this item (dense form: an unused row tile).
template <int MODE>
__device__ __forceinline__ bool ws_item(const WsArgs &a, uint32_t w, uint32_t ft_count, uint32_t kblocks, WsItem &it) {
    if (MODE == MM_DENSE) {
        // splits, then chunks, then feature tiles: CTAs that run together share weight tiles, so that a weight
        // matrix larger than L2 (a vocabulary) comes from HBM once
        const uint32_t nch = (a.rows + a.per - 1u) / a.per;
        const uint32_t q = w / a.splits;
        it.split = w - q * a.splits;
        it.ft = q / nch;
        it.row0 = (q - it.ft * nch) * a.per;
        it.nvalid = min(a.per, a.rows - it.row0);
        it.ntok = (it.nvalid + 15u) & ~15u;
        it.kb0 = it.split * a.ksplit;
        it.kb1 = min(it.kb0 + a.ksplit, kblocks);
        it.e = a.tiles != NULL ? a.tiles[it.row0 / MOE_TILE] : 0u;
        return it.e < a.experts;
    }
    it.kb0 = 0;
    it.kb1 = kblocks;
    uint32_t c = w / ft_count;
    it.ft = w - c * ft_count;
    uint4 ch = a.chunks[c];
    it.e = ch.x;
    it.row0 = ch.y;
    it.ntok = ch.z;
    it.nvalid = ch.w;
    return true;
}

template <int MODE, int PAIR>
__global__ void __launch_bounds__(WS_THREADS, 1)
moe_mm_ws_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ moe_xmaps tmX, WsArgs a) {
    using G = Geo<PAIR>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t *turn = smem + G::STAGES * G::STAGE_BYTES;
    WsBarriers *bars = reinterpret_cast<WsBarriers *>(turn + TURN_BYTES);
    const uint32_t stage0 = smem_u32(smem);
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t rank = PAIR == 2 ? cluster_rank() : 0u;
    volatile uint32_t *abort = &bars->abort;

    // feature tiles: SwiGLU 64 outputs (64 gate + 64 up rows) per CTA, otherwise 128 weight rows per CTA
    const uint32_t ft_count = MODE == MOE_MM_SWIGLU_F16 ? (a.n / 2u) / (64u * PAIR) : (a.n + 128u * PAIR - 1u) / (128u * PAIR);
    const uint32_t kblocks = (a.k + BK - 1) / BK;
    const uint32_t cluster_id = blockIdx.x / PAIR, n_clusters = gridDim.x / PAIR;

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < G::STAGES; s += 1) {
            mbar_init(smem_u32(&bars->full[s]), 1);
            mbar_init(smem_u32(&bars->empty[s]), 1);
        }
        for (uint32_t s = 0; s < 2; s += 1) {
            mbar_init(smem_u32(&bars->tmem_full[s]), 1);
            mbar_init(smem_u32(&bars->tmem_empty[s]), 4 * PAIR);  // one arrival per epilogue warp of each CTA
        }
        bars->abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        if (PAIR == 2) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&bars->tmem_base)),
                         "r"(TMEM_COLS)
                         : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&bars->tmem_base)),
                         "r"(TMEM_COLS)
                         : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    tc_fence_before();
    __syncthreads();
    if (PAIR == 2) cluster_sync_all();  // the peer's barriers exist before anything is sent to them
    tc_fence_after();
    moe_pdl_begin();
    const uint32_t total = MODE == MM_DENSE ? (a.rows + a.per - 1u) / a.per * ft_count * a.splits : *a.n_chunks * ft_count;
    const uint32_t tmem_base = bars->tmem_base;

    if (warp == 0 || warp >= 6) {
        // ---------------- TMA producers (both CTAs) ----------------
        // One thread gets at most one tile load issued per ~300 ns, whatever its size (measured: 4 KB to 32 KB
        // boxes, tiled or untiled, L2 or HBM source; threads of different warps add up).  A K step of the
        // tensor pipe is shorter than that, so each operand has NPROD issuing threads that take K steps in
        // turn: warps 0, 7, 9 load weight tiles, warps 6, 8, 10 token tiles.  All follow the same stage ring;
        // the completion bytes of the four loads of a stage (two CTAs x two operands) are counted on the
        // leader's full barrier, whose one arrival is the weight producer's expect_tx.
        if (lane == 0) {
            const bool wprod = warp == 0 || (warp >= 7 && (warp & 1u) != 0);
            const uint32_t turn_of = warp < 7 ? 0u : (warp - 5u) / 2u;  // 0, 1, 2: which K steps this thread takes
            uint32_t s = 0, ph = 0, issued = 0, last_par = 0, gstep = 0;
            bool ok = true;
            for (uint32_t w = cluster_id; w < total && ok; w += n_clusters) {
                WsItem it;
                if (!ws_item<MODE>(a, w, ft_count, kblocks, it)) continue;
                const uint32_t half = it.ntok / PAIR;            // token rows this CTA loads
                const uint32_t xbytes = x_rows_loaded(half) * (BK * 2u);
                const int32_t f0 = (int32_t)((it.ft * PAIR + rank) * (MODE == MOE_MM_SWIGLU_F16 ? 64u : 128u));
                const int32_t xrow = (int32_t)(it.row0 + rank * half);
                for (uint32_t kb = it.kb0; kb < it.kb1; kb += 1, gstep += 1) {
                    if (gstep % NPROD != turn_of) continue;
                    s = gstep % G::STAGES;
                    ph = (gstep / G::STAGES) & 1u;
                    if (!mbar_wait(smem_u32(&bars->empty[s]), ph ^ 1u, abort, a.status, wprod ? 11 : 15, a.wait_ns)) {
                        ok = false;
                        break;
                    }
                    const uint32_t base = stage0 + s * G::STAGE_BYTES;
                    const int32_t kc = (int32_t)(kb * BK);
                    const uint32_t full = PAIR == 2 ? map_to_cta(smem_u32(&bars->full[s]), 0) : smem_u32(&bars->full[s]);
                    if (wprod) {
                        if (rank == 0) mbar_expect_tx(smem_u32(&bars->full[s]), (uint32_t)PAIR * (W_BYTES + xbytes));
                        if (MODE == MOE_MM_SWIGLU_F16) tma_4d<PAIR>(base, &tmW, full, kc, 0, f0, (int32_t)it.e);
                        else tma_2d<PAIR>(base, &tmW, full, kc, (int32_t)(it.e * a.n) + f0);
                    } else {
                        uint32_t done = 0;
                        while (done < half) {  // boxes of 16, 32, ... 128 token rows: at most 15 rows more than needed
                            const uint32_t rows = x_box_rows(half - done);
                            tma_2d<PAIR>(base + W_BYTES + done * (BK * 2u), &tmX.m[rows / 16u - 1u], full, kc, xrow + (int32_t)done);
                            done += rows;
                        }
                    }
                    issued |= 1u << s;
                    last_par = (last_par & ~(1u << s)) | (ph << s);
                }
            }
            if (!ok && rank == 0 && wprod) {
                for (uint32_t q = 0; q < G::STAGES; q += 1) {  // bounded wait for copies in flight
                    if (((issued >> q) & 1u) == 0) continue;
                    for (uint32_t spin = 0; spin < (1u << 16); spin += 1) {
                        if (mbar_try_wait(smem_u32(&bars->full[q]), (last_par >> q) & 1u)) break;
                    }
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ---------------- MMA issuer (leader CTA only) ----------------
        // The whole warp runs the loop, so that barrier addresses and descriptors are warp-uniform values, and one
        // elected lane issues; one look at the full barriers covers the whole ring (mbar_ring_wait).
        if (rank == 0) {
            uint32_t gstep = 0, n_item = 0, ready = 0;
            bool ok = true;
            for (uint32_t w = cluster_id; w < total && ok; w += n_clusters) {
                WsItem it;
                if (!ws_item<MODE>(a, w, ft_count, kblocks, it)) continue;
                const uint32_t as = n_item & 1u, aph = (n_item >> 1) & 1u;
                if (!mbar_wait(smem_u32(&bars->tmem_empty[as]), aph ^ 1u, abort, a.status, 12, a.wait_ns)) break;
                tc_fence_after();
                const uint32_t tmem_d = tmem_base + as * MAX_TOK;
                const uint32_t idesc = umma_idesc(128u * PAIR, it.ntok);
                for (uint32_t kb = it.kb0; kb < it.kb1; kb += 1, gstep += 1) {
                    const uint32_t s = gstep % G::STAGES;
                    if (((ready >> s) & 1u) == 0 &&
                        !mbar_ring_wait<G::STAGES>(bars->full, gstep, ready, abort, a.status, 13, a.wait_ns)) {
                        ok = false;
                        break;
                    }
                    ready &= ~(1u << s);
                    tc_fence_after();
                    const uint32_t base = stage0 + s * G::STAGE_BYTES;
                    const uint64_t ad = umma_desc(base), bd = umma_desc(base + W_BYTES);
                    if (elect_one()) {
#pragma unroll
                        for (uint32_t kk = 0; kk < BK / 16; kk += 1) {
                            if (PAIR == 2) umma_f16_pair(tmem_d, ad + 2ull * kk, bd + 2ull * kk, idesc, ((kb - it.kb0) | kk) != 0 ? 1u : 0u);
                            else umma_f16(tmem_d, ad + 2ull * kk, bd + 2ull * kk, idesc, ((kb - it.kb0) | kk) != 0 ? 1u : 0u);
                        }
                        if (PAIR == 2) umma_commit_both(smem_u32(&bars->empty[s]));  // frees the stage in both CTAs
                        else umma_commit(smem_u32(&bars->empty[s]));
                    }
                    __syncwarp();
                }
                if (ok && elect_one()) {
                    if (PAIR == 2) umma_commit_both(smem_u32(&bars->tmem_full[as]));
                    else umma_commit(smem_u32(&bars->tmem_full[as]));
                }
                __syncwarp();
                n_item += 1;
            }
        }
        __syncwarp();
    } else {
        // ---------------- epilogue (warps 2..5 of both CTAs) ----------------
        const uint32_t q = warp & 3u;    // TMEM lane quarter this warp may read
        const uint32_t ew = warp - 2u;   // 0..3: which rows of the turn-round tile this warp stores
        const uint32_t empty_leader = PAIR == 2 ? map_to_cta(smem_u32(&bars->tmem_empty[0]), 0) : smem_u32(&bars->tmem_empty[0]);
        uint32_t n_item = 0, tb = 0;
        float scale = 1.0f;  // a power of two: partial sums scaled one by one add up to the scaled sum
        if (MODE == MM_DENSE) scale = 1.0f / (moe_slot_scale(a.amax, a.sa) * moe_slot_scale(a.amax, a.sb));
        for (uint32_t w = cluster_id; w < total; w += n_clusters) {
            WsItem it;
            if (!ws_item<MODE>(a, w, ft_count, kblocks, it)) continue;
            const uint32_t as = n_item & 1u, aph = (n_item >> 1) & 1u;
            bool ok = true;
            if (lane == 0) ok = mbar_wait(smem_u32(&bars->tmem_full[as]), aph, abort, a.status, 14, a.wait_ns);
            if (!epi_all(ok)) break;
            tc_fence_after();
            const uint32_t taddr = tmem_base + as * MAX_TOK + ((q * 32u) << 16);
            const uint32_t nch = (it.ntok + ET - 1u) / ET;
            if (MODE == MOE_MM_SWIGLU_F16) {
                // lane 2i holds gate feature i of this warp's 16, lane 2i+1 the matching up feature
                const uint32_t fl = q * 16u + (lane >> 1);
                const uint32_t odd = lane & 1u;
                __half *out = reinterpret_cast<__half *>(a.C) + (size_t)it.row0 * a.ldc + (it.ft * PAIR + rank) * 64u + (lane & 7u) * 8u;
#pragma unroll 1
                for (uint32_t cch = 0; cch < nch; cch += 1) {
                    uint32_t v[32];
                    tmem_ld32(taddr + cch * ET, v);
                    tmem_ld_wait();
                    uint8_t *tp = turn + tb * ET * PITCH_F16;
                    __half *mine = reinterpret_cast<__half *>(tp + odd * PITCH_SW) + fl;
#pragma unroll
                    for (uint32_t jj = 0; jj < 16; jj += 1) {
                        const uint32_t send = odd ? v[2 * jj] : v[2 * jj + 1];
                        const uint32_t recv = __shfl_xor_sync(0xffffffffu, send, 1);
                        const float g = __uint_as_float(odd ? recv : v[2 * jj]);
                        const float u = __uint_as_float(odd ? v[2 * jj + 1] : recv);
                        const float h = __fdividef(g, 1.0f + __expf(-g)) * u;
                        mine[jj * (2u * PITCH_SW / 2u)] = __float2half_rn(h);  // token 2jj + odd
                    }
                    epi_sync();
                    const uint32_t t0c = cch * ET;
#pragma unroll
                    for (uint32_t i = 0; i < 2; i += 1) {
                        const uint32_t r = ew * 8u + i * 4u + (lane >> 3);
                        if (t0c + r < it.nvalid) {
                            const uint4 val = *reinterpret_cast<const uint4 *>(tp + r * PITCH_SW + (lane & 7u) * 16u);
                            *reinterpret_cast<uint4 *>(out + (size_t)(t0c + r) * a.ldc) = val;
                        }
                    }
                    tb ^= 1u;
                }
            } else if (MODE == MOE_MM_F16) {
                // Each warp turns its own 32 features x 32 tokens round: fragments as the tensor core's 16x256b loads
                // give them (a lane: two neighbouring tokens of features lane/4 and lane/4 + 8), packed to fp16, go
                // through stmatrix.trans, so that a token's 32 features lie in a row of shared memory; no barrier
                // with the other warps.  With the relaxed arrival below, 16384 x 2048 outputs of top-10 of 512 experts, K 512:
                // 526 us with 2-byte stores into a tile of all four warps, 429 us this way; K 768, 4096 x top-8: 126, 115.
                uint8_t *tp = turn + ew * (ET * PITCH_T);
                const uint32_t st_addr = smem_u32(tp) + (lane & 7u) * PITCH_T + (lane >> 3) * 16u;
                const uint8_t *ld = tp + (lane >> 2) * PITCH_T + (lane & 3u) * 16u;
                __half *out = reinterpret_cast<__half *>(a.C) + (size_t)(it.row0 + (lane >> 2)) * a.ldc +
                              (it.ft * PAIR + rank) * 128u + q * 32u + (lane & 3u) * 8u;
#pragma unroll 1
                for (uint32_t cch = 0; cch < nch; cch += 1) {
                    uint32_t lo[16], hi[16];  // features 0..15 and 16..31 of this warp
                    tmem_ld_16x256b_x4(taddr + cch * ET, lo);
                    tmem_ld_16x256b_x4(taddr + (16u << 16) + cch * ET, hi);
                    tmem_ld_wait();
                    __syncwarp();  // the previous chunk has been read
#pragma unroll
                    for (uint32_t i = 0; i < 4; i += 1) {
                        stmatrix_x4_trans(st_addr + i * 8u * PITCH_T,
                                          pack_h2(__uint_as_float(lo[4 * i]), __uint_as_float(lo[4 * i + 1])),
                                          pack_h2(__uint_as_float(lo[4 * i + 2]), __uint_as_float(lo[4 * i + 3])),
                                          pack_h2(__uint_as_float(hi[4 * i]), __uint_as_float(hi[4 * i + 1])),
                                          pack_h2(__uint_as_float(hi[4 * i + 2]), __uint_as_float(hi[4 * i + 3])));
                    }
                    __syncwarp();
                    const uint32_t t0 = cch * ET + (lane >> 2);
#pragma unroll
                    for (uint32_t i = 0; i < 4; i += 1) {
                        const uint4 val = *reinterpret_cast<const uint4 *>(ld + i * 8u * PITCH_T);
                        if (t0 + i * 8u < it.nvalid) *reinterpret_cast<uint4 *>(out + (size_t)(cch * ET + i * 8u) * a.ldc) = val;
                    }
                }
            } else {
                // fp32 output: 32 lanes = 32 neighbouring features = one 128-byte piece of a token's row per store
                const uint32_t cfeat = (it.ft * PAIR + rank) * 128u + q * 32u + lane;
                // dense form: the last pair may reach beyond n (n is a multiple of 128, not of 256)
                const uint32_t nvalid = MODE == MM_DENSE && cfeat >= a.n ? 0u : it.nvalid;
                float *C = reinterpret_cast<float *>(a.C);
                if (MODE == MM_DENSE && it.split != 0u) C = a.part + (size_t)(it.split - 1u) * a.rows * a.ldc;
#pragma unroll 1
                for (uint32_t cch = 0; cch < nch; cch += 1) {
                    uint32_t v[32];
                    tmem_ld32(taddr + cch * ET, v);
                    tmem_ld_wait();
                    const uint32_t t0c = cch * ET;
                    float *out = C + (size_t)(it.row0 + t0c) * a.ldc + cfeat;
                    if (t0c + 32u <= nvalid) {  // one test for the whole chunk: a test per store costs ten times the stores
#pragma unroll
                        for (uint32_t j = 0; j < 32; j += 1) {
                            *out = MODE == MM_DENSE ? __uint_as_float(v[j]) * scale : __uint_as_float(v[j]);
                            out += a.ldc;
                        }
                    } else {
#pragma unroll
                        for (uint32_t j = 0; j < 32; j += 1) {
                            if (t0c + j < nvalid) out[(size_t)j * a.ldc] = MODE == MM_DENSE ? __uint_as_float(v[j]) * scale : __uint_as_float(v[j]);
                        }
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                if (PAIR == 2) mbar_arrive_cluster(empty_leader + as * 8u);
                else mbar_arrive(empty_leader + as * 8u);
            }
            n_item += 1;
        }
    }
    tc_fence_before();
    __syncthreads();
    if (PAIR == 2) cluster_sync_all();  // neither CTA leaves while the other may still touch its memory
    if (warp == 1) {
        tc_fence_after();
        if (PAIR == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
}

// The chunk list as a kernel of its own (expert-parallel layer: the counts come from the plan): one block, thread =
// expert.  The single-GPU layer builds the same list in the last block of its column scan.
static_assert(MAX_TOK == MOE_CHUNK_TOK, "the chunk list is cut for the MMA width of this kernel");
__global__ void __launch_bounds__(512)
moe_chunk_kernel(const uint32_t *__restrict__ count, const uint32_t *__restrict__ off, uint32_t experts,
                 uint4 *__restrict__ chunks, uint32_t *__restrict__ n_chunks, uint32_t max_chunks) {
    moe_chunk_body(count, off, experts, chunks, n_chunks, max_chunks);
}

// C += the partial products of the other splits of K, in split order.  n and with it every row is a multiple of four.
__global__ void __launch_bounds__(256)
moe_ksum_kernel(const float4 *part, float4 *C, uint32_t total4, uint32_t splits) {
    moe_pdl_begin();
    const uint32_t i = blockIdx.x * 256u + threadIdx.x;
    if (i >= total4) return;
    float4 acc = C[i];
    for (uint32_t p = 1; p < splits; p += 1) {
        const float4 v = __ldcg(part + (size_t)(p - 1u) * total4 + i);
        acc.x += v.x;
        acc.y += v.y;
        acc.z += v.z;
        acc.w += v.w;
    }
    C[i] = acc;
}

template <int MODE, int PAIR>
void ws_launch(moe_cuda_ctx *c, const CUtensorMap &tmW, const moe_xmaps &tmX, WsArgs &a, uint32_t grid) {
    int slot = MODE * 2 + (PAIR - 1);
    if (!c->sw_attr_set[slot]) {
        MOE_CUDA_TRY(c, cudaFuncSetAttribute(moe_mm_ws_kernel<MODE, PAIR>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)ws_smem<PAIR>()));
        c->sw_attr_set[slot] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid, 1, 1);
    cfg.blockDim = dim3(WS_THREADS, 1, 1);
    cfg.dynamicSmemBytes = ws_smem<PAIR>();
    cfg.stream = c->stream;
    cudaLaunchAttribute attr[2];  // the second as in moe_run
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = PAIR;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = c->ep == NULL ? 2 : 1;
    MOE_CUDA_TRY(c, cudaLaunchKernelEx(&cfg, moe_mm_ws_kernel<MODE, PAIR>, tmW, tmX, a));
    c->launches += 1;
}

}  // namespace

void moe_launch_chunks(moe_cuda_ctx *c, const uint32_t *count, const uint32_t *off, uint32_t experts, void *chunks,
                       uint32_t *n_chunks, uint32_t max_chunks) {
    if (!MOE_LIVE(c)) return;
    MOE_REQUIRE(c, experts >= 1 && experts <= MOE_MAX_EXPERTS, "chunks: experts %u outside 1..512", experts);
    moe_chunk_kernel<<<1, 512, 0, c->stream>>>(count, off, experts, (uint4 *)chunks, n_chunks, max_chunks);
    MOE_LAUNCHED(c);
}

// X [rows_x x k] fp16 token rows, W [experts_in_W][n x k] fp16, C token-major with row stride ldc.
void moe_launch_mm_ws(moe_cuda_ctx *c, int mode, int pair, const void *X, uint32_t rows_x, const void *W,
                      uint32_t experts_in_W, void *C, uint32_t ldc, const void *chunks, const uint32_t *n_chunks,
                      uint32_t max_chunks, uint32_t n, uint32_t k) {
    if (!MOE_LIVE(c)) return;
    MOE_REQUIRE(c, X != NULL && W != NULL && C != NULL && chunks != NULL && n_chunks != NULL, "mm_ws: null buffer");
    MOE_REQUIRE(c, pair == 1 || pair == 2, "mm_ws: pair %d", pair);
    MOE_REQUIRE(c, n % (128u * (uint32_t)pair) == 0, "mm_ws: n %u does not tile into %d x 128 weight rows", n, pair);
    MOE_REQUIRE(c, k % 8u == 0 && k >= 8u && rows_x >= 1, "mm_ws: k %u", k);
    MOE_REQUIRE(c, (uint64_t)experts_in_W * n < (1ull << 31), "mm_ws: expert count");
    MOE_REQUIRE(c, ((uintptr_t)C & 15) == 0 && (mode == MOE_MM_F32 || ldc % 8u == 0), "mm_ws: C not 16-byte addressable");
    CUtensorMap tmW;
    if (mode == MOE_MM_SWIGLU_F16 ? !moe_tmap_gate_up_f16(c, &tmW, W, experts_in_W, n / 2u, k)
                                  : !moe_tmap_2d_f16(c, &tmW, W, (uint64_t)experts_in_W * n, k, 128)) return;
    moe_xmaps tmX;
    if (!moe_tmap_tokens_f16(c, &tmX, X, rows_x, k)) return;
    WsArgs a = {};
    a.C = C;
    a.chunks = (const uint4 *)chunks;
    a.n_chunks = n_chunks;
    a.n = n;
    a.k = k;
    a.ldc = ldc;
    a.status = c->dev_status_dev;
    a.wait_ns = c->wait_ns;
    uint32_t ft = mode == MOE_MM_SWIGLU_F16 ? (n / 2u) / (64u * (uint32_t)pair) : n / (128u * (uint32_t)pair);
    uint64_t total = (uint64_t)max_chunks * ft * (uint32_t)pair;
    uint32_t sms = (uint32_t)c->sm_count / (uint32_t)pair * (uint32_t)pair;
    uint32_t grid = total < sms ? (uint32_t)total : sms;
#define WS_CASE(M, P)                                      \
    if (mode == M && pair == P) {                          \
        ws_launch<M, P>(c, tmW, tmX, a, grid);             \
        return;                                            \
    }
    WS_CASE(MOE_MM_SWIGLU_F16, 1)
    WS_CASE(MOE_MM_SWIGLU_F16, 2)
    WS_CASE(MOE_MM_F16, 1)
    WS_CASE(MOE_MM_F16, 2)
    WS_CASE(MOE_MM_F32, 1)
    WS_CASE(MOE_MM_F32, 2)
#undef WS_CASE
}

namespace {
// Rows per item and K splits of the dense form: the pair with the least estimated time.  Unit: 128 bytes loaded into
// an SM (1.8 ns at the 70 B/ns that an SM gets from L2).  A K step brings 128 weight rows and half of the item's token
// rows of 128 bytes; an epilogue stores 512 bytes per token and is hidden but for the last one; a split costs a second
// launch (4 us) and its partial sums a write and a read through L2 (5 TB/s).  Splits whose sums beside C do not fit the
// context's work area are not taken: nothing is allocated here.  The most that any shape tried asks for is 69 MiB.
// 3001 x 384, K 8192, one call after another: 26 us as 3 splits against 64 us whole on the token-major kernel; 384 x 384:
// 12 against 64 us.
void ws_dense_plan(WsArgs &a, uint32_t rows, uint32_t n, uint32_t ft, uint32_t kblocks, uint32_t clusters, bool tiled, size_t work_bytes) {
    const uint32_t nch0 = (rows + MAX_TOK - 1u) / MAX_TOK;
    uint64_t best = ~0ull;
    for (uint32_t i = 0; i < (tiled ? 3u : 4u); i += 1) {
        // tile schedule given: parts of its 128-row tiles; else the fewest chunks, and finer cuts where these are few
        const uint32_t nch = nch0 * (i + 1u);
        const uint32_t per = tiled ? MOE_TILE >> i : ((rows + nch - 1u) / nch + 15u) & ~15u;
        const uint64_t items = (uint64_t)((rows + per - 1u) / per) * ft;
        for (uint32_t s = 1; s <= (tiled ? 1u : 32u) && (s == 1 || s * 4u <= kblocks); s += 1) {
            const uint32_t ks = (kblocks + s - 1u) / s;
            const uint64_t waves = (items * s + clusters - 1u) / clusters;
            uint64_t t = waves * ks * (128u + per / 2u) + per * 4u;
            if (s > 1) t += 2200u + (uint64_t)s * rows * n * 8u / 9000u;
            const uint32_t splits = (kblocks + ks - 1u) / ks;  // no empty split
            if (t < best && (uint64_t)(splits - 1u) * rows * n * 4u <= work_bytes) {
                best = t;
                a.per = per;
                a.ksplit = ks;
                a.splits = splits;
            }
            if (items * s >= 4u * (uint64_t)clusters) break;  // the last wave no longer matters
        }
    }
}
}  // namespace

// Dense product on the same kernel, pairs of CTAs only: C[rows x n] = X[rows x k] * W[e][n x k]^T / scales, where e is 0
// or, with `tiles`, the expert of the 128-row tile.
//   tiles == NULL: chunks of up to 256 rows; K may be split, the fp32 partial sums (the first split's in C, the others' in
//     the context's work area) are then added in split order by a second kernel.
//   tiles != NULL: chunks of 128, 64 or 32 rows, K whole, no scratch.
void moe_launch_mm_dense(moe_cuda_ctx *c, const void *X, const void *W, float *C, const uint32_t *amax, const uint32_t *tiles,
                         uint32_t rows, uint32_t n, uint32_t k, uint32_t sa, uint32_t sb, uint32_t experts_in_W) {
    if (!MOE_LIVE(c)) return;
    MOE_REQUIRE(c, X != NULL && W != NULL && C != NULL, "mm_dense: null buffer");
    MOE_REQUIRE(c, rows >= 1 && n % 128u == 0 && n >= 128u && k % 8u == 0 && k >= 8u, "mm_dense: rows %u n %u k %u", rows, n, k);
    MOE_REQUIRE(c, experts_in_W >= 1 && (uint64_t)experts_in_W * n < (1ull << 31) && rows < (1u << 31), "mm_dense: size");
    MOE_REQUIRE(c, (sa == MDA_PC_NO_SLOT && sb == MDA_PC_NO_SLOT) || amax != NULL, "mm_dense: scale slot without amax");
    MOE_REQUIRE(c, ((uintptr_t)C & 15) == 0, "mm_dense: C not 16-byte aligned");
    CUtensorMap tmW;
    moe_xmaps tmX;
    if (!moe_tmap_2d_f16(c, &tmW, W, (uint64_t)experts_in_W * n, k, 128) || !moe_tmap_tokens_f16(c, &tmX, X, rows, k)) return;
    const uint32_t clusters = (uint32_t)c->sm_count / 2u, ft = (n + 255u) / 256u, kblocks = (k + BK - 1u) / BK;
    WsArgs a = {};
    ws_dense_plan(a, rows, n, ft, kblocks, clusters, tiles != NULL, c->work_bytes);
    a.C = C;
    a.part = (float *)c->work;
    a.n = n;
    a.k = k;
    a.ldc = n;
    a.rows = rows;
    a.tiles = tiles;
    a.experts = experts_in_W;
    a.amax = amax;
    a.sa = sa;
    a.sb = sb;
    a.status = c->dev_status_dev;
    a.wait_ns = c->wait_ns;
    const uint64_t total = (uint64_t)((rows + a.per - 1u) / a.per) * ft * a.splits;
    MOE_REQUIRE(c, total < (1ull << 31), "mm_dense: too many tiles");
    ws_launch<MM_DENSE, 2>(c, tmW, tmX, a, (uint32_t)(total < clusters ? total : clusters) * 2u);
    if (a.splits > 1 && MOE_LIVE(c)) {
        const uint32_t total4 = rows * (n / 4u);
        moe_run(c, moe_ksum_kernel, (total4 + 255u) / 256u, 256, 0, (const float4 *)a.part, (float4 *)C, total4, a.splits);
        MOE_LAUNCHED(c);
    }
}
