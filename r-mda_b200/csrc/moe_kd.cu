// The teacher's distillation sink (shader/kd_bytes.comp; call mda_teach_sink,
// src/teach.c:108-128): next-token logits over a byte-level vocabulary become
// per-byte distributions along the true continuation.  For depth l < nd, among
// the tokens longer than l bytes that agree with the continuation on its first
// l bytes: the probability that byte l is the true one (entry 0) and the seven
// most probable other bytes (entries 1..7), each packed as byte | fp16(p) << 16.
//
// Three kernels per call:
//   sort   every chunk of 768 tokens is ordered by its first two bytes, and the rows by their
//          continuation's first byte;
//   mass   one sweep over the logits: for every row the exponentials summed by
//          first byte, and, within the row's own first byte, by second byte;
//   rows   the partial sums of a row put together; only the tokens that share the
//          continuation's first two bytes (a few per cent of a sub-word
//          vocabulary, found in the sorted chunks) are looked at one by one for
//          the depths from 2 on; totals and the top-7 selection.
// The shader adds each token into a shared-memory bin of its row (:122-125) in two
// passes over the row (maximum, then masses).  Here the sweep turns the tile round:
// a block holds 32 rows x 768 tokens of exponentials in shared memory, a lane
// owns a row and a warp walks a piece of the chunk in sorted order.  The order is
// the same for all rows, so where a run of equal bytes ends is the same for the
// whole warp: masses add up in a register, and one add per run and row leaves it.
#include <stddef.h>

#include "moe_common.cuh"

#define KD_D 16u        // MDA_KD_DEPTH, src/kd.h:11
#define KD_K 8u         // MDA_KD_K, src/kd.h:12
#define KD_CHUNK 768u   // tokens per sorted chunk: a tile of 32 rows of them fits an SM twice
#define KD_SORTED 1024u // entries of the sorting network
#define KD_ROWS 32u     // rows per block of the sweep, one per lane
#define KD_THREADS 512u
#define KD_RPW (KD_ROWS * 32u / KD_THREADS)  // rows a warp fetches
#define KD_PITCH (KD_ROWS + 1u)  // words per token of the tile and per bin: no bank conflicts either way
#define KD_BINS 512u    // per row: 256 by first byte, 256 by second byte behind the row's first byte
#define KD_RTHREADS 512u
#define KD_RWARPS (KD_RTHREADS / 32u)
#define KD_RU 2u        // tokens a lane of the last kernel has in flight
#define KD_MAX_SPLITS 256u  // at most one per thread of the last kernel

// A sorted chunk's entry: token's index in the chunk, then the sort key, so that the whole word is the sort's key.
// Tokens of one byte come before the longer ones of the same first byte; tokens without bytes come last.
// After the sort the four top bits hold the number of bytes behind the first one.
#define KD_IDX_BITS 10u
#define KD_IDX_MASK 1023u
#define KD_LEN_SHIFT 28u
#define KD_KEY_MASK ((1u << KD_LEN_SHIFT) - 1u)
__device__ __forceinline__ uint32_t kd_key2(uint32_t b0, uint32_t b1) { return b0 << 9 | 1u << 8 | b1; }
#define KD_NOKEY (1u << 17)

__device__ __forceinline__ uint32_t kd_byte_at(const uint32_t (&w)[4], uint32_t i) {  // :26-28
    const uint32_t lo = i < 4u ? w[0] : w[1], hi = i < 12u ? w[2] : w[3];  // selects: an indexed array would live in memory
    return ((i < 8u ? lo : hi) >> ((i & 3u) * 8u)) & 0xffu;
}

// :30-39: index of the first of the 16 bytes in which a and b differ, or 16
__device__ __forceinline__ uint32_t kd_common_prefix(const uint32_t (&a)[4], const uint32_t (&b)[4]) {
    uint32_t n = 16u;
#pragma unroll
    for (int i = 3; i >= 0; i -= 1) {
        const uint32_t x = a[i] ^ b[i];
        if (x != 0u) n = (uint32_t)i * 4u + ((uint32_t)__ffs((int)x) - 1u) / 8u;
    }
    return n;
}

__device__ __forceinline__ uint32_t kd_pack_entry(uint32_t b, float p) {  // :70-72
    return b | ((uint32_t)__half_as_ushort(__float2half_rn(p)) << 16);
}

// The block behind them: the rows of a batch in order of their continuation's first byte, so that the 32 rows of a block of the sweep
// share few first bytes and most runs of the sweep end at a first byte only.
#define KD_SORT_THREADS (KD_SORTED / 8u)
__device__ __forceinline__ void kd_order_rows(uint32_t *s, const uint32_t *cont, uint32_t *row_map, uint32_t rows) {
    for (uint32_t i = threadIdx.x; i < 256u; i += KD_SORT_THREADS) s[i] = 0u;
    __syncthreads();
#pragma unroll 4
    for (uint32_t r = threadIdx.x; r < rows; r += KD_SORT_THREADS) atomicAdd(&s[cont[(size_t)r * 5u] & 0xffu], 1u);
    __syncthreads();
    if (threadIdx.x < 32u) {
        uint32_t n[8], sum = 0;
#pragma unroll
        for (uint32_t i = 0; i < 8; i += 1) sum += n[i] = s[threadIdx.x * 8u + i];
        uint32_t incl = sum;
#pragma unroll
        for (uint32_t o = 1; o < 32; o <<= 1) {
            const uint32_t u = __shfl_up_sync(0xffffffffu, incl, o);
            if (threadIdx.x >= o) incl += u;
        }
        uint32_t at = incl - sum;
#pragma unroll
        for (uint32_t i = 0; i < 8; i += 1) {
            s[threadIdx.x * 8u + i] = at;
            at += n[i];
        }
    }
    __syncthreads();
#pragma unroll 4
    for (uint32_t r = threadIdx.x; r < rows; r += KD_SORT_THREADS) row_map[atomicAdd(&s[cont[(size_t)r * 5u] & 0xffu], 1u)] = r;
}

// The first n_chunks blocks, one per chunk: bitonic sort of eight consecutive entries per thread.  Strides below 8 are
// register to register, up to 128 by shuffle, so 52 of the 55 steps need no barrier (151,936 tokens: 10 us from a cold L2).
__global__ void __launch_bounds__(KD_SORT_THREADS)
moe_kd_sort_kernel(const uint32_t *toks, uint32_t *sorted, uint4 *bytes, uint32_t vocab, const uint32_t *cont, uint32_t *row_map,
                   uint32_t rows, uint32_t n_chunks) {
    moe_pdl_begin();
    __shared__ uint32_t s[KD_SORTED];
    if (blockIdx.x >= n_chunks) {
        kd_order_rows(s, cont, row_map, rows);
        return;
    }
    const uint32_t i0 = threadIdx.x * 8u, t0 = blockIdx.x * KD_CHUNK + i0;
    uint32_t v[8];
#pragma unroll
    for (uint32_t e = 0; e < 8; e += 1) {
        uint32_t key = KD_NOKEY;
        if (i0 + e < KD_CHUNK && t0 + e < vocab) {
            const uint32_t len = toks[(size_t)(t0 + e) * 5u + 4u], w = toks[(size_t)(t0 + e) * 5u];
            if (len == 1u) key = (w & 0xffu) << 9;
            else if (len > 1u) key = kd_key2(w & 0xffu, (w >> 8) & 0xffu);
        }
        v[e] = key << KD_IDX_BITS | (i0 + e);
    }
#pragma unroll
    for (uint32_t k = 2; k <= KD_SORTED; k <<= 1) {
#pragma unroll
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            if (j >= 256u) {
                __syncthreads();
#pragma unroll
                for (uint32_t e = 0; e < 8; e += 1) s[e * KD_SORT_THREADS + threadIdx.x] = v[e];
                __syncthreads();
            }
#pragma unroll
            for (uint32_t e = 0; e < 8; e += 1) {
                if (j < 8u) {
                    if ((e & j) != 0u) continue;
                    const uint32_t lo = min(v[e], v[e | j]), hi = max(v[e], v[e | j]);
                    const bool up = ((i0 + e) & k) == 0u;
                    v[e] = up ? lo : hi;
                    v[e | j] = up ? hi : lo;
                } else {
                    const uint32_t o = j < 256u ? __shfl_xor_sync(0xffffffffu, v[e], j / 8u) : s[e * KD_SORT_THREADS + (threadIdx.x ^ (j / 8u))];
                    const bool up = (i0 & k) == 0u, low = (i0 & j) == 0u;
                    v[e] = up == low ? min(v[e], o) : max(v[e], o);
                }
            }
        }
    }
    if (i0 >= KD_CHUNK) return;  // the filling sorts behind the chunk's own tokens
#pragma unroll
    for (uint32_t e = 0; e < 8; e += 1) {
        if (v[e] >> KD_IDX_BITS >= KD_NOKEY) continue;
        // the token's bytes in sorted order too, for the kernel that looks at single tokens (sorted: coalesced there)
        const uint32_t *tp = toks + (size_t)(blockIdx.x * KD_CHUNK + (v[e] & KD_IDX_MASK)) * 5u;
        bytes[t0 + e] = make_uint4(tp[0], tp[1], tp[2], tp[3]);
        v[e] |= (min(tp[4], 16u) - 1u) << KD_LEN_SHIFT;
    }
    uint4 *out = reinterpret_cast<uint4 *>(sorted + t0);
    out[0] = make_uint4(v[0], v[1], v[2], v[3]);
    out[1] = make_uint4(v[4], v[5], v[6], v[7]);
}

struct kd_mass_smem {
    float tile[(KD_CHUNK + 1u) * KD_PITCH];  // exponentials [slot][row]; the last slot is zero (for tokens without bytes)
    __align__(16) uint2 pos[KD_CHUNK];       // by position in the sorted chunk: word offset of the token's slot in the tile, KD_RUN_*
    uint32_t used[8];                        // first bytes of the block's rows, one bit each
};
static_assert(offsetof(kd_mass_smem, pos) % 16 == 0 && sizeof(kd_mass_smem) <= 113 * 1024, "pos is read 16 bytes at a time; two blocks per SM");
// What ends at a position of the sorted chunk: low byte the second byte, then 9 bits "first byte, has a second one" of the
// two-byte run that ends here (zero, which no row waits for, if none does), the first byte, and the two flags.
#define KD_RUN_MASK (0x1ffu << 8)
#define KD_RUN_END2 (1u << 30)
#define KD_RUN_END1 (1u << 31)
// A block of 128 tokens is fetched with four tokens per lane; token 4 l + q of it sits in slot 32 q + l, so that the
// lanes of a store fall into 32 banks.
__device__ __forceinline__ uint32_t kd_slot(uint32_t idx) { return (idx & ~127u) | (idx & 3u) << 5 | (idx >> 2 & 31u); }

// Grid: row groups x splits of the chunk list, two blocks per SM (one sums while the other fills its tile).  Every logit
// is read once: the row's maximum is not needed before the sweep, see `ref`.  Run sums go to the block's bins in L2
// with fire-and-forget adds; bins in shared memory would leave room for one block per SM.  Issue slots are 55 % busy, DRAM
// 26 %, the rest is waiting: ~10 instructions per logit to fetch, exponentiate and store it, ~11 to add it up.  384 rows of
// 151,936: 116 us.
template <bool VEC>  // rows can be read 16 bytes at a time
__global__ void __launch_bounds__(KD_THREADS, 2)
moe_kd_mass_kernel(const float *logits, const uint32_t *sorted, const uint32_t *cont, const uint32_t *row_map, float *bins, float2 *refs,
                   uint32_t vocab, uint32_t rows, uint32_t splits) {
    moe_pdl_begin();
    extern __shared__ __align__(16) uint8_t kd_raw[];
    kd_mass_smem &sm = *reinterpret_cast<kd_mass_smem *>(kd_raw);
    const uint32_t lid = threadIdx.x, lane = lid & 31u, warp = lid >> 5;
    const uint32_t group = blockIdx.x / splits, split = blockIdx.x - group * splits;
    const uint32_t n_chunks = (vocab + KD_CHUNK - 1u) / KD_CHUNK;
    const uint32_t c_lo = (uint32_t)((uint64_t)n_chunks * split / splits), c_hi = (uint32_t)((uint64_t)n_chunks * (split + 1u) / splits);
    const uint32_t slot0 = group * KD_ROWS + warp * KD_RPW, lslot = group * KD_ROWS + lane;
    const uint32_t c0 = lslot < rows ? cont[(size_t)row_map[lslot] * 5u] & 0xffu : ~0u;  // of the row this lane sums
    uint32_t row[KD_RPW];  // the rows this warp fetches
#pragma unroll
    for (uint32_t k = 0; k < KD_RPW; k += 1) row[k] = slot0 + k < rows ? row_map[slot0 + k] : ~0u;
    bins += (size_t)blockIdx.x * KD_BINS * KD_ROWS;         // [bin][row]
    for (uint32_t i = lid; i < KD_BINS * KD_ROWS; i += KD_THREADS) bins[i] = 0.0f;
    if (lid < KD_PITCH) sm.tile[KD_CHUNK * KD_PITCH + lid] = 0.0f;
    if (lid < 8u) sm.used[lid] = 0u;
    __threadfence();
    __syncthreads();
    if (warp == 0 && c0 != ~0u) atomicOr(&sm.used[c0 >> 5], 1u << (c0 & 31u));
    __syncthreads();

    constexpr uint32_t NV = KD_CHUNK / 32u;  // values of a row per lane
    auto fetch = [&](uint32_t c, uint32_t r, float (&v)[NV]) {
        const float *lg = logits + (size_t)(r != ~0u ? r : 0u) * vocab + c * KD_CHUNK;
        const uint32_t left = r != ~0u ? vocab - c * KD_CHUNK : 0u;
        if (VEC && left >= KD_CHUNK) {
#pragma unroll
            for (uint32_t i = 0; i < NV; i += 4) {
                const float4 x = __ldcs(reinterpret_cast<const float4 *>(lg) + (i / 4u) * 32u + lane);
                v[i] = x.x;
                v[i + 1] = x.y;
                v[i + 2] = x.z;
                v[i + 3] = x.w;
            }
        } else {
#pragma unroll
            for (uint32_t i = 0; i < NV; i += 1) {
                const uint32_t t = (i / 4u) * 128u + lane * 4u + (i & 3u);
                v[i] = t < left ? __ldcs(lg + t) : -3.0e38f;
            }
        }
    };
    // A position's run: tokens that share two bytes where some row of the block has the first one, else one byte.
    auto run_of = [&](uint32_t r) -> uint32_t {
        const uint32_t key = (r & KD_KEY_MASK) >> KD_IDX_BITS, b0 = key >> 9;
        if (b0 >= 256u) return ~0u;  // no bytes, or no neighbour
        return (sm.used[b0 >> 5] >> (b0 & 31u) & 1u) != 0u ? key : b0 << 9;
    };
    // first byte and "has a second one" of the runs this lane's second bins take
    const uint32_t want = (c0 << 1 | 1u) << 8 & KD_RUN_MASK;
    // The exponentials of a row are taken against `ref`, a maximum of the chunks seen so far: any reference within e^40
    // of the true maximum gives the same fp32 accuracy, so it only moves (and the row's bins are rescaled) when a chunk
    // exceeds it by more than that.  expf itself gives -inf, NaN and +inf their results (a packed approximation around
    // ex2 took 6 us less for 384 rows of 151,936, but was off by up to 2.5 units in the last place against expf's 1.9).
    // this thread's positions of the sorted chunk (lid, lid + 512) and the ones behind them
    constexpr uint32_t NP = (KD_CHUNK + KD_THREADS - 1u) / KD_THREADS;
    uint32_t rec[NP], nxt[NP];
    auto fetch_sorted = [&](uint32_t c) {
#pragma unroll
        for (uint32_t h = 0; h < NP; h += 1) {
            const uint32_t p = h * KD_THREADS + lid;
            rec[h] = p < KD_CHUNK ? sorted[c * KD_CHUNK + p] : ~0u;
            nxt[h] = p + 1u < KD_CHUNK ? sorted[c * KD_CHUNK + p + 1u] : ~0u;
        }
    };
    float ref[KD_RPW], top[KD_RPW], va[NV];
#pragma unroll
    for (uint32_t k = 0; k < KD_RPW; k += 1) ref[k] = top[k] = -3.0e38f;
    if (c_lo < c_hi) {
        fetch_sorted(c_lo);
        fetch(c_lo, row[0], va);
    }
    for (uint32_t c = c_lo; c < c_hi; c += 1) {
        float shrink[KD_RPW];
        // where runs end; every eighth position ends what is open, because the next one belongs to another warp
#pragma unroll
        for (uint32_t h = 0; h < NP; h += 1) {
            const uint32_t p = h * KD_THREADS + lid;
            if (p >= KD_CHUNK) continue;
            const uint32_t run = run_of(rec[h]), after = run_of(nxt[h]);
            uint32_t info = 0u, off = KD_CHUNK * KD_PITCH;
            if (run != ~0u) {
                off = kd_slot(rec[h] & KD_IDX_MASK) * KD_PITCH;
                if (run != after || (p & 7u) == 7u) info = run & 0x1ffffu | KD_RUN_END2;
                info |= run >> 9 << 17;
                if (run >> 9 != after >> 9 || (p & 7u) == 7u) info |= KD_RUN_END1;
            }
            sm.pos[p] = make_uint2(off, info);
        }
#pragma unroll
        for (uint32_t k = 0; k < KD_RPW; k += 1) {
            shrink[k] = 0.0f;
            float m = va[0];
#pragma unroll
            for (uint32_t i = 1; i < NV; i += 1) m = fmaxf(m, va[i]);
#pragma unroll
            for (uint32_t o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
            top[k] = fmaxf(top[k], m);
            if (c == c_lo) {
                ref[k] = top[k];
            } else if (top[k] > ref[k] + 40.0f) {
                shrink[k] = ref[k] - top[k];
                ref[k] = top[k];
            }
            float *dst = sm.tile + lane * KD_PITCH + warp * KD_RPW + k;
#pragma unroll
            for (uint32_t i = 0; i < NV; i += 1) dst[(i / 4u * 128u + (i & 3u) * 32u) * KD_PITCH] = expf(va[i] - ref[k]);
            if (k + 1u < KD_RPW) fetch(c, row[k + 1u < KD_RPW ? k + 1u : 0u], va);  // the other block of the SM covers this one
        }
        bool moved = false;
#pragma unroll
        for (uint32_t k = 0; k < KD_RPW; k += 1) moved = moved || shrink[k] != 0.0f;
        if (__syncthreads_or(moved ? 1 : 0) != 0) {  // the tile is complete; a reference moved: rescale what earlier chunks added
            __threadfence();
            __syncthreads();
#pragma unroll 1
            for (uint32_t k = 0; k < KD_RPW; k += 1) {
                if (shrink[k] == 0.0f) continue;
                const float f = expf(shrink[k]);
                for (uint32_t b = lane; b < KD_BINS; b += 32u) {
                    float *h = bins + b * KD_ROWS + warp * KD_RPW + k;
                    __stcg(h, __ldcg(h) * f);
                }
            }
            __threadfence();
            __syncthreads();
        }
        if (c + 1u < c_hi) {
            fetch_sorted(c + 1u);
            fetch(c + 1u, row[0], va);
        }

        // groups of eight positions in turn: neighbouring groups (alike in how many runs they hold) go to different warps
        float tot = 0.0f, a2 = 0.0f;  // of the current first byte; of the current two-byte run
        const float *tl = sm.tile + lane;
        float *bins1 = bins + lane, *bins2 = bins + 256u * KD_ROWS + lane;
#pragma unroll 1
        for (uint32_t g = warp; g < KD_CHUNK / 8u; g += KD_THREADS / 32u) {
            const uint4 *pp = reinterpret_cast<const uint4 *>(sm.pos + g * 8u);
            const uint4 p0 = pp[0], p1 = pp[1], p2 = pp[2], p3 = pp[3];
            const float e[8] = {tl[p0.x], tl[p0.z], tl[p1.x], tl[p1.z], tl[p2.x], tl[p2.z], tl[p3.x], tl[p3.z]};
            const uint32_t info[8] = {p0.y, p0.w, p1.y, p1.w, p2.y, p2.w, p3.y, p3.w};
#pragma unroll
            for (uint32_t i = 0; i < 8; i += 1) {
                tot += e[i];
                a2 += e[i];
                if (((info[i] ^ want) & KD_RUN_MASK) == 0u) atomicAdd(bins2 + (info[i] & 0xffu) * KD_ROWS, a2);
                a2 = (info[i] & KD_RUN_END2) != 0u ? 0.0f : a2;
                if ((info[i] & KD_RUN_END1) != 0u) {
                    atomicAdd(bins1 + (info[i] >> 17 & 0xffu) * KD_ROWS, tot);
                    tot = 0.0f;
                }
            }
        }
        __syncthreads();  // the tile is free again
    }
    __threadfence();  // the adds come before the loads below
    __syncthreads();
    // the bins turned to [row][bin] for the kernel that puts a row together
    for (uint32_t i = lid; i < KD_BINS * KD_ROWS; i += KD_THREADS) sm.tile[(i / KD_ROWS) * KD_PITCH + i % KD_ROWS] = __ldcg(bins + i);
    __syncthreads();
    for (uint32_t i = lid; i < KD_BINS * KD_ROWS; i += KD_THREADS) bins[i] = sm.tile[(i % KD_BINS) * KD_PITCH + i / KD_BINS];
#pragma unroll
    for (uint32_t k = 0; k < KD_RPW; k += 1) {
        if (lane == 0) refs[(size_t)blockIdx.x * KD_ROWS + warp * KD_RPW + k] = make_float2(ref[k], top[k]);
    }
}

// One block per row.
__global__ void __launch_bounds__(KD_RTHREADS, 3)
moe_kd_rows_kernel(const float *logits, const uint4 *bytes, const uint32_t *sorted, const uint32_t *cont, const uint32_t *row_map,
                   const float *bins, const float2 *refs, uint32_t *outp, uint32_t vocab, uint32_t splits) {
    moe_pdl_begin();
    __shared__ float H[KD_D][256];
    __shared__ float H2[KD_RWARPS][256];  // depth 2, a copy per warp: its bins take most of the adds
    __shared__ float A[KD_D + 1u];
    __shared__ float ztrue01[2];
    __shared__ float scale[KD_MAX_SPLITS];
    __shared__ uint32_t seg_pos[KD_RTHREADS], seg_end[KD_RTHREADS];
    __shared__ uint32_t wsum[KD_RWARPS];
    __shared__ float s_max;
    const uint32_t lid = threadIdx.x, lane = lid & 31u, warp = lid >> 5, r = row_map[blockIdx.x];
    uint32_t cw[4];
#pragma unroll
    for (uint32_t i = 0; i < 4; i += 1) cw[i] = cont[(size_t)r * 5u + i];
    const uint32_t nd = min(cont[(size_t)r * 5u + 4u], KD_D);  // :100
    const uint32_t c0 = cw[0] & 0xffu, c1 = (cw[0] >> 8) & 0xffu;
    uint32_t *o = outp + (size_t)r * KD_D * KD_K;
    for (uint32_t i = nd * KD_K + lid; i < KD_D * KD_K; i += KD_RTHREADS) o[i] = 0u;  // :101-103
    if (nd == 0u) return;  // the whole block

    // the row's maximum (:110-114) and its splits' factors
    const size_t blk0 = (size_t)(blockIdx.x / KD_ROWS) * splits * KD_ROWS + blockIdx.x % KD_ROWS;  // entry of split 0
    float2 rf = make_float2(-3.0e38f, -3.0e38f);
    if (lid < splits) rf = refs[blk0 + (size_t)lid * KD_ROWS];
    if (lid <= KD_D) A[lid] = 0.0f;
    for (uint32_t i = 512u + lid; i < KD_D * 256u; i += KD_RTHREADS) (&H[0][0])[i] = 0.0f;
    for (uint32_t i = lid; i < KD_RWARPS * 256u; i += KD_RTHREADS) (&H2[0][0])[i] = 0.0f;
    float m = rf.y;
#pragma unroll
    for (uint32_t s = 16; s > 0; s >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, s));
    if (lane == 0) wsum[warp] = __float_as_uint(m);
    __syncthreads();
    m = __uint_as_float(wsum[0]);
#pragma unroll
    for (uint32_t w = 1; w < KD_RWARPS; w += 1) m = fmaxf(m, __uint_as_float(wsum[w]));
    if (lid < splits) scale[lid] = rf.x == m ? 1.0f : expf(rf.x - m);  // equal infinities: no difference to form
    if (lid == 0) s_max = m;
    __syncthreads();
    m = s_max;
#pragma unroll
    for (uint32_t b = lid; b < KD_BINS; b += KD_RTHREADS) {
        const float *p = bins + blk0 * KD_BINS + b;
        float sum = 0.0f;
#pragma unroll 8
        for (uint32_t s = 0; s < splits; s += 1) sum += p[(size_t)s * KD_ROWS * KD_BINS] * scale[s];
        const bool mine = b == c0 || b == 256u + c1;  // the true byte is no candidate of its depth
        if (mine) ztrue01[b >> 8] = sum;
        (&H[0][0])[b] = mine ? 0.0f : sum;
    }

    if (nd > 2u) {
        // the tokens that share two bytes, chunk by chunk of the sorted lists
        const float *lg = logits + (size_t)r * vocab;
        const uint32_t n_chunks = (vocab + KD_CHUNK - 1u) / KD_CHUNK;
        const uint32_t key = kd_key2(c0, c1) << KD_IDX_BITS;
        float a_reg[3] = {0.0f, 0.0f, 0.0f};  // A[2..4], where nearly everything goes
        for (uint32_t cb = 0; cb < n_chunks; cb += KD_RTHREADS) {
            uint32_t lo = 0, len = 0;
            if (cb + lid < n_chunks) {
                const uint32_t *ch = sorted + (size_t)(cb + lid) * KD_CHUNK;
                uint32_t l0 = 0, l1 = 0;  // entries below key / below the next one; three probes a step: loads are what takes the time
#pragma unroll 1
                for (uint32_t step = KD_SORTED / 4u; step > 0; step >>= 2) {
                    uint32_t n0 = 0, n1 = 0;
#pragma unroll
                    for (uint32_t q = 1; q < 4; q += 1) {
                        n0 += l0 + q * step <= KD_CHUNK && (ch[l0 + q * step - 1u] & KD_KEY_MASK) < key ? 1u : 0u;
                        n1 += l1 + q * step <= KD_CHUNK && (ch[l1 + q * step - 1u] & KD_KEY_MASK) < key + KD_IDX_MASK + 1u ? 1u : 0u;
                    }
                    l0 += n0 * step;
                    l1 += n1 * step;
                }
                lo = (cb + lid) * KD_CHUNK + l0;
                len = l1 - l0;
            }
            uint32_t incl = len;
#pragma unroll
            for (uint32_t s = 1; s < 32; s <<= 1) {
                const uint32_t u = __shfl_up_sync(0xffffffffu, incl, s);
                if (lane >= s) incl += u;
            }
            __syncthreads();  // wsum and the segment tables are free
            if (lane == 31u) wsum[warp] = incl;
            __syncthreads();
            uint32_t before = 0, total = 0;
#pragma unroll
            for (uint32_t w = 0; w < KD_RWARPS; w += 1) {
                if (w < warp) before += wsum[w];
                total += wsum[w];
            }
            incl += before;
            seg_end[lid] = incl;
            seg_pos[lid] = lo - (incl - len);  // position in `sorted` of flattened index 0, modulo 2^32
            __syncthreads();
            // a warp takes a contiguous part of the flattened tokens, so that a lane finds its segment a step or two further on
            const uint32_t j_hi = (uint32_t)((uint64_t)total * (warp + 1u) / KD_RWARPS);
            uint32_t q = 0;  // the segment that holds flattened index j: the first with seg_end > j
            {
                const uint32_t j = (uint32_t)((uint64_t)total * warp / KD_RWARPS);
#pragma unroll
                for (uint32_t step = KD_RTHREADS / 2u; step > 0; step >>= 1) {
                    if (seg_end[q + step - 1u] <= j) q += step;
                }
            }
            for (uint32_t j0 = (uint32_t)((uint64_t)total * warp / KD_RWARPS) + lane; j0 - lane < j_hi; j0 += 32u * KD_RU) {
                uint32_t len1[KD_RU];  // bytes behind the first one; 0: nothing here (every token of these segments has two)
                uint4 tw[KD_RU];
                float x[KD_RU];
#pragma unroll
                for (uint32_t u = 0; u < KD_RU; u += 1) {
                    const uint32_t j = j0 + u * 32u;
                    len1[u] = 0u;
                    if (j < j_hi) {
                        while (seg_end[q] <= j) q += 1u;
                        const uint32_t pos = seg_pos[q] + j, rec = sorted[pos];
                        tw[u] = bytes[pos];
                        len1[u] = rec >> KD_LEN_SHIFT;
                        x[u] = lg[(cb + q) * KD_CHUNK + (rec & KD_IDX_MASK)];
                    }
                }
#pragma unroll
                for (uint32_t u = 0; u < KD_RU; u += 1) {
                    if (len1[u] == 0u) continue;
                    const float e = expf(x[u] - m);
                    const uint32_t w[4] = {tw[u].x, tw[u].y, tw[u].z, tw[u].w}, len = len1[u] + 1u;
                    const uint32_t lcp = kd_common_prefix(w, cw);
                    if (lcp < nd && lcp < len) {
                        const uint32_t b = kd_byte_at(w, lcp);
                        atomicAdd(lcp == 2u ? &H2[warp][b] : &H[lcp][b], e);
                    }
                    const uint32_t a = min(lcp, min(len, nd));
                    if (a == 2u) a_reg[0] += e;
                    else if (a == 3u) a_reg[1] += e;
                    else if (a == 4u) a_reg[2] += e;
                    else atomicAdd(&A[a], e);
                }
            }
        }
#pragma unroll
        for (uint32_t k = 0; k < 3; k += 1) {
#pragma unroll
            for (uint32_t s = 16; s > 0; s >>= 1) a_reg[k] += __shfl_xor_sync(0xffffffffu, a_reg[k], s);
            if (lane == 0 && a_reg[k] != 0.0f) atomicAdd(&A[2u + k], a_reg[k]);
        }
        __syncthreads();
        for (uint32_t b = lid; b < 256u; b += KD_RTHREADS) {
            float sum = 0.0f;
#pragma unroll
            for (uint32_t w = 0; w < KD_RWARPS; w += 1) sum += H2[w][b];
            H[2][b] = sum;
        }
    }
    __syncthreads();

    for (uint32_t l = warp; l < nd; l += KD_RWARPS) {  // :129-146, one warp per depth
        float ztrue = 0.0f;
        if (l < 2u) {
            ztrue = ztrue01[l];
        } else {
            for (uint32_t k = l + 1u; k <= KD_D; k += 1) ztrue += A[k];
        }
        float v[8];  // byte b = lane + 32 * i
        float sum = 0.0f;
#pragma unroll
        for (uint32_t i = 0; i < 8; i += 1) {
            v[i] = H[l][lane + 32u * i];
            sum += v[i];
        }
#pragma unroll
        for (uint32_t s = 16; s > 0; s >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, s);
        const float total = fmaxf(ztrue + sum, 1e-30f);
        if (lane == 0) o[l * KD_K] = kd_pack_entry(kd_byte_at(cw, l), ztrue / total);
        for (uint32_t j = 1; j < KD_K; j += 1) {
            // largest remaining mass, lowest byte among equals (:74-94)
            float bv = v[0];
            uint32_t bi = lane;
#pragma unroll
            for (uint32_t i = 1; i < 8; i += 1) {
                if (v[i] > bv) {
                    bv = v[i];
                    bi = lane + 32u * i;
                }
            }
#pragma unroll
            for (uint32_t s = 16; s > 0; s >>= 1) {
                const float ov = __shfl_xor_sync(0xffffffffu, bv, s);
                const uint32_t oi = __shfl_xor_sync(0xffffffffu, bi, s);
                if (ov > bv || (ov == bv && oi < bi)) {
                    bv = ov;
                    bi = oi;
                }
            }
            if ((bi & 31u) == lane) {
                o[l * KD_K + j] = kd_pack_entry(bi, bv / total);
#pragma unroll
                for (uint32_t i = 0; i < 8; i += 1) {
                    if (i == (bi >> 5)) v[i] = -1.0f;
                }
            }
        }
    }
}

// Rows in batches of `groups` groups of 32, the chunk list of each cut `splits` ways: two blocks per SM, and the rounds of
// blocks (each a share of the chunks plus ~2 chunks' worth of set-up and write-out, a further batch ~4) take the least time.
// The bins of a batch's blocks, at most max_blocks, lie in the work area: up to 2800 rows (of a vocabulary of 256,000; 4200
// of 151,936) that decides nothing, beyond it more batches take the place of more blocks.
static void kd_plan(uint32_t groups_all, uint32_t n_chunks, uint32_t slots, size_t max_blocks, uint32_t *groups, uint32_t *splits) {
    const uint32_t least = (groups_all + slots - 1u) / slots;
    uint64_t best = ~0ull;
    for (uint32_t n = least; n < least + 8u && n <= groups_all; n += 1) {
        const uint32_t g = (groups_all + n - 1u) / n;
        for (uint32_t s = 1; s <= n_chunks && s <= KD_MAX_SPLITS && (size_t)g * s <= max_blocks; s += 1) {
            const uint64_t cost = (uint64_t)n * (((g * s + slots - 1u) / slots) * (uint64_t)((n_chunks + s - 1u) / s + 2u) + (n > 1u ? 4u : 0u));
            if (cost < best) {
                best = cost;
                *groups = g;
                *splits = s;
            }
        }
    }
}

extern "C" void moe_cuda_kd_bytes(moe_cuda_ctx_t *c, const float *logits, const uint32_t *toks, const uint32_t *cont,
                                  uint32_t *outp, struct mda_pc_kd_bytes_t pc) {
    if (!MOE_LIVE(c)) return;
    MOE_REQUIRE(c, logits != NULL && toks != NULL && cont != NULL && outp != NULL, "kd_bytes: null buffer");
    MOE_REQUIRE(c, pc.vocab >= 1, "kd_bytes: empty vocabulary");
    if (pc.rows == 0) return;
    // Scratch grows with the vocabulary only; what depends on the rows lies in the context's work area (without one, in
    // scratch for one round of blocks).
    const uint32_t n_chunks = (pc.vocab + KD_CHUNK - 1u) / KD_CHUNK, slots = 2u * (uint32_t)c->sm_count;
    const size_t tokens = (size_t)n_chunks * KD_CHUNK, block_bytes = KD_ROWS * (KD_BINS * sizeof(float) + sizeof(float2));
    const size_t max_blocks = c->work != NULL ? c->work_bytes / block_bytes : slots;
    uint8_t *scr = (uint8_t *)moe_scratch(c, MOE_SCR_KD, tokens * (sizeof(uint4) + sizeof(uint32_t)) + (size_t)slots * KD_ROWS * sizeof(uint32_t) +
                                                             (c->work != NULL ? 0 : max_blocks * block_bytes));
    if (scr == NULL) return;
    uint32_t groups = 1, splits = 1;
    kd_plan((pc.rows + KD_ROWS - 1u) / KD_ROWS, n_chunks, slots, max_blocks, &groups, &splits);
    uint4 *bytes = (uint4 *)scr;
    uint32_t *sorted = (uint32_t *)(bytes + tokens);
    uint32_t *row_map = sorted + tokens;  // of a batch
    float *bins = (float *)(c->work != NULL ? c->work : (void *)(row_map + slots * KD_ROWS));
    float2 *refs = (float2 *)(bins + (size_t)groups * splits * KD_ROWS * KD_BINS);
    const bool vec = pc.vocab % 4u == 0 && ((uintptr_t)logits & 15) == 0;
    if (!c->kd_attr_set) {
        MOE_CUDA_TRY(c, cudaFuncSetAttribute(moe_kd_mass_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(kd_mass_smem)));
        MOE_CUDA_TRY(c, cudaFuncSetAttribute(moe_kd_mass_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(kd_mass_smem)));
        c->kd_attr_set = true;
    }
    const uint32_t batch = groups * KD_ROWS;
    for (uint32_t row0 = 0; row0 < pc.rows; row0 += batch) {
        const uint32_t rows = pc.rows - row0 < batch ? pc.rows - row0 : batch, blocks = (rows + KD_ROWS - 1u) / KD_ROWS * splits;
        const uint32_t sort = row0 == 0 ? n_chunks : 0u;  // the chunks serve all batches
        const float *lg = logits + (size_t)row0 * pc.vocab;
        const uint32_t *ct = cont + (size_t)row0 * 5u;
        moe_run(c, moe_kd_sort_kernel, sort + 1u, KD_SORT_THREADS, 0, toks, sorted, bytes, pc.vocab, ct, row_map, rows, sort);
        MOE_LAUNCHED(c);
        if (vec) moe_run(c, moe_kd_mass_kernel<true>, blocks, KD_THREADS, sizeof(kd_mass_smem), lg, sorted, ct, row_map, bins, refs, pc.vocab, rows, splits);
        else moe_run(c, moe_kd_mass_kernel<false>, blocks, KD_THREADS, sizeof(kd_mass_smem), lg, sorted, ct, row_map, bins, refs, pc.vocab, rows, splits);
        MOE_LAUNCHED(c);
        // started early its blocks fill the first SMs that the sweep leaves: fine for few, uneven for many (64 rows of 32,000:
        // 33 against 35 us, 100 rows: 45 against 40)
        if (rows <= 64u) moe_run(c, moe_kd_rows_kernel, rows, KD_RTHREADS, 0, lg, bytes, sorted, ct, row_map, bins, refs, outp + (size_t)row0 * KD_D * KD_K, pc.vocab, splits);
        else moe_kd_rows_kernel<<<rows, KD_RTHREADS, 0, c->stream>>>(lg, bytes, sorted, ct, row_map, bins, refs, outp + (size_t)row0 * KD_D * KD_K, pc.vocab, splits);
        MOE_LAUNCHED(c);
    }
}
