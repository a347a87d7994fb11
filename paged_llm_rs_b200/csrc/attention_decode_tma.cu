// Attention over the paged cache in bfloat16, head sizes 64 and 128, with the pages
// brought in by the bulk-copy engine: the serving kernel for decoding (one query
// token per request against its whole context, bound by the bytes of the keys and
// values) and for portions of prompts.  The reference's decode kernel
// (crates/pagedllm/src/kernels/paged_attention.cu:42-148) launches one block per
// (row, query head), re-reads every key once per query head of a group and keeps
// its scores in a buffer as long as the context; its prefill gathers the pages
// into a rectangle first (crates/pagedllm/src/model/attention.rs:190-214).  Here
// one CTA serves all query heads of a kv head from one copy of the keys, a long
// context is split over CTAs, nothing is gathered, and the softmax runs online.
//
// Pages come in with cp.async.bulk (the untiled TMA): a page's rows for one kv head
// are contiguous in the cache ([pages, kv_heads, page_size, head_dim]), so one
// thread moves a whole page slab (up to 64 rows) with one instruction and
// an mbarrier counts the bytes; a tile's slabs go out by as many lanes in one go (issued one after the
// other by one lane they took it some 280 clocks each, 2200 a tile of pages of 16 tokens, which bounded a CTA: 0.6B shape, us a step, 8 requests at
// 4096 1317 -> 1240, 16 at 1500 1169 -> 1101, one at 900 721 -> 695).  Nobody computes addresses per 16 bytes.  The
// cache stores each row's 16-byte chunks XOR-ed with the row's offset in its page
// (see qk_norm_rope_kv.cu), which is the layout ldmatrix wants in shared memory,
// so the slab is copied as it lies.
//
// A CTA has four consumer warps (or two, or eight: launch_tma) and one producer warp.  Tiles of 64 (32, 128) keys go round
// a ring of three stages (eight warps: two or three); every consumer warp reads every tile in turn (a parity wait tells
// two phases of a barrier apart and no more, so no warp may run a whole turn of the
// ring ahead of another: taking tiles in turn keeps them within it).  q.k^T and p.v
// run on mma.sync.m16n8k16.  For one query token the group's heads are the (padded)
// 16 rows of one block, each warp multiplies its own 16 keys of every tile and keeps
// a running (max, sum, output) of its own; the warps meet in shared memory at the
// end.  For several query tokens the rows (token, head) are spread over the warps,
// 16 each, and every warp multiplies whole tiles.  Every wait on an mbarrier is
// bounded: a waiter that gives up raises a status bit, tells the others and the
// CTA returns.
//
// It takes items whose key range starts on a multiple of 64 (of 32, by two warps) and has no window, in
// caches whose pages hold a power of two of at least 8 tokens; the rest is the
// cp.async kernel's (attention_mma.cu).
#include "common.cuh"

#define TD_KEYS 16       // keys of a tile for each consumer warp
#define TD_STAGES 3
#define TD_CONSUMERS 4
#define TD_QROWS 64      // query rows (token, head) a CTA may hold
#define TD_SPIN_LIMIT (1 << 18)

struct AttnWork { int seg, q_token0, q_count, q_pos0, kv_begin, kv_end, part_slot, split; };   // split: count << 16 | index

namespace {

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// Waits until the barrier's phase `parity` is over; gives up after a bounded number
// of polls or when another thread has given up.  Returns false then.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
    for (int spin = 0; spin < TD_SPIN_LIMIT; spin++) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((spin & 1023) == 1023 && *abort_flag) return false;
    }
    *abort_flag = 1;
    return false;
}
__device__ __forceinline__ void bulk_copy(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldsm4_t(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// An 8x8 block of 16-bit values held one row in four lanes, transposed across the warp.
__device__ __forceinline__ uint32_t movmatrix_t(uint32_t a) {
    uint32_t d;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;\n" : "=r"(d) : "r"(a));
    return d;
}
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
    __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&h);
}
template <int HD> __device__ __forceinline__ uint32_t toff(int row, int chunk) {
    return (uint32_t)(row * (HD * 2) + ((chunk ^ (row & 7)) << 4));
}

}  // namespace

// What the kernel needs to do the work of the q/k norm + rotation + cache-write kernel itself, for
// steps of single decoded tokens (qkv null: not asked to).  The reference does these as separate
// tensor operations before its attention (crates/pagedllm/src/model/attention.rs:148-158); in a
// decode step each is a launch of a few microseconds for a few kilobytes.
struct FusedQK {
    const bf16* qkv;                 // [tokens, (nh + 2 nkv) * hd], the projection's output
    const float *q_gain, *k_gain;    // [hd] or null: no norm
    const float *cos_t, *sin_t;      // [max_pos, hd / 2] or null: no rotation
    bf16 *k_pool, *v_pool;           // the pools again, to write the token's own row
    float eps;
    int max_pos;
};

// What a head's row is made with, hd / 32 values a lane (lane l: dims l * VPL ..): the gain and the token's rotation, by vector loads where
// they lie on such boundaries.
template <int HD>
struct RowConsts {
    static constexpr int VPL = HD / 32;      // 2 or 4
    float g[VPL], c[VPL], s[VPL];
    __device__ __forceinline__ static void load(const float* p, float (&f)[VPL]) {
        if ((uintptr_t)p & (4 * VPL - 1)) {
#pragma unroll
            for (int k = 0; k < VPL; k++) f[k] = p[k];
        } else if constexpr (VPL == 4) {
            const float4 v = *reinterpret_cast<const float4*>(p);
            f[0] = v.x; f[1] = v.y; f[2] = v.z; f[3] = v.w;
        } else {
            const float2 v = *reinterpret_cast<const float2*>(p);
            f[0] = v.x; f[1] = v.y;
        }
    }
    __device__ __forceinline__ void gain(const float* gain, int lane) { if (gain) load(gain + lane * VPL, g); }
    __device__ __forceinline__ void rotation(const float* cs, const float* sn, int lane) {
        if (cs) { load(cs + (lane & 15) * VPL, c); load(sn + (lane & 15) * VPL, s); }
    }
};
template <int HD>
__device__ __forceinline__ void row_values(const bf16* src, int lane, float (&f)[HD / 32]) {
    if constexpr (HD == 128) {
        const uint2 v = *reinterpret_cast<const uint2*>(src + lane * 4);
        f[0] = __uint_as_float(v.x << 16); f[1] = __uint_as_float(v.x & 0xffff0000u);
        f[2] = __uint_as_float(v.y << 16); f[3] = __uint_as_float(v.y & 0xffff0000u);
    } else {
        const uint32_t v = *reinterpret_cast<const uint32_t*>(src + lane * 2);
        f[0] = __uint_as_float(v << 16); f[1] = __uint_as_float(v & 0xffff0000u);
    }
}
// A head's row: the norm over it, then the rotation of dim d with d +- hd / 2 (16 lanes away), in float; the arithmetic of qk_norm_rope_kv.cu.
template <int HD>
__device__ __forceinline__ void norm_rope_row(const RowConsts<HD>& with, bool norm, bool rotate, float eps, int lane, float (&f)[HD / 32]) {
    constexpr int VPL = HD / 32;
    if (norm) {
        float ss = 0.f;
#pragma unroll
        for (int k = 0; k < VPL; k++) ss += f[k] * f[k];
        ss = warp_sum(ss);
        const float inv = 1.0f / sqrtf(ss / (float)HD + eps);
#pragma unroll
        for (int k = 0; k < VPL; k++) f[k] = f[k] * inv * with.g[k];
    }
    if (rotate) {
        const bool upper = lane >= 16;
#pragma unroll
        for (int k = 0; k < VPL; k++) {
            const float other = __shfl_xor_sync(0xffffffffu, f[k], 16);
            f[k] = upper ? f[k] * with.c[k] + other * with.s[k] : f[k] * with.c[k] - other * with.s[k];
        }
    }
}

template <int HD, bool KEYS_AS_ROWS, int CONSUMERS = TD_CONSUMERS, int STAGES = TD_STAGES, bool TWO_PARTS = CONSUMERS != TD_CONSUMERS>
__global__ void __launch_bounds__((CONSUMERS + 1) * 32, CONSUMERS == 8 ? 1 : 8 / CONSUMERS) attention_decode_tma_kernel(
    const bf16* q, const bf16* k_pool, const bf16* v_pool,   // written by the kernels before this one: no __restrict__
    const int* __restrict__ block_tables, const AttnWork* __restrict__ work, const int* __restrict__ n_work_ptr,
    bf16* __restrict__ out, float* __restrict__ part_o, float* __restrict__ part_ml,
    int nh, int nkv, int page_size, int page_shift, int n_pages, int table_width, float scale_log2,
    int heads_per_cta, int kinds_mask, FusedQK fq, int* status) {
    // The work items and block tables came from the host before the step, and the cache below
    // the step's own positions was written by earlier steps: neither depends on the kernels
    // just before this one.  So nobody waits for those kernels yet: the producer starts the
    // first tiles of old keys on their way at once, and waits only before a tile that may hold
    // a key of this step; the consumers wait before they read the queries.
    if ((int)blockIdx.y >= *n_work_ptr) return;
    const AttnWork w = work[blockIdx.y];
    // rows of a slab at most: a range may begin at any multiple of 64 (a chunk's start), of which a page of 128 tokens or more need not hold a whole tile
    constexpr int SLAB = TD_KEYS * CONSUMERS < 64 ? TD_KEYS * CONSUMERS : 64;
    if (!(kinds_mask & (w.q_count == 1 ? 1 : 2))) return;   // another kernel's item
    if (KEYS_AS_ROWS && w.q_count != 1) return;             // (this variant is for single tokens only)
    if (w.kv_begin & (SLAB - 1)) {
        // slabs and the swizzle need the range to start on a slab's boundary
        if (threadIdx.x == 0) atomicOr(status, 32);
        return;
    }
    const int group = nh / nkv;
    const int gparts = (group + heads_per_cta - 1) / heads_per_cta;
    const int kh = blockIdx.x / gparts;
    const int head0 = kh * group + (blockIdx.x % gparts) * heads_per_cta;
    const int n_heads = min(heads_per_cta, kh * group + group - head0);
    const int rows = w.q_count * n_heads;          // <= 64: (token, head) pairs
    const bool decode = w.q_count == 1;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int BK = TD_KEYS * CONSUMERS, QROWS = KEYS_AS_ROWS ? 16 : TD_QROWS;      // keys a tile; rows of q
    constexpr int KSTEPS = HD / 16, DTILES = HD / 8, CH = HD / 8;
    constexpr int TILE_BYTES = BK * HD * 2;          // keys (or values) of one tile
    constexpr int STAGE_BYTES = 2 * TILE_BYTES;

    extern __shared__ __align__(128) unsigned char smem[];
    const uint32_t base = smem_u32(smem);
    const uint32_t q_s = base + STAGES * STAGE_BYTES;
    const uint32_t bars = q_s + QROWS * HD * 2;       // full[S], empty[S]
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + STAGES * STAGE_BYTES + QROWS * HD * 2 + 16 * STAGES);

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; s++) {
            mbar_init(bars + 8 * s, 1);                      // full: the producer's arrive, plus the bytes
            mbar_init(bars + 8 * (STAGES + s), CONSUMERS);   // empty: every consumer warp's release
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::);
        asm volatile("fence.proxy.async.shared::cta;\n" ::);
    }
    __syncthreads();   // the barriers are set up; the producer goes its own way from here

    const int n_tiles = (w.kv_end - w.kv_begin + BK - 1) / BK;
    const int slab_rows = page_size < SLAB ? page_size : SLAB;
    const int slabs = BK / slab_rows;          // at most 16 (pages of at least 8 tokens)
    const uint32_t slab_bytes = (uint32_t)slab_rows * HD * 2;

    if (warp == CONSUMERS) {
        // ---- producer: page slabs into the ring ---------------------------------------------
        const int* table = block_tables + (size_t)w.seg * table_width;
        // the table entries of the key range, 32 at a time, one in each lane: no tile waits for a lookup
        int win0 = w.kv_begin >> page_shift;
        int tbl = (win0 + lane < table_width) ? table[win0 + lane] : -1;
        bool waited = false;
        for (int t = 0; t < n_tiles; t++) {
            const int s = t % STAGES;
            const int kv0 = w.kv_begin + t * BK;
            // A decoded token's own key is the only one this step writes for its request; a
            // portion's tiles read keys that other tiles of the portion bring, so they wait first.
            if (!waited && (!decode || kv0 + BK > w.q_pos0)) { pdl_wait(); waited = true; }
            if (((kv0 + BK - 1) >> page_shift) >= win0 + 32) {
                win0 = kv0 >> page_shift;
                tbl = (win0 + lane < table_width) ? table[win0 + lane] : -1;
            }
            if (t >= STAGES && !mbar_wait(bars + 8 * (STAGES + s), ((t / STAGES) - 1) & 1, abort_flag)) break;
            // lane i takes slab i of the keys, lane slabs + i that of the values: its page of the table, at or before the range's last key
            const int slab = lane & (slabs - 1), j = kv0 + slab * slab_rows;
            int page = __shfl_sync(0xffffffffu, tbl, ((j >> page_shift) - win0) & 31);
            if (lane >= 2 * slabs || j >= w.kv_end) page = -1;
            if (page >= n_pages) { atomicOr(status, 8); page = -1; }
            const uint32_t have = __ballot_sync(0xffffffffu, page >= 0) & ((1u << slabs) - 1);
            // slabs with no page behind them are zeroed by hand: nothing stale or unset is multiplied
            if (have != (1u << slabs) - 1) {
                for (int i = 0; i < slabs; i++) {
                    if (have & (1u << i)) continue;
                    for (int o = lane * 16; o < (int)slab_bytes; o += 32 * 16) {
                        *reinterpret_cast<uint4*>(smem + s * STAGE_BYTES + i * slab_bytes + o) = make_uint4(0, 0, 0, 0);
                        *reinterpret_cast<uint4*>(smem + s * STAGE_BYTES + TILE_BYTES + i * slab_bytes + o) = make_uint4(0, 0, 0, 0);
                    }
                }
                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");   // the zeros before the copies
                __syncwarp();
            }
            if (lane == 0) mbar_expect_tx(bars + 8 * s, 2 * slab_bytes * __popc(have));
            __syncwarp();
            if (page >= 0) {
                const size_t src = (((size_t)page * nkv + kh) * page_size + (j & (page_size - 1))) * HD;
                bulk_copy(base + s * STAGE_BYTES + (lane >= slabs ? TILE_BYTES : 0) + slab * slab_bytes, (lane >= slabs ? v_pool : k_pool) + src, slab_bytes,
                          bars + 8 * s);
            }
        }
        return;
    }

    // the query rows, zero beyond them (the first tiles are on their way meanwhile)
    const bool fused = fq.qkv != nullptr && decode;
    // fused: this CTA's range ends with the token's own key, which it makes itself (norm, rotation),
    // stores to the cache for later steps and puts into the last tile in shared memory
    const bool owns_new = fused && w.kv_end == w.q_pos0 + 1 && w.kv_end > w.kv_begin;   // (not an empty item that ends there)
    constexpr int VPL = HD / 32;
    uint32_t new_k[VPL / 2], new_v[VPL / 2];       // the row's values of this lane, packed (warps 2 and 3)
    if (fused) {
        int pos = w.q_pos0;
        if (fq.cos_t && (pos < 0 || pos >= fq.max_pos)) { if (threadIdx.x == 0) atomicOr(status, 4); pos = 0; }
        const float* cs = fq.cos_t ? fq.cos_t + (size_t)pos * (HD / 2) : nullptr;
        const float* sn = fq.sin_t ? fq.sin_t + (size_t)pos * (HD / 2) : nullptr;
        const int heads_total = nh + 2 * nkv;
        // (gains, rotation and the page of the token's own row are there before the projection is: fetched ahead of the wait.  0.6B shape, us a step, one
        // request at 300 tokens 609 -> 599, 64 at 512 1580 -> 1548)
        RowConsts<HD> rc;
        rc.gain(fq.q_gain, lane);
        rc.rotation(cs, sn, lane);
        const bool is_k = warp == CONSUMERS - 2, makes_row = owns_new && warp >= CONSUMERS - 2;
        RowConsts<HD> rk = rc;
        if (makes_row && is_k) rk.gain(fq.k_gain, lane);
        const int page = makes_row ? block_tables[(size_t)w.seg * table_width + (w.q_pos0 >> page_shift)] : 0;
        pdl_wait(KID_ATT_TMA);
        const bf16* tok = fq.qkv + (size_t)w.q_token0 * heads_total * HD;
        for (int row = warp; row < 16; row += CONSUMERS) {
            uint32_t pk[VPL / 2];
#pragma unroll
            for (int k = 0; k < VPL / 2; k++) pk[k] = 0;
            if (row < n_heads) {
                float f[VPL];
                row_values<HD>(tok + (size_t)(head0 + row) * HD, lane, f);
                norm_rope_row<HD>(rc, fq.q_gain != nullptr, cs != nullptr, fq.eps, lane, f);
#pragma unroll
                for (int k = 0; k < VPL / 2; k++) pk[k] = pack2(f[2 * k], f[2 * k + 1]);
            }
            // lane l's values are dims l * VPL ..: chunk (l * VPL) / 8 of the row, (l * VPL) % 8 values in
            unsigned char* dst = smem + STAGES * STAGE_BYTES + toff<HD>(row, lane * VPL / 8) + (lane * VPL % 8) * 2;
#pragma unroll
            for (int k = 0; k < VPL / 2; k++) reinterpret_cast<uint32_t*>(dst)[k] = pk[k];
        }
        if (makes_row) {
            float f[VPL];
            row_values<HD>(tok + (size_t)(nh + (is_k ? 0 : nkv) + kh) * HD, lane, f);
            norm_rope_row<HD>(rk, is_k && fq.k_gain, is_k && cs, fq.eps, lane, f);
            uint32_t pk[VPL / 2];
#pragma unroll
            for (int k = 0; k < VPL / 2; k++) pk[k] = pack2(f[2 * k], f[2 * k + 1]);
            // into the cache, chunk c at c ^ (offset in page & 7), for the steps to come
            const int off = w.q_pos0 & (page_size - 1);
            if (page >= 0 && page < n_pages) {
                bf16* row_w = (is_k ? fq.k_pool : fq.v_pool) + (((size_t)page * nkv + kh) * page_size + off) * HD;
                uint32_t* dst = reinterpret_cast<uint32_t*>(reinterpret_cast<unsigned char*>(row_w) +
                                                            (((lane * VPL / 8) ^ (off & 7)) << 4) + (lane * VPL % 8) * 2);
#pragma unroll
                for (int k = 0; k < VPL / 2; k++) dst[k] = pk[k];
            } else if (lane == 0) {
                atomicOr(status, 2);
            }
#pragma unroll
            for (int k = 0; k < VPL / 2; k++) { if (is_k) new_k[k] = pk[k]; else new_v[k] = pk[k]; }
        }
    } else {
        pdl_wait(KID_ATT_TMA);
        for (int idx = threadIdx.x; idx < (decode ? 16 : QROWS) * CH; idx += CONSUMERS * 32) {
            const int row = idx / CH, chunk = idx % CH;
            uint4 v = make_uint4(0, 0, 0, 0);
            if (row < rows)
                v = *reinterpret_cast<const uint4*>(q + ((size_t)(w.q_token0 + row / n_heads) * nh + head0 + row % n_heads) * HD + chunk * 8);
            *reinterpret_cast<uint4*>(smem + STAGES * STAGE_BYTES + toff<HD>(row, chunk)) = v;
        }
    }
    asm volatile("bar.sync 1, %0;\n" ::"n"(CONSUMERS * 32));

    float* o_s = reinterpret_cast<float*>(smem);          // [warps][16][HD], once the ring is no longer read
    float* ml_s = o_s + CONSUMERS * 16 * HD;           // [warps][16][2]
    // TWO_PARTS: the weights are multiplied as what bfloat16 holds of them and what it holds of the rest.  A warp's largest weight is 1 and rounds
    // exactly, so that the distance from 64 bits of weights in one part goes with how many warps and parts share the keys (64 requests at 512, group of 2:
    // 0.00208 by four warps, 0.00213 by two, 0.00166 in two parts, of which the result's rounding is nearly all).  With four heads at most the rest rides in
    // the columns beyond them, whose scores are the heads' again; with more it is a product of its own.
    const bool beside = TWO_PARTS && n_heads <= 4;
    if constexpr (KEYS_AS_ROWS) {
    // ---- consumers, one query token of at most 8 heads: the KEYS are the 16 rows of the score block --------
    // and the heads its 8 columns, S^T = K q^T and O^T = V^T P^T.  A block of 16 keys costs 8 + HD / 16
    // mma instead of twice that with the (two, four, eight) heads padded to 16 rows, the output is
    // HD / 16 x 4 registers instead of HD / 8 x 4, and the queries are 2 registers a k-step instead of 4.
    const bool rest_here = beside && (lane & 2);
    uint32_t qb[KSTEPS][2];
    {
#pragma unroll
        for (int kp = 0; kp < KSTEPS / 2; kp++) {
            uint32_t r[4];
            ldsm4(r, q_s + toff<HD>(lane & (beside ? 3 : 7), kp * 4 + (lane >> 3)));
            qb[2 * kp][0] = r[0]; qb[2 * kp][1] = r[1]; qb[2 * kp + 1][0] = r[2]; qb[2 * kp + 1][1] = r[3];
        }
    }
    const int hi0 = min(w.kv_end, w.q_pos0 + 1);     // keys the token may see, the same for all its heads
    // this thread: keys lane / 4 and + 8 of the warp's 16, heads 2 * (lane % 4) and + 1
    float m_run[2] = {-CUDART_INF_F, -CUDART_INF_F}, l_run[2] = {0.f, 0.f};
    constexpr int MT = HD / 16;
    float o_acc[MT][4];
#pragma unroll
    for (int d = 0; d < MT; d++) { o_acc[d][0] = o_acc[d][1] = o_acc[d][2] = o_acc[d][3] = 0.f; }
    const int key_base = warp * 16;
    const int mat = lane >> 3;
    for (int t = 0; t < n_tiles; t++) {
        const int s = t % STAGES;
        if (!mbar_wait(bars + 8 * s, (t / STAGES) & 1, abort_flag)) break;
        const int kv0 = w.kv_begin + t * BK + key_base;
        const uint32_t k_s = base + s * STAGE_BYTES, v_s = k_s + TILE_BYTES;
        if (owns_new && t == n_tiles - 1) {
            // the token's own key and value over what the copy brought for that row (whatever the page held)
            if (warp >= CONSUMERS - 2) {
                const int r = w.q_pos0 - (w.kv_begin + t * BK);
                unsigned char* dst = smem + s * STAGE_BYTES + (warp == CONSUMERS - 2 ? 0 : TILE_BYTES) +
                                     toff<HD>(r, lane * VPL / 8) + (lane * VPL % 8) * 2;
#pragma unroll
                for (int k = 0; k < VPL / 2; k++)
                    reinterpret_cast<uint32_t*>(dst)[k] = warp == CONSUMERS - 2 ? new_k[k] : new_v[k];
            }
            asm volatile("bar.sync 1, %0;\n" ::"n"(CONSUMERS * 32));
        }
        if (kv0 < hi0) {
            // the warp's 16 keys and values into registers, and the stage goes back to the producer
            // before the arithmetic: the next copy into it is on its way while this one is multiplied
            const int krow = key_base + (lane & 7) + (mat & 1) * 8;
            const int vkey = key_base + (lane & 7) + (mat >> 1) * 8;
            uint32_t kf[KSTEPS][4], vf[MT][4];
#pragma unroll
            for (int ks = 0; ks < KSTEPS; ks++) ldsm4(kf[ks], k_s + toff<HD>(krow, ks * 2 + (mat >> 1)));
#pragma unroll
            for (int d = 0; d < MT; d++) ldsm4_t(vf[d], v_s + toff<HD>(vkey, d * 2 + (mat & 1)));
            __syncwarp();
            if (lane == 0) mbar_arrive(bars + 8 * (STAGES + s));
            // two chains of mma over the k-steps, added at the end
            float sa[4] = {0.f, 0.f, 0.f, 0.f}, sb[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int ks = 0; ks < KSTEPS; ks += 2) {
                mma(sa, kf[ks], qb[ks][0], qb[ks][1]);
                mma(sb, kf[ks + 1], qb[ks + 1][0], qb[ks + 1][1]);
            }
            const int j0 = kv0 + (lane >> 2);
            const bool see0 = j0 < hi0, see1 = j0 + 8 < hi0;
            float sc[4];
            sc[0] = see0 ? (sa[0] + sb[0]) * scale_log2 : -CUDART_INF_F;
            sc[1] = see0 ? (sa[1] + sb[1]) * scale_log2 : -CUDART_INF_F;
            sc[2] = see1 ? (sa[2] + sb[2]) * scale_log2 : -CUDART_INF_F;
            sc[3] = see1 ? (sa[3] + sb[3]) * scale_log2 : -CUDART_INF_F;
            float mx[2] = {fmaxf(sc[0], sc[2]), fmaxf(sc[1], sc[3])};
            float corr[2], m_use[2];
#pragma unroll
            for (int i = 0; i < 2; i++) {
                mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 4));
                mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 8));
                mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 16));
                const float m_new = fmaxf(m_run[i], mx[i]);
                m_use[i] = m_new == -CUDART_INF_F ? 0.f : m_new;
                corr[i] = exp2f(m_run[i] - m_use[i]);
                m_run[i] = m_new;
                l_run[i] *= corr[i];
            }
            const float p0 = exp2f(sc[0] - m_use[0]), p1 = exp2f(sc[1] - m_use[1]);
            const float p2 = exp2f(sc[2] - m_use[0]), p3 = exp2f(sc[3] - m_use[1]);
            l_run[0] += p0 + p2;
            l_run[1] += p1 + p3;
            // P^T as the second operand: (key, head pair) in this thread becomes (head, key pair)
            uint32_t h0 = pack2(p0, p1), h1 = pack2(p2, p3), rest0 = 0, rest1 = 0;
            if constexpr (TWO_PARTS) {
                rest0 = pack2(p0 - __uint_as_float(h0 << 16), p1 - __uint_as_float(h0 & 0xffff0000u));
                rest1 = pack2(p2 - __uint_as_float(h1 << 16), p3 - __uint_as_float(h1 & 0xffff0000u));
                if (rest_here) { h0 = rest0; h1 = rest1; }
            }
            const uint32_t pb0 = movmatrix_t(h0), pb1 = movmatrix_t(h1);
            if (__any_sync(0xffffffffu, corr[0] != 1.f || corr[1] != 1.f)) {
#pragma unroll
                for (int d = 0; d < MT; d++) {
                    o_acc[d][0] *= corr[0]; o_acc[d][1] *= corr[1];
                    o_acc[d][2] *= corr[0]; o_acc[d][3] *= corr[1];
                }
            }
#pragma unroll
            for (int d = 0; d < MT; d++) mma(o_acc[d], vf[d], pb0, pb1);
            if (TWO_PARTS && !beside) {
                const uint32_t rb0 = movmatrix_t(rest0), rb1 = movmatrix_t(rest1);
#pragma unroll
                for (int d = 0; d < MT; d++) mma(o_acc[d], vf[d], rb0, rb1);
            }
        } else {
            __syncwarp();
            if (lane == 0) mbar_arrive(bars + 8 * (STAGES + s));
        }
    }
#pragma unroll
    for (int i = 0; i < 2; i++) {
        l_run[i] += __shfl_xor_sync(0xffffffffu, l_run[i], 4);
        l_run[i] += __shfl_xor_sync(0xffffffffu, l_run[i], 8);
        l_run[i] += __shfl_xor_sync(0xffffffffu, l_run[i], 16);
    }
    pdl_launch_dependents();   // the key tiles are done: the next kernel's CTAs may take their places
    asm volatile("bar.sync 1, %0;\n" ::"n"(CONSUMERS * 32));
    if (*abort_flag) {
        if (threadIdx.x == 0) atomicOr(status, 16);
        return;
    }
    // the four warps' results meet, head by head
    {
        const int qh = (lane & 3) * 2;
#pragma unroll
        for (int d = 0; d < MT; d++) {
            float* a = o_s + ((size_t)(warp * 16 + qh) * HD + d * 16 + (lane >> 2));
            a[0] = o_acc[d][0]; a[HD] = o_acc[d][1];
            a[8] = o_acc[d][2]; a[HD + 8] = o_acc[d][3];
        }
        if (lane < 4) {
            ml_s[(warp * 16 + qh) * 2] = m_run[0]; ml_s[(warp * 16 + qh) * 2 + 1] = l_run[0];
            ml_s[(warp * 16 + qh + 1) * 2] = m_run[1]; ml_s[(warp * 16 + qh + 1) * 2 + 1] = l_run[1];
        }
    }
    } else {
    // ---- consumers ------------------------------------------------------------------------------
    // One query token: the group's heads are ONE 16-row block and the warps share each tile's
    // keys (16 each).  Several query tokens: the rows (token, head) are spread over the warps,
    // 16 each, and every warp multiplies all 64 keys of a tile.
    const int rbase = decode ? 0 : warp * 16;
    uint32_t qf[KSTEPS][4];
    {
        const int mat = lane >> 3;
        const int row = rbase + (lane & 7) + (mat & 1) * 8;
#pragma unroll
        for (int ks = 0; ks < KSTEPS; ks++) ldsm4(qf[ks], q_s + toff<HD>(row, ks * 2 + (mat >> 1)));
    }
    // the two rows of this thread and the keys they may see
    const int r0 = rbase + (lane >> 2), r1 = r0 + 8;
    int hi[2];
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const int r = i ? r1 : r0;
        hi[i] = r < rows ? min(w.kv_end, w.q_pos0 + r / n_heads + 1) : 0;
    }
    int warp_hi = max(hi[0], hi[1]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) warp_hi = max(warp_hi, __shfl_xor_sync(0xffffffffu, warp_hi, o));
    float m_run[2] = {-CUDART_INF_F, -CUDART_INF_F}, l_run[2] = {0.f, 0.f};
    float o_acc[DTILES][4];
#pragma unroll
    for (int d = 0; d < DTILES; d++) { o_acc[d][0] = o_acc[d][1] = o_acc[d][2] = o_acc[d][3] = 0.f; }
    bool alive = true;

    const int key_base = decode ? warp * (BK / CONSUMERS) : 0;
    const int np_count = decode ? BK / CONSUMERS / 16 : BK / 16;   // pairs of 8-key score tiles: 1 or 4
    for (int t = 0; t < n_tiles && alive; t++) {
        const int s = t % STAGES;
        if (!mbar_wait(bars + 8 * s, (t / STAGES) & 1, abort_flag)) { alive = false; break; }
        const int kv0 = w.kv_begin + t * BK + key_base;
        const uint32_t k_s = base + s * STAGE_BYTES, v_s = k_s + TILE_BYTES;
        if (owns_new && t == n_tiles - 1) {
            // the token's own key and value over what the copy brought for that row (whatever the page held)
            if (warp >= CONSUMERS - 2) {
                const int r = w.q_pos0 - (w.kv_begin + t * BK);
                unsigned char* dst = smem + s * STAGE_BYTES + (warp == CONSUMERS - 2 ? 0 : TILE_BYTES) +
                                     toff<HD>(r, lane * VPL / 8) + (lane * VPL % 8) * 2;
#pragma unroll
                for (int k = 0; k < VPL / 2; k++)
                    reinterpret_cast<uint32_t*>(dst)[k] = warp == CONSUMERS - 2 ? new_k[k] : new_v[k];
            }
            asm volatile("bar.sync 1, %0;\n" ::"n"(CONSUMERS * 32));
        }
        if (kv0 < warp_hi) {   // some key of this warp's share is visible to one of its rows
            float s_acc[8][4];
#pragma unroll
            for (int n = 0; n < 8; n++) { s_acc[n][0] = s_acc[n][1] = s_acc[n][2] = s_acc[n][3] = 0.f; }
            {
                // one k-step at a time over all key tiles: neighbouring mma write different accumulators
                const int mat = lane >> 3;
                const int key0 = key_base + (lane & 7) + (mat >> 1) * 8;
#pragma unroll
                for (int ks = 0; ks < KSTEPS; ks++) {
                    uint32_t kf[4][4];
#pragma unroll
                    for (int np = 0; np < 4; np++)
                        if (np < np_count) ldsm4(kf[np], k_s + toff<HD>(key0 + np * 16, ks * 2 + (mat & 1)));
#pragma unroll
                    for (int np = 0; np < 4; np++) {
                        if (np >= np_count) break;
                        mma(s_acc[np * 2], qf[ks], kf[np][0], kf[np][1]);
                        mma(s_acc[np * 2 + 1], qf[ks], kf[np][2], kf[np][3]);
                    }
                }
            }
            float mx[2] = {-CUDART_INF_F, -CUDART_INF_F};
            const bool whole = kv0 + np_count * 16 <= min(hi[0], hi[1]);   // every key visible to both rows
#pragma unroll
            for (int n = 0; n < 8; n++) {
                if (n >= np_count * 2) break;
                const int j = kv0 + n * 8 + (lane & 3) * 2;
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const float v = (whole || j + (e & 1) < hi[e >> 1]) ? s_acc[n][e] * scale_log2 : -CUDART_INF_F;
                    s_acc[n][e] = v;
                    mx[e >> 1] = fmaxf(mx[e >> 1], v);
                }
            }
            float corr[2], m_use[2];
#pragma unroll
            for (int i = 0; i < 2; i++) {
                mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 1));
                mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 2));
                const float m_new = fmaxf(m_run[i], mx[i]);
                m_use[i] = m_new == -CUDART_INF_F ? 0.f : m_new;
                corr[i] = exp2f(m_run[i] - m_use[i]);
                m_run[i] = m_new;
                l_run[i] *= corr[i];
            }
            uint32_t pf[4][4];
#pragma unroll
            for (int n = 0; n < 8; n++) {
                if (n >= np_count * 2) break;
                const float p0 = exp2f(s_acc[n][0] - m_use[0]), p1 = exp2f(s_acc[n][1] - m_use[0]);
                const float p2 = exp2f(s_acc[n][2] - m_use[1]), p3 = exp2f(s_acc[n][3] - m_use[1]);
                l_run[0] += p0 + p1;
                l_run[1] += p2 + p3;
                pf[n >> 1][(n & 1) * 2] = pack2(p0, p1);
                pf[n >> 1][(n & 1) * 2 + 1] = pack2(p2, p3);
            }
            // the running maximum seldom moves after the first tiles: rescale only when it did
            if (__any_sync(0xffffffffu, corr[0] != 1.f || corr[1] != 1.f)) {
#pragma unroll
                for (int d = 0; d < DTILES; d++) {
                    o_acc[d][0] *= corr[0]; o_acc[d][1] *= corr[0];
                    o_acc[d][2] *= corr[1]; o_acc[d][3] *= corr[1];
                }
            }
            {
                const int mat = lane >> 3;
#pragma unroll
                for (int kk = 0; kk < 4; kk++) {
                    if (kk >= np_count) break;
                    const int key = key_base + kk * 16 + (lane & 7) + (mat & 1) * 8;
                    // four fragment loads in flight, then their eight mma
#pragma unroll
                    for (int d4 = 0; d4 < DTILES / 2; d4 += 4) {
                        uint32_t vf[4][4];
#pragma unroll
                        for (int i = 0; i < 4; i++) ldsm4_t(vf[i], v_s + toff<HD>(key, (d4 + i) * 2 + (mat >> 1)));
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            mma(o_acc[(d4 + i) * 2], pf[kk], vf[i][0], vf[i][1]);
                            mma(o_acc[(d4 + i) * 2 + 1], pf[kk], vf[i][2], vf[i][3]);
                        }
                    }
                }
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(bars + 8 * (STAGES + s));   // this warp is done with the stage
    }
#pragma unroll
    for (int i = 0; i < 2; i++) {
        l_run[i] += __shfl_xor_sync(0xffffffffu, l_run[i], 1);
        l_run[i] += __shfl_xor_sync(0xffffffffu, l_run[i], 2);
    }
    pdl_launch_dependents();   // the key tiles are done: the next kernel's CTAs may take their places
    // (named barriers from here on: the producer warp has left)
    asm volatile("bar.sync 1, %0;\n" ::"n"(CONSUMERS * 32));
    if (*abort_flag) {   // set before the warp that gave up reached the barrier: all see it alike
        if (threadIdx.x == 0) atomicOr(status, 16);
        return;
    }
    if (!decode) {
        // ---- several query tokens: every warp owns its rows' results ----------------------------
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const int r = i ? r1 : r0;
            if (r >= rows) continue;
            const int tq = r / n_heads, head = head0 + r % n_heads;
            if (w.part_slot < 0) {
                const float inv = l_run[i] > 0.f ? 1.0f / l_run[i] : 0.f;
                bf16* o = out + ((size_t)(w.q_token0 + tq) * nh + head) * HD + (lane & 3) * 2;
#pragma unroll
                for (int d = 0; d < DTILES; d++)
                    *reinterpret_cast<uint32_t*>(o + d * 8) = pack2(o_acc[d][i * 2] * inv, o_acc[d][i * 2 + 1] * inv);
            } else {
                const size_t pr = (size_t)(w.part_slot + tq) * nh + head;
                float* o = part_o + pr * HD + (lane & 3) * 2;
#pragma unroll
                for (int d = 0; d < DTILES; d++) { o[d * 8] = o_acc[d][i * 2]; o[d * 8 + 1] = o_acc[d][i * 2 + 1]; }
                if ((lane & 3) == 0) { part_ml[pr * 2] = m_run[i] * 0.6931471805599453f; part_ml[pr * 2 + 1] = l_run[i]; }
            }
        }
    } else {
    // ---- one query token: the four warps' results meet ---------------------------------------
#pragma unroll
    for (int d = 0; d < DTILES; d++) {
        const int c = d * 8 + (lane & 3) * 2;
        float* a = o_s + ((size_t)(warp * 16 + (lane >> 2)) * HD + c);
        a[0] = o_acc[d][0]; a[1] = o_acc[d][1];
        a[8 * HD] = o_acc[d][2]; a[8 * HD + 1] = o_acc[d][3];
    }
    if ((lane & 3) == 0) {
        ml_s[(warp * 16 + (lane >> 2)) * 2] = m_run[0]; ml_s[(warp * 16 + (lane >> 2)) * 2 + 1] = l_run[0];
        ml_s[(warp * 16 + (lane >> 2) + 8) * 2] = m_run[1]; ml_s[(warp * 16 + (lane >> 2) + 8) * 2 + 1] = l_run[1];
    }
    }
    }
    if (decode) {
    asm volatile("bar.sync 1, %0;\n" ::"n"(CONSUMERS * 32));
    for (int idx = threadIdx.x; idx < rows * HD; idx += CONSUMERS * 32) {
        const int r = idx / HD, c = idx % HD;
        float M = -CUDART_INF_F;
#pragma unroll
        for (int wi = 0; wi < CONSUMERS; wi++) M = fmaxf(M, ml_s[(wi * 16 + r) * 2]);
        float L = 0.f, o = 0.f;
#pragma unroll
        for (int wi = 0; wi < CONSUMERS; wi++) {
            const float mw = ml_s[(wi * 16 + r) * 2];
            const float f = mw == -CUDART_INF_F ? 0.f : exp2f(mw - M);
            L += ml_s[(wi * 16 + r) * 2 + 1] * f;
            o += (o_s[(size_t)(wi * 16 + r) * HD + c] + (beside ? o_s[(size_t)(wi * 16 + r + 4) * HD + c] : 0.f)) * f;
        }
        const int head = head0 + r;
        if (w.part_slot < 0) {
            out[((size_t)w.q_token0 * nh + head) * HD + c] = __float2bfloat16_rn(L > 0.f ? o / L : 0.f);
        } else {
            const size_t pr = (size_t)w.part_slot * nh + head;
            part_o[pr * HD + c] = o;
            if (c == 0) { part_ml[pr * 2] = M * 0.6931471805599453f; part_ml[pr * 2 + 1] = L; }   // natural-log units
        }
    }
    }

}

// Whether this kernel takes decode items of this shape and cache layout.
PLLM_EXPORT int pllm_attention_decode_tma_supports(int dtype, int nh, int nkv, int hd, int page_size, int window) {
    return dtype == PLLM_BF16 && (hd == 64 || hd == 128) && nkv > 0 && nh % nkv == 0 && window <= 0 && page_size >= 8 &&
           (page_size & (page_size - 1)) == 0;
}

template <int HD>
static int launch_tma(const void* q, const void* k_pool, const void* v_pool, const int* block_tables, const int* work,
                      const int* n_work_ptr, int max_work, void* out, float* part_o, float* part_ml, int nh, int nkv,
                      int page_size, int n_pages, int table_width, float scale, int kinds_mask, int singles, int whole,
                      FusedQK fq, int* status, cudaStream_t stream) {
    const int group = nh / nkv;
    const int heads_per_cta = group < 16 ? group : 16;
    const int gparts = (group + heads_per_cta - 1) / heads_per_cta;
    int page_shift = 0;
    while ((1 << page_shift) < page_size) page_shift++;
    auto smem_of = [](int consumers, int stages, int q_rows) {
        return (size_t)stages * 2 * TD_KEYS * consumers * HD * 2 + (size_t)q_rows * HD * 2 + 16 * stages + 16;
    };
    const float scale_log2 = scale * 1.4426950408889634f;
    // single tokens of groups of at most 8 heads go to the variant with the keys as rows; what else the
    // caller asked for (several query tokens) to the other, as a launch of its own
    int rest = kinds_mask;
    if (group <= 8 && (kinds_mask & 1)) {
        // Two consumer warps and tiles of 32 keys, four CTAs an SM, where a step of single tokens has more CTAs than two an SM: with four warps each and
        // two CTAs an SM the last turn of them was nearly empty (64 requests over 8 kv heads: 512 CTAs on 296 places).  0.6B shape, us a step of
        // 64 requests at 60 / 512 / 2500 tokens 1280 / 1730 / 3882 -> 1156 / 1600 / 3590, 48 at 1000 2194 -> 1941, 40 at 300 1425 -> 1325, 33 at 700
        // 1611 -> 1473; 6 layers of the 8B shape, 64 at 900 1095 -> 1055.  In fewer CTAs the larger ones have twice the bytes under way each.
        const bool small = singles > 2 * sm_count();
        // Eight warps and tiles of 128 keys where no token is split and every CTA gets an SM: half as many turns, and what fits in
        // shared memory is on its way before the wait for the projection.  A ring of two stages leaves the projection's CTAs room on the same SM, so that
        // these can be there before it is over; three where a CTA meets one on few SMs (us a step, three / two stages / four warps: 12 requests at 141
        // tokens 836 / 723 / 737, 16 at 500 862 / 797, eight at 100 677 / 653 / 671 and at 500 743 / 734 / 782, one at 300 609 / 630).
        const bool large = whole && singles > 0 && singles <= sm_count(), deep = large && 8 * singles <= sm_count();
        // (four warps take the weights in two parts where contexts are whole that were cut: the others' results stay as they are)
        auto* kernel = small ? attention_decode_tma_kernel<HD, true, 2> : deep ? attention_decode_tma_kernel<HD, true, 8, 3>
                     : large ? attention_decode_tma_kernel<HD, true, 8, 2>
                     : whole ? attention_decode_tma_kernel<HD, true, TD_CONSUMERS, TD_STAGES, true> : attention_decode_tma_kernel<HD, true, TD_CONSUMERS>;
        const int consumers = small ? 2 : large ? 8 : TD_CONSUMERS, stages = large && !deep ? 2 : TD_STAGES;
        const size_t smem = smem_of(consumers, stages, 16);
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        launch_chained(kernel, dim3(nkv * gparts, max_work), dim3((consumers + 1) * 32), smem,
                       stream, (const bf16*)q, (const bf16*)k_pool, (const bf16*)v_pool, block_tables, (const AttnWork*)work,
                       n_work_ptr, (bf16*)out, part_o, part_ml, nh, nkv, page_size, page_shift, n_pages, table_width,
                       scale_log2, heads_per_cta, 1, fq, status);
        rest &= ~1;
    }
    if (rest) {
        const size_t smem = smem_of(TD_CONSUMERS, TD_STAGES, TD_QROWS);
        cudaFuncSetAttribute(attention_decode_tma_kernel<HD, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        launch_chained(attention_decode_tma_kernel<HD, false>, dim3(nkv * gparts, max_work), dim3((TD_CONSUMERS + 1) * 32), smem,
                       stream, (const bf16*)q, (const bf16*)k_pool, (const bf16*)v_pool, block_tables, (const AttnWork*)work,
                       n_work_ptr, (bf16*)out, part_o, part_ml, nh, nkv, page_size, page_shift, n_pages, table_width,
                       scale_log2, heads_per_cta, rest, fq, status);
    }
    return launch_status();
}

static int dispatch_tma(const void* q, const void* k_pool, const void* v_pool, const int* block_tables, const int* work,
                        const int* n_work_ptr, int max_work, void* out, float* part_o, float* part_ml, int nh, int nkv,
                        int hd, int page_size, int n_pages, int table_width, float scale, int kinds_mask, int single_tokens, int whole,
                        FusedQK fq, int* status, cudaStream_t stream) {
    if (max_work <= 0) return PLLM_OK;
    if (!pllm_attention_decode_tma_supports(PLLM_BF16, nh, nkv, hd, page_size, 0)) return PLLM_ERR_SIZE;
    const int group = nh / nkv, singles = single_tokens * nkv * ((group + 15) / 16);
    if (hd == 128)
        return launch_tma<128>(q, k_pool, v_pool, block_tables, work, n_work_ptr, max_work, out, part_o, part_ml, nh, nkv,
                               page_size, n_pages, table_width, scale, kinds_mask, singles, whole, fq, status, stream);
    return launch_tma<64>(q, k_pool, v_pool, block_tables, work, n_work_ptr, max_work, out, part_o, part_ml, nh, nkv,
                          page_size, n_pages, table_width, scale, kinds_mask, singles, whole, fq, status, stream);
}

PLLM_EXPORT int pllm_attention_decode_tma(const void* q, const void* k_pool, const void* v_pool, const int* block_tables,
                                          const int* work, const int* n_work_ptr, int max_work, void* out,
                                          float* part_o, float* part_ml, int nh, int nkv, int hd, int page_size,
                                          int n_pages, int table_width, float scale, int kinds_mask, int* status,
                                          cudaStream_t stream) {
    FusedQK none = {};
    return dispatch_tma(q, k_pool, v_pool, block_tables, work, n_work_ptr, max_work, out, part_o, part_ml, nh, nkv, hd,
                        page_size, n_pages, table_width, scale, kinds_mask, 0, 0, none, status, stream);
}

// The same for a step of single decoded tokens, straight from the projection's output: the kernel
// norms and rotates the queries and each token's new key itself and writes key and value to the
// cache (rotation over the whole head or none; gains and tables may be null).  n_tokens: of the step (a captured one: the most it holds); whole: no item is
// part of a token's keys.
PLLM_EXPORT int pllm_attention_decode_tma_fused(const void* qkv, const float* q_gain, const float* k_gain, float eps,
                                                const float* cos_t, const float* sin_t, int max_pos, void* k_pool,
                                                void* v_pool, const int* block_tables, const int* work,
                                                const int* n_work_ptr, int max_work, void* out, float* part_o,
                                                float* part_ml, int nh, int nkv, int hd, int page_size, int n_pages,
                                                int table_width, float scale, int n_tokens, int whole, int* status, cudaStream_t stream) {
    if (qkv == nullptr || ((uintptr_t)qkv & 15)) return PLLM_ERR_ALIGN;
    FusedQK fq = {(const bf16*)qkv, q_gain, k_gain, cos_t, sin_t, (bf16*)k_pool, (bf16*)v_pool, eps, max_pos};
    return dispatch_tma(nullptr, k_pool, v_pool, block_tables, work, n_work_ptr, max_work, out, part_o, part_ml, nh, nkv, hd,
                        page_size, n_pages, table_width, scale, 1, n_tokens, whole, fq, status, stream);
}

PLLM_TRACE_EXPORT(attention_decode_tma)
