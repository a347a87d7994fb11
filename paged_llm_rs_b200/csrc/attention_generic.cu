// Paged attention for any head size (a multiple of 8 up to 256), any number of
// heads and groups, any page size, with an optional window: a kernel for bfloat16
// shapes that the tuned kernels do not take, and below it the kernel of the true
// 32-bit path.  Arithmetic in float on the CUDA cores.
//
// What it computes is the reference's attention
// (crates/pagedllm/src/model/attention.rs:198-214 and
// crates/pagedllm/src/kernels/paged_attention.cu:86-147): for query head h the
// keys and values of kv head h / group; score = q.k * scale; key j is visible to
// the query at position p iff j <= p (and, with a window w, j > p - w);
// softmax in float; weighted sum of values.  Unlike the reference's kernel it
// keeps no score buffer as long as the context: the softmax runs online over
// tiles of 32 keys, so the context is bounded by the cache alone.
//
// Work comes as a list of items prepared on the host, one CTA per (item, kv
// head, part of the group):
//   item = {seg, q_token0, q_count, q_pos0, kv_begin, kv_end, part_slot, split}
// q_count consecutive tokens of one request (token index q_token0.. in the step,
// positions q_pos0..) attend over keys [kv_begin, kv_end) of the request's block
// table row `seg`.  part_slot < 0: the item sees all keys its queries may see and
// writes the normalised output.  part_slot >= 0: the item is one split of a long
// key range and writes (max, sum, unnormalised output) for attention_reduce.
#include "common.cuh"

#define ATT_BK 32        // keys per tile
#define ATT_MAX_ROWS 16  // query rows (token x head of the group) per CTA, one warp each
#define ATT_MAX_HD 256

struct AttnWork { int seg, q_token0, q_count, q_pos0, kv_begin, kv_end, part_slot, split; };   // split: count << 16 | index (0: not split)

template <typename T>
__global__ void attention_generic_kernel(
    // q and the pools are written by the kernels before this one: not __restrict__, so that they are
    // read with coherent loads after the wait and never through the read-only cache
    const T* q,            // [n_tokens, nh, hd]
    const T* k_pool, const T* v_pool,  // [pages, nkv, page_size, hd]
    const int* __restrict__ block_tables,  // [n_segs, table_width]
    const AttnWork* __restrict__ work, const int* __restrict__ n_work_ptr,
    T* __restrict__ out,                // [n_tokens, nh, hd]
    float* __restrict__ part_o,         // [parts, nh, hd]
    float* __restrict__ part_ml,        // [parts, nh, 2]
    int nh, int nkv, int hd, int page_size, int n_pages, int table_width, int window, float scale,
    int heads_per_cta, int* status) {
    pdl_launch_dependents();
    pdl_wait(KID_ATT_GENERIC);
    const int group = nh / nkv;
    const int gparts = (group + heads_per_cta - 1) / heads_per_cta;
    const int item = blockIdx.x / (nkv * gparts), cta = blockIdx.x % (nkv * gparts);     // (an item's CTAs are neighbours in the grid)
    if (item >= *n_work_ptr) return;
    const AttnWork w = work[item];
    const int kh = cta / gparts;
    const int head0 = kh * group + (cta % gparts) * heads_per_cta;       // first q head of this CTA
    const int n_heads = min(heads_per_cta, kh * group + group - head0);
    const int rows = w.q_count * n_heads;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int hdp = hd + 4;  // padded row: conflict-free float4 reads across keys

    extern __shared__ float smem[];
    float* q_s = smem;                               // [ATT_MAX_ROWS][hd]
    float* k_s = q_s + ATT_MAX_ROWS * hd;            // [ATT_BK][hdp]
    float* v_s = k_s + ATT_BK * hdp;                 // [ATT_BK][hdp]
    __shared__ int page_s[ATT_BK];

    // Row r of the CTA: token r / n_heads of the item, head head0 + r % n_heads.
    const bool active = warp < rows;
    const int tq = active ? warp / n_heads : 0;
    const int head = active ? head0 + warp % n_heads : head0;
    const int pos = w.q_pos0 + tq;
    if (active) {
        const T* qr = q + ((size_t)(w.q_token0 + tq) * nh + head) * hd;
        for (int e = lane; e < hd; e += 32) q_s[warp * hd + e] = to_f32(qr[e]) * scale;
    }
    // Keys this row may see inside the item's range.
    const int lo = max(w.kv_begin, window > 0 ? pos - window + 1 : 0);
    const int hi = min(w.kv_end, pos + 1);

    float m = -CUDART_INF_F, l = 0.f;
    float acc[ATT_MAX_HD / 32];
#pragma unroll
    for (int k = 0; k < ATT_MAX_HD / 32; k++) acc[k] = 0.f;

    constexpr int N = Vec16<T>::N;
    const int vec_per_row = hd / N;
    const int* table = block_tables + (size_t)w.seg * table_width;

    for (int kv0 = w.kv_begin; kv0 < w.kv_end; kv0 += ATT_BK) {
        __syncthreads();  // the previous tile is no longer read
        if (threadIdx.x < ATT_BK) {
            const int j = kv0 + threadIdx.x;
            int page = -1;
            if (j < w.kv_end) {
                const int b = j / page_size;
                page = b < table_width ? table[b] : -1;
                // A freed page of a window layer holds -1 and is never visible to a
                // query of this item; anything else out of range is a fault.
                if (page >= n_pages) { atomicOr(status, 8); page = -1; }
            }
            page_s[threadIdx.x] = page;
        }
        __syncthreads();
        for (int idx = threadIdx.x; idx < ATT_BK * vec_per_row; idx += blockDim.x) {
            const int j = idx / vec_per_row, c = (idx % vec_per_row) * N;
            const int page = page_s[j];
            float fk[N], fv[N];
            if (page >= 0) {
                const size_t base = (((size_t)page * nkv + kh) * page_size + (kv0 + j) % page_size) * hd + c;
                Vec16<T> vk, vv;
                vk.load(k_pool + base); vv.load(v_pool + base);
                vk.unpack(fk); vv.unpack(fv);
            } else {
#pragma unroll
                for (int k = 0; k < N; k++) { fk[k] = 0.f; fv[k] = 0.f; }
            }
#pragma unroll
            for (int k = 0; k < N; k++) { k_s[j * hdp + c + k] = fk[k]; v_s[j * hdp + c + k] = fv[k]; }
        }
        __syncthreads();
        if (!active) continue;
        const int j = kv0 + lane;
        const bool visible = j >= lo && j < hi;
        if (!__any_sync(0xffffffffu, visible)) continue;
        float s = 0.f;
        {
            const float4* kr = reinterpret_cast<const float4*>(k_s + lane * hdp);
            const float4* qr = reinterpret_cast<const float4*>(q_s + warp * hd);
            for (int c = 0; c < hd / 4; c++) {
                const float4 a = qr[c], b = kr[c];
                s = fmaf(a.x, b.x, s); s = fmaf(a.y, b.y, s); s = fmaf(a.z, b.z, s); s = fmaf(a.w, b.w, s);
            }
        }
        s = visible ? s : -CUDART_INF_F;
        const float m_new = fmaxf(m, warp_max(s));
        const float p = visible ? expf(s - m_new) : 0.f;
        const float corr = expf(m - m_new);  // m = -inf on the first visible tile: exp(-inf) = 0
        l = l * corr + warp_sum(p);
        m = m_new;
#pragma unroll
        for (int k = 0; k < ATT_MAX_HD / 32; k++) acc[k] *= corr;
        for (int jj = 0; jj < ATT_BK; jj++) {
            const float pj = __shfl_sync(0xffffffffu, p, jj);
            if (pj == 0.f) continue;  // uniform across the warp
            const float* vr = v_s + jj * hdp;
#pragma unroll
            for (int k = 0; k < ATT_MAX_HD / 32; k++)
                if (k * 32 + lane < hd) acc[k] = fmaf(pj, vr[k * 32 + lane], acc[k]);
        }
    }
    if (!active) return;
    if (w.part_slot < 0) {
        const float inv = l > 0.f ? 1.0f / l : 0.f;
        T* o = out + ((size_t)(w.q_token0 + tq) * nh + head) * hd;
#pragma unroll
        for (int k = 0; k < ATT_MAX_HD / 32; k++)
            if (k * 32 + lane < hd) o[k * 32 + lane] = from_f32<T>(acc[k] * inv);
    } else {
        const size_t pr = (size_t)(w.part_slot + tq) * nh + head;
        float* o = part_o + pr * hd;
#pragma unroll
        for (int k = 0; k < ATT_MAX_HD / 32; k++)
            if (k * 32 + lane < hd) o[k * 32 + lane] = acc[k];
        if (lane == 0) { part_ml[pr * 2] = m; part_ml[pr * 2 + 1] = l; }
    }
}

// ---- float32 ------------------------------------------------------------------------------------
// The same in float32, which is bound by the multiply-adds of a prompt's portion and by its keys and values for decoded
// tokens.  A CTA of 128 threads (256 for heads of more than 128 entries) holds up to 32 rows (token, head) of an item and takes 64 keys a turn;
// a turn's keys come in by cp.async while the turn before it is summed, its values while its scores are formed (each buffer is asked for
// again as soon as it has been read).  More than four rows: a thread makes R x 4 scores (R: 4, or 2 of 256 threads) and then R rows x 4 HDV
// output entries, so that a value read from shared memory serves four sums (the kernel above reads two for each).  Up to
// four rows (a decoded token): a key belongs to NT / 64 threads, each taking a share of the head, and a row's softmax to a warp.
// Scores are sums of even and of odd entries (fma.rn.f32x2).  Measured at the 0.6B shape (16 heads over 8 kv heads of 128),
// 4 requests at 500 beside a portion of 252 tokens: 60 us a layer, the kernel above in its place 136.  It is bound by the
// latency of its own chains: a warp a scheduler (242 registers a thread), 35% of the issue slots and 37% of the
// shared-memory pipe in use.  A turn that is not full leaves out what it does not have: a prompt of 37 tokens takes 11.2 us, the kernel
// above 12.2.  Heads of more than 128 entries: a CTA with place for 32 rows and 64 keys fills an SM's shared memory, so a step of single
// tokens takes a kernel with place for four rows and 32 keys, three of which fit (64 requests at 1024, 16 heads over 2 of 256: 187 us, the kernel above 222;
// 8 over 1: 115 and 126; 8 requests at 2048, 16 over 2: 56 and 51, 8 over 1: 31 and 49.  With the CTA for 32 rows the first two took 260 and 141
// with the caches cold, the kernel above 229 and 135).
constexpr int AF_ROWS = 32, AF_BK = 64, AF_HEADS = 4;

__device__ __forceinline__ uint32_t af_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void af_copy16(uint32_t dst, const float* src, bool live) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ void af_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void af_wait_older() { asm volatile("cp.async.wait_group 1;\n" ::: "memory"); }
__device__ __forceinline__ void af_fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;\n" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long af_pack(float lo, float hi) {
    return (unsigned long long)__float_as_uint(lo) | ((unsigned long long)__float_as_uint(hi) << 32);
}
__device__ __forceinline__ float af_lo(unsigned long long v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float af_hi(unsigned long long v) { return __uint_as_float((uint32_t)(v >> 32)); }

// The weights of a turn's first `keys` keys (a multiple of four) times their values: rows ty + AF_ROWS / R a, the head's chunks tx + 16 h.
template <int R, int HDV, bool GUARD>
__device__ __forceinline__ void sum_values(const float* p_s, const float* v_s, int keys, int hdp, int chunks, int tx, int ty,
                                           unsigned long long (&acc)[R][HDV][2]) {
#pragma unroll 2
    for (int j = 0; j < keys; j += 4) {
        float4 p[R];
#pragma unroll
        for (int a = 0; a < R; a++) p[a] = *reinterpret_cast<const float4*>(p_s + (ty + AF_ROWS / R * a) * AF_BK + j);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            ulonglong2 v[HDV];
#pragma unroll
            for (int h = 0; h < HDV; h++)
                v[h] = *reinterpret_cast<const ulonglong2*>(v_s + (j + i) * hdp + ((tx + 16 * h < chunks ? tx + 16 * h : 0) << 2));
#pragma unroll
            for (int a = 0; a < R; a++) {
                const float pa = i == 0 ? p[a].x : i == 1 ? p[a].y : i == 2 ? p[a].z : p[a].w;
                const unsigned long long p2 = af_pack(pa, pa);
                if (!GUARD || pa != 0.f) {
#pragma unroll
                    for (int h = 0; h < HDV; h++) {
                        af_fma2(acc[a][h][0], p2, v[h].x);
                        af_fma2(acc[a][h][1], p2, v[h].y);
                    }
                }
            }
        }
    }
}

// A turn's scores: rows ty + AF_ROWS / R a with keys tx + 16 b, b < B.
template <int R, int B>
__device__ __forceinline__ void score_keys(const float* q_s, const float* k_s, int hdp, int chunks, int tx, int ty, float (&sc)[R][4]) {
    unsigned long long s2[R][B];
#pragma unroll
    for (int a = 0; a < R; a++)
#pragma unroll
        for (int b = 0; b < B; b++) s2[a][b] = 0ull;
#pragma unroll 2
    for (int c = 0; c < chunks; c++) {
        ulonglong2 qv[R];
#pragma unroll
        for (int a = 0; a < R; a++) {
            const int r = ty + AF_ROWS / R * a;
            qv[a] = *reinterpret_cast<const ulonglong2*>(q_s + r * hdp + ((c ^ (r & 7)) << 2));
        }
#pragma unroll
        for (int b = 0; b < B; b++) {
            const int j = tx + 16 * b;
            const ulonglong2 kv = *reinterpret_cast<const ulonglong2*>(k_s + j * hdp + ((c ^ (j & 7)) << 2));
#pragma unroll
            for (int a = 0; a < R; a++) {
                af_fma2(s2[a][b], qv[a].x, kv.x);
                af_fma2(s2[a][b], qv[a].y, kv.y);
            }
        }
    }
#pragma unroll
    for (int a = 0; a < R; a++)
#pragma unroll
        for (int b = 0; b < 4; b++) sc[a][b] = b < B ? af_lo(s2[a][b < B ? b : 0]) + af_hi(s2[a][b < B ? b : 0]) : 0.f;
}

// HDV: 64-entry parts of a head, hd <= 64 HDV.  NT: threads; R rows each.  BK: keys a turn (64 unless FEW).  FEW: no item has more than four rows.
template <int HDV, int NT, int BK = AF_BK, bool FEW = false>
__global__ void __launch_bounds__(NT, FEW ? 3 : HDV <= 2 ? 2 : 1) attention_f32_kernel(
    const float* q, const float* k_pool, const float* v_pool, const int* __restrict__ block_tables,
    const AttnWork* __restrict__ work, const int* __restrict__ n_work_ptr, float* __restrict__ out, float* __restrict__ part_o,
    float* __restrict__ part_ml, int nh, int nkv, int hd, int page_size, int n_pages, int table_width, int window, float scale, int* status) {
    pdl_launch_dependents();
    // The list of items and the block tables are the host's (the step's packed buffer): what they say is fetched before the wait
    // for the kernel that makes q and the newest keys.  The CTAs of an item are neighbours in the grid, so that the live ones
    // are the first and every SM gets one before any gets two.
    const int ctas = nkv * ((nh / nkv + AF_HEADS - 1) / AF_HEADS), item = blockIdx.x / ctas, part = blockIdx.x % ctas;
    if (item >= *n_work_ptr) return;
    const AttnWork w = work[item];
    const int group = nh / nkv, heads_per_cta = min(group, AF_HEADS), gparts = (group + heads_per_cta - 1) / heads_per_cta;
    const int kh = part / gparts, head0 = kh * group + (part % gparts) * heads_per_cta;
    const int n_heads = min(heads_per_cta, kh * group + group - head0);
    const int rows = min(w.q_count * n_heads, FEW ? 4 : AF_ROWS);
    const bool few = FEW || rows <= 4;
    static_assert(FEW || BK == AF_BK, "many rows take their keys 64 a turn");
    constexpr int R = AF_ROWS * 16 / NT, RS = AF_ROWS / R;                     // rows ty, ty + RS, ... of a thread
    constexpr int KT = NT / BK;                                                // few rows: threads that share a key
    constexpr int DIMS = 64 * HDV, VG = NT > DIMS ? NT / DIMS : 1, VE = NT < DIMS ? DIMS / NT : 1;     // ... groups of keys a value entry, entries a thread
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, tx = tid & 15, ty = tid >> 4;
    const int hdp = (hd + 31) & ~31, chunks = hd / 4;          // a row of shared memory holds whole groups of eight 16-byte chunks

    extern __shared__ __align__(128) float smem_f[];
    float* q_s = smem_f;                             // [32 (FEW: 4)][hdp], chunk c of row r at c ^ (r & 7)
    float* k_s = q_s + (FEW ? 4 : AF_ROWS) * hdp;    // [BK][hdp], likewise
    float* v_s = k_s + BK * hdp;                     // [BK][hdp], as it lies
    float* p_s = v_s + BK * hdp;                     // scores, then weights: [32][64] (few rows: [BK][4])
    __shared__ long long off_s[2][BK];               // where a key's row of this kv head starts in the pools; -1: nowhere
    __shared__ float row_s[2][4];                    // few rows: a row's factor for what it holds; at the end its sum

    // rows past the item's are never visible to anything
    int lo[4], hi[4], my_tok[4], my_head[4];        // (R of them where the rows are many)
#pragma unroll
    for (int a = 0; a < 4; a++) {
        const int r = few ? a : ty + RS * a;
        const bool live = r < rows && (few || a < R);
        my_tok[a] = live ? r / n_heads : 0;
        my_head[a] = live ? head0 + r % n_heads : head0;
        const int pos = w.q_pos0 + my_tok[a];
        lo[a] = max(w.kv_begin, window > 0 ? pos - window + 1 : 0);
        hi[a] = live ? min(w.kv_end, pos + 1) : 0;
    }
    const int* table = block_tables + (size_t)w.seg * table_width;
    auto find = [&](int t) {
        if (tid < BK) {
            const int j = w.kv_begin + t * BK + tid;
            int page = -1;
            if (j < w.kv_end) {
                const int b = j / page_size;
                page = b < table_width ? table[b] : -1;
                // A freed page of a window layer holds -1 and is never visible to a query of this item; anything else out of range is a fault.
                if (page >= n_pages) { atomicOr(status, 8); page = -1; }
            }
            off_s[t & 1][tid] = page < 0 ? -1 : (((long long)page * nkv + kh) * page_size + j % page_size) * hd;
        }
    };
    // (a thread's rows and chunks: NT further on is NT / chunks rows and NT % chunks chunks further on)
    const int first_row = tid / chunks, first_chunk = tid % chunks, row_step = NT / chunks, chunk_step = NT % chunks;
    auto load = [&](int t, float* dst, const float* pool, bool swizzled) {
        const uint32_t to = af_smem(dst);
        int j = first_row, c = first_chunk;
#pragma unroll 4
        while (j < BK) {
            const long long off = off_s[t & 1][j];
            af_copy16(to + (j * hdp + ((swizzled ? c ^ (j & 7) : c) << 2)) * 4, pool + (off < 0 ? 0 : off + c * 4), off >= 0);
            j += row_step;
            c += chunk_step;
            if (c >= chunks) { c -= chunks; j++; }
        }
        af_commit();
    };
    float m[4], l[4];
    unsigned long long acc[R][HDV][2];
    float acc1[4][VE];                               // few rows: entry tid % DIMS (+ NT) of each row's output, over keys of group tid / DIMS
#pragma unroll
    for (int a = 0; a < 4; a++) {
        m[a] = -CUDART_INF_F;
        l[a] = 0.f;
#pragma unroll
        for (int h = 0; h < VE; h++) acc1[a][h] = 0.f;
    }
#pragma unroll
    for (int a = 0; a < R; a++)
#pragma unroll
        for (int h = 0; h < HDV; h++) acc[a][h][0] = acc[a][h][1] = 0ull;
    const int turns = (w.kv_end - w.kv_begin + BK - 1) / BK;
    const int seen_by_all = min(w.kv_end, w.q_pos0 + 1), seen_from = window > 0 ? w.q_pos0 + w.q_count - window : 0;
    find(0);
    pdl_wait(KID_ATT_GENERIC);
    __syncthreads();
    load(0, k_s, k_pool, true);
    load(0, v_s, v_pool, false);
    for (int i = tid; i < (FEW ? 4 : AF_ROWS) * chunks; i += NT) {
        const int r = i / chunks, c = i % chunks;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < rows) {
            const float* from = q + ((size_t)(w.q_token0 + r / n_heads) * nh + head0 + r % n_heads) * hd + c * 4;
            v = make_float4(from[0], from[1], from[2], from[3]);
        }
        *reinterpret_cast<float4*>(q_s + r * hdp + ((c ^ (r & 7)) << 2)) = make_float4(v.x * scale, v.y * scale, v.z * scale, v.w * scale);
    }
    for (int t = 0; t < turns; t++) {
        const int kv0 = w.kv_begin + t * BK, live_keys = min(BK, w.kv_end - kv0);
        af_wait_older();
        __syncthreads();          // this turn's keys are there
        if (t + 1 < turns) find(t + 1);
        float sc[R][4];
        if (few) {
            const int j = tid / KT, share = tid % KT, c0 = chunks * share / KT, c1 = chunks * (share + 1) / KT;
            unsigned long long s2[4] = {0ull, 0ull, 0ull, 0ull};
            // (a key's threads begin at chunks of their own, so that what they read of q lies in other banks)
            int c = c0 + share < c1 ? c0 + share : c0;
            for (int i = c0; i < c1; i++) {
                const ulonglong2 kv = *reinterpret_cast<const ulonglong2*>(k_s + j * hdp + ((c ^ (j & 7)) << 2));
#pragma unroll
                for (int a = 0; a < 4; a++) {
                    const ulonglong2 qv = *reinterpret_cast<const ulonglong2*>(q_s + a * hdp + ((c ^ a) << 2));
                    af_fma2(s2[a], qv.x, kv.x);
                    af_fma2(s2[a], qv.y, kv.y);
                }
                if (++c == c1) c = c0;
            }
#pragma unroll
            for (int a = 0; a < 4; a++) {
                float v = af_lo(s2[a]) + af_hi(s2[a]);
#pragma unroll
                for (int o = 1; o < KT; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                const int key = kv0 + j;
                if (share == 0) p_s[j * 4 + a] = key >= lo[a] && key < hi[a] ? v : -CUDART_INF_F;
            }
        } else {
            // (a turn that is not full, a short prompt's only one as a rule, leaves out the sixteens of keys that it does not have)
            if (live_keys > 48) score_keys<R, 4>(q_s, k_s, hdp, chunks, tx, ty, sc);
            else if (live_keys > 32) score_keys<R, 3>(q_s, k_s, hdp, chunks, tx, ty, sc);
            else if (live_keys > 16) score_keys<R, 2>(q_s, k_s, hdp, chunks, tx, ty, sc);
            else score_keys<R, 1>(q_s, k_s, hdp, chunks, tx, ty, sc);
#pragma unroll
            for (int a = 0; a < R; a++)
#pragma unroll
                for (int b = 0; b < 4; b++) {
                    const int key = kv0 + tx + 16 * b;
                    if (key < lo[a] || key >= hi[a]) sc[a][b] = -CUDART_INF_F;
                }
        }
        __syncthreads();          // the keys have been read, the next turn's places are known (few rows: the scores are there)
        if (t + 1 < turns) load(t + 1, k_s, k_pool, true); else af_commit();
        if (few) {
            if (warp < rows) {
                // row `warp` is this warp's, two keys a lane (one of 32)
                const float s0 = p_s[lane * 4 + warp], s1 = BK > 32 ? p_s[(lane + 32) * 4 + warp] : -CUDART_INF_F;
                const float top = fmaxf(m[0], warp_max(fmaxf(s0, s1)));
                const float p0 = s0 == -CUDART_INF_F ? 0.f : expf(s0 - top), p1 = s1 == -CUDART_INF_F ? 0.f : expf(s1 - top);
                const float corr = top == -CUDART_INF_F ? 1.f : expf(m[0] - top);
                l[0] = l[0] * corr + warp_sum(p0 + p1);
                m[0] = top;
                p_s[lane * 4 + warp] = p0;
                if (BK > 32) p_s[(lane + 32) * 4 + warp] = p1;
                if (lane == 0) row_s[0][warp] = corr;
            } else if (lane == 0 && warp < 4) row_s[0][warp] = 1.f;
        } else {
#pragma unroll
            for (int a = 0; a < R; a++) {
                float top = fmaxf(fmaxf(sc[a][0], sc[a][1]), fmaxf(sc[a][2], sc[a][3]));
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));     // (the 16 lanes of the row)
                top = fmaxf(top, m[a]);
                const float corr = top == -CUDART_INF_F ? 1.f : expf(m[a] - top);
                float sum = 0.f;
#pragma unroll
                for (int b = 0; b < 4; b++) {
                    const float p = sc[a][b] == -CUDART_INF_F ? 0.f : expf(sc[a][b] - top);
                    sum += p;
                    p_s[(ty + RS * a) * AF_BK + tx + 16 * b] = p;
                }
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
                l[a] = l[a] * corr + sum;
                m[a] = top;
                const unsigned long long c2 = af_pack(corr, corr), zero = 0ull;
#pragma unroll
                for (int h = 0; h < HDV; h++)
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        unsigned long long v = zero;
                        af_fma2(v, acc[a][h][e], c2);
                        acc[a][h][e] = v;
                    }
            }
        }
        af_wait_older();
        __syncthreads();          // this turn's values and weights are there
        if (few) {
            const int j0 = tid / DIMS * (BK / VG), j1 = min(j0 + BK / VG, live_keys);
#pragma unroll
            for (int h = 0; h < VE; h++) {
                const int d = tid % DIMS + NT * h;
#pragma unroll
                for (int a = 0; a < 4; a++) acc1[a][h] *= row_s[0][a];
                if (d < hd) {
#pragma unroll 8
                    for (int j = j0; j < j1; j++) {
                        const float4 p = *reinterpret_cast<const float4*>(p_s + j * 4);
                        const float v = v_s[j * hdp + d];
                        if (p.x != 0.f) acc1[0][h] = fmaf(p.x, v, acc1[0][h]);
                        if (p.y != 0.f) acc1[1][h] = fmaf(p.y, v, acc1[1][h]);
                        if (p.z != 0.f) acc1[2][h] = fmaf(p.z, v, acc1[2][h]);
                        if (p.w != 0.f) acc1[3][h] = fmaf(p.w, v, acc1[3][h]);
                    }
                }
            }
        } else {
            // (a key that a row does not see adds nothing, whatever its value holds, since an infinity times zero is no zero:
            // where a turn has such keys its weights are looked at one by one)
            if (kv0 + AF_BK <= seen_by_all && kv0 >= seen_from) sum_values<R, HDV, false>(p_s, v_s, AF_BK, hdp, chunks, tx, ty, acc);
            else sum_values<R, HDV, true>(p_s, v_s, (live_keys + 3) & ~3, hdp, chunks, tx, ty, acc);
        }
        __syncthreads();          // the values and weights have been read
        if (t + 1 < turns) load(t + 1, v_s, v_pool, false); else af_commit();
    }
    if (few) {
        if (lane == 0 && warp < 4) { row_s[0][warp] = m[0]; row_s[1][warp] = l[0]; }
        if (VG > 1) {
            // the groups' shares, [group][row][entry] where the keys were, added in the order of the groups
#pragma unroll
            for (int a = 0; a < 4; a++) k_s[(tid / DIMS * 4 + a) * DIMS + tid % DIMS] = acc1[a][0];
        }
        __syncthreads();
        if (VG > 1) {
            if (tid >= DIMS) return;
#pragma unroll
            for (int a = 0; a < 4; a++)
                for (int g = 1; g < VG; g++) acc1[a][0] += k_s[(g * 4 + a) * DIMS + tid];
        }
#pragma unroll
        for (int a = 0; a < 4; a++) {
            if (a >= rows) break;
            const float sum = row_s[1][a], inv = w.part_slot >= 0 ? 1.f : sum > 0.f ? 1.0f / sum : 0.f;
            const size_t pr = (size_t)((w.part_slot >= 0 ? w.part_slot : w.q_token0) + my_tok[a]) * nh + my_head[a];
            float* o = (w.part_slot >= 0 ? part_o : out) + pr * hd;
#pragma unroll
            for (int h = 0; h < VE; h++)
                if (tid + NT * h < hd) o[tid + NT * h] = acc1[a][h] * inv;
            if (w.part_slot >= 0 && tid == 0) { part_ml[pr * 2] = row_s[0][a]; part_ml[pr * 2 + 1] = sum; }
        }
        return;
    }
#pragma unroll
    for (int a = 0; a < R; a++) {
        if (ty + RS * a >= rows) continue;
        const float inv = w.part_slot >= 0 ? 1.f : l[a] > 0.f ? 1.0f / l[a] : 0.f;
        const size_t pr = (size_t)((w.part_slot >= 0 ? w.part_slot : w.q_token0) + my_tok[a]) * nh + my_head[a];
        float* o = (w.part_slot >= 0 ? part_o : out) + pr * hd;
#pragma unroll
        for (int h = 0; h < HDV; h++)
            if (tx + 16 * h < chunks) {
                float* to = o + (tx + 16 * h) * 4;
                to[0] = af_lo(acc[a][h][0]) * inv; to[1] = af_hi(acc[a][h][0]) * inv;
                to[2] = af_lo(acc[a][h][1]) * inv; to[3] = af_hi(acc[a][h][1]) * inv;
            }
        if (w.part_slot >= 0 && tx == 0) { part_ml[pr * 2] = m[a]; part_ml[pr * 2 + 1] = l[a]; }
    }
}

// Combine the splits of a token: for entry t,
// red[t] = {token, first, count, stride}: its parts are first + s * stride, s < count.
// One CTA per (entry, head), RED_GROUPS groups of hd threads.  The weights exp(m_s - M) are
// formed once in shared memory (one warp, every split's (m, l) fetched in one trip); then group
// g sums the splits s = g, g + RED_GROUPS, ... of its output dimension, all its loads in flight
// together, and the groups' sums are added in the order of the groups: always the same order,
// whatever ran where.
#define RED_MAX_SPLITS 256
#define RED_GROUPS 4
template <typename T>
__global__ void attention_reduce_kernel(const float* part_o, const float* part_ml,   // just written: no __restrict__
                                        const int* __restrict__ red, const int* __restrict__ n_red_ptr,
                                        T* __restrict__ out, int nh, int hd) {
    __shared__ float wgt[RED_MAX_SPLITS];
    __shared__ float inv_s;
    extern __shared__ float gsum[];     // [RED_GROUPS][hd]
    pdl_launch_dependents();
    // The list of reductions is the host's (part of the step's packed buffer): how many there are and this
    // CTA's first entry are fetched before the wait for the attention kernel, two trips to L2 that then
    // lie beside that kernel's end and not behind it.
    const int head = blockIdx.y, n_red = *n_red_ptr;
    int4 entry = make_int4(0, 0, 0, 0);
    if ((int)blockIdx.x < n_red) entry = make_int4(red[blockIdx.x * 4], red[blockIdx.x * 4 + 1], red[blockIdx.x * 4 + 2], red[blockIdx.x * 4 + 3]);   // (the list need not lie on a 16-byte boundary)
    pdl_wait(KID_ATT_REDUCE);
    const int ng = blockDim.x / hd;                               // groups of hd threads: 1 or RED_GROUPS
    const int grp = threadIdx.x / hd, d = threadIdx.x % hd;
    // a CTA takes entries blockIdx.x, blockIdx.x + gridDim.x, ...: a captured step launches a grid for
    // the most entries a step could have, and CTAs with nothing to do must be few
    for (int t = blockIdx.x; t < n_red; t += gridDim.x) {
        if (t != (int)blockIdx.x) entry = make_int4(red[t * 4], red[t * 4 + 1], red[t * 4 + 2], red[t * 4 + 3]);
        const int token = entry.x, first = entry.y, count = min(entry.z, RED_MAX_SPLITS), stride = entry.w;
        if (count <= 0) continue;
        if (count <= 8 && ng == 1) {
            // few splits (the usual case away from batch 1): every thread fetches the entry's (m, l) pairs and
            // its own column of the partial rows in one trip, nothing goes through shared memory and no
            // thread waits for another, so a CTA's entries follow one another at the pace of the loads
            float2 ml[8];
            float v[8], M = -CUDART_INF_F;
            const float* po = part_o + ((size_t)first * nh + head) * hd + d;
            const size_t s_stride = (size_t)stride * nh * hd;
#pragma unroll
            for (int s = 0; s < 8; s++) {
                ml[s] = make_float2(-CUDART_INF_F, 0.f);
                v[s] = 0.f;
                if (s < count) {
                    ml[s] = *reinterpret_cast<const float2*>(part_ml + ((size_t)(first + s * stride) * nh + head) * 2);
                    v[s] = po[(size_t)s * s_stride];
                }
                M = fmaxf(M, ml[s].x);
            }
            float L = 0.f, o = 0.f;
#pragma unroll
            for (int s = 0; s < 8; s++) {
                if (s >= count) break;
                const float f = ml[s].x == -CUDART_INF_F ? 0.f : expf(ml[s].x - M);
                L += ml[s].y * f;
                o = fmaf(v[s], f, o);
            }
            out[((size_t)token * nh + head) * hd + d] = from_f32<T>(o * (L > 0.f ? 1.0f / L : 0.f));
            continue;
        }
        __syncthreads();       // the weights and sums of the entry before are no longer read
        if (threadIdx.x < 32) {
            // up to 8 splits a lane, their (m, l) pairs fetched together
            float2 ml[RED_MAX_SPLITS / 32];
            float M = -CUDART_INF_F;
#pragma unroll
            for (int i = 0; i < RED_MAX_SPLITS / 32; i++) {
                const int s = threadIdx.x + 32 * i;
                ml[i] = make_float2(-CUDART_INF_F, 0.f);
                if (s < count) ml[i] = *reinterpret_cast<const float2*>(part_ml + ((size_t)(first + s * stride) * nh + head) * 2);
                M = fmaxf(M, ml[i].x);
            }
            M = warp_max(M);
            float L = 0.f;
#pragma unroll
            for (int i = 0; i < RED_MAX_SPLITS / 32; i++) {
                const int s = threadIdx.x + 32 * i;
                if (s >= count) continue;
                const float f = ml[i].x == -CUDART_INF_F ? 0.f : expf(ml[i].x - M);
                wgt[s] = f;
                L += ml[i].y * f;
            }
            L = warp_sum(L);
            if (threadIdx.x == 0) inv_s = L > 0.f ? 1.0f / L : 0.f;
        }
        __syncthreads();
        {
            const float* po = part_o + ((size_t)first * nh + head) * hd + d;
            const size_t s_stride = (size_t)stride * nh * hd;
            float o = 0.f;
            for (int s0 = grp; s0 < count; s0 += ng * 4) {
                float v[4];
#pragma unroll
                for (int i = 0; i < 4; i++) v[i] = s0 + i * ng < count ? po[(size_t)(s0 + i * ng) * s_stride] : 0.f;
#pragma unroll
                for (int i = 0; i < 4; i++)
                    if (s0 + i * ng < count) o = fmaf(v[i], wgt[s0 + i * ng], o);
            }
            gsum[grp * hd + d] = o;
        }
        __syncthreads();
        if (grp == 0) {
            float o = gsum[d];
#pragma unroll
            for (int g2 = 1; g2 < RED_GROUPS; g2++)
                if (g2 < ng) o += gsum[g2 * hd + d];
            out[((size_t)token * nh + head) * hd + d] = from_f32<T>(o * inv_s);
        }
    }
}

PLLM_EXPORT int pllm_attention_generic(int dtype, const void* q, const void* k_pool, const void* v_pool,
                                       const int* block_tables, const int* work, const int* n_work_ptr,
                                       int max_work, void* out, float* part_o, float* part_ml, int nh, int nkv,
                                       int hd, int page_size, int n_pages, int table_width, int window,
                                       int singles, float scale, int* status, cudaStream_t stream) {
    if (max_work <= 0) return PLLM_OK;
    if (nh <= 0 || nkv <= 0 || nh % nkv != 0 || page_size <= 0) return PLLM_ERR_SIZE;
    if (hd <= 0 || hd > ATT_MAX_HD || hd % 8 != 0) return PLLM_ERR_SIZE;
    const int group = nh / nkv;
    if (dtype == PLLM_F32) {
        if (((uintptr_t)k_pool | (uintptr_t)v_pool) & 15) return PLLM_ERR_ALIGN;
        const int gparts = (group + AF_HEADS - 1) / AF_HEADS, hdp = (hd + 31) & ~31;
        // Heads of more than 128 entries: twice the threads, since one CTA fits an SM (a prompt of 37 tokens 16.0 us, the kernel above 19.2; with 128
        // threads, caches cold, 34.8 and 26.7); and where no item has many rows the kernel without place for them, three of whose CTAs fit.
        const bool few = singles != 0 && hd > 128;
        const int threads = hd <= 128 || few ? 128 : 256;
        const size_t smem = few ? ((size_t)(4 + 2 * 32) * hdp + 4 * 32) * sizeof(float)
                                : ((size_t)(AF_ROWS + 2 * AF_BK) * hdp + AF_ROWS * AF_BK) * sizeof(float);
        auto* kernel = few ? attention_f32_kernel<4, 128, 32, true>
                           : hd <= 64 ? attention_f32_kernel<1, 128> : hd <= 128 ? attention_f32_kernel<2, 128> : attention_f32_kernel<4, 256>;
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        launch_chained(kernel, dim3((unsigned)max_work * nkv * gparts), dim3(threads), smem, stream, (const float*)q, (const float*)k_pool,
                       (const float*)v_pool, block_tables, (const AttnWork*)work, n_work_ptr, (float*)out, part_o, part_ml, nh, nkv, hd,
                       page_size, n_pages, table_width, window, scale, status);
        return launch_status();
    }
    if (dtype != PLLM_BF16) return PLLM_ERR_DTYPE;
    const int heads_per_cta = group < ATT_MAX_ROWS ? group : ATT_MAX_ROWS;
    const int gparts = (group + heads_per_cta - 1) / heads_per_cta;
    const size_t smem = ((size_t)ATT_MAX_ROWS * hd + 2 * (size_t)ATT_BK * (hd + 4)) * sizeof(float);
    typedef bf16 T;
    cudaFuncSetAttribute(attention_generic_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    launch_chained(attention_generic_kernel<T>, dim3((unsigned)max_work * nkv * gparts), dim3(ATT_MAX_ROWS * 32), smem, stream,
                   (const T*)q, (const T*)k_pool, (const T*)v_pool, block_tables, (const AttnWork*)work, n_work_ptr,
                   (T*)out, part_o, part_ml, nh, nkv, hd, page_size, n_pages, table_width, window, scale,
                   heads_per_cta, status);
    return launch_status();
}

// The most query tokens one work item may hold for a given group size, so that
// the host cuts tiles the kernel accepts; and the CTAs that share an item.
PLLM_EXPORT int pllm_attention_generic_tile_tokens(int dtype, int nh, int nkv) {
    const int group = nh / nkv;
    if (dtype == PLLM_F32) return AF_ROWS / (group < AF_HEADS ? group : AF_HEADS);
    const int heads_per_cta = group < ATT_MAX_ROWS ? group : ATT_MAX_ROWS;
    return ATT_MAX_ROWS / heads_per_cta;
}

PLLM_EXPORT int pllm_attention_generic_ctas_per_item(int dtype, int nh, int nkv) {
    const int heads = dtype == PLLM_F32 ? AF_HEADS : ATT_MAX_ROWS;
    return nkv * ((nh / nkv + heads - 1) / heads);
}

// many_splits: the entries have eight splits or more each (a step of very few tokens): four groups of
// threads share an entry's splits; else one group (measured, 0.6B shape: batch 1, 16 splits: 0.911
// against 0.933 ms a step with four; batch 8, 4 splits: 1.503 against 1.478).
PLLM_EXPORT int pllm_attention_reduce(int dtype, const float* part_o, const float* part_ml, const int* red,
                                      const int* n_red_ptr, int max_red, void* out, int nh, int hd, int many_splits,
                                      cudaStream_t stream) {
    if (max_red <= 0) return PLLM_OK;
    const int groups = many_splits && RED_GROUPS * hd <= 1024 ? RED_GROUPS : 1;
    PLLM_DISPATCH_DTYPE(dtype, {
        // (a captured step launches its capacity, and every CTA of it costs its start even with nothing to do:
        // 256 x heads instead of 64 cost the 2048-token step 4 us a layer; the CTAs loop over the entries)
        dim3 grid(max_red < 64 ? max_red : 64, nh);
        launch_chained(attention_reduce_kernel<T>, grid, dim3(groups * hd), (size_t)groups * hd * sizeof(float), stream,
                       part_o, part_ml, red,
                       n_red_ptr, (T*)out, nh, hd);
    });
    return launch_status();
}

PLLM_TRACE_EXPORT(attention_generic)
