// The gated delta rule over a prompt's portion in blocks of 64 tokens (matrix_memory.cu has it token by token, for decoded
// tokens and short portions, and says what is computed).
//
// Per head, with G_t the sum of log g since the block's start, the writes u_t of a block solve
//     u_t + sum_{s < t} beta_t exp(G_t - G_s) (k_t . k_s) u_s = beta_t v_t - beta_t exp(G_t) S0^T k_t
// so u = U - W S0, where the rows of U and W solve the same triangular system with beta_t v_t and beta_t exp(G_t) k_t on the right
// and do not depend on the state: all blocks solve it AT THE SAME TIME.  What goes from block to block is two products,
//     u = U - W S0,   S <- exp(G_L) S0 + sum_s exp(G_L - G_s) k_s u_s^T
// (the chunkwise form of the delta rule: Yang et al., "Parallelizing Linear Transformers with the Delta Rule over Sequence Length", 2024, and "Gated Delta
// Networks", 2024), and the outputs follow, again for all blocks at once: o_t = exp(G_t) S0^T q_t + sum_{s <= t} exp(G_t - G_s) (q_t . k_s) u_s.
//   delta_solve_kernel    unit vectors, G, the triangular system by forward substitution (16 rows at a time)
//   delta_states_kernel   a head's 16 columns of S through the blocks of a segment
//   delta_outputs_kernel  the outputs
// Sums of log g and their differences are formed in double; everything else is float,
// as in the recurrence, whose every write the forward substitution repeats.  No decay is divided by.
//
// What bounds the recurrence is its chain (440 ns a token and head); what bounds the blocks is delta_states_kernel's chain, a few
// microseconds a block of 64 tokens.  1016 tokens beside 8 decoded ones, 8 heads of 128 x 128 over 4 key heads (us, caches cold): the
// recurrence 446; these kernels 45 + 76 + 49, and 13 for the decoded tokens.  A segment that is not long goes through the recurrence all the same
// (kernels/ops.py, DELTA_LONGEST).
#pragma once

#include "matrix_memory.cuh"
#include "mlstm_blocks.cuh"

#define DB_L 64                // tokens a block
#define DB_THREADS 256
#define DB_COLS 16             // columns of S a CTA of delta_states_kernel
#define DB_C 64                // columns of the outputs a CTA
#define DB_MAX_D 128

struct DBBuffers {
    float* W;                  // [blocks of longer segments][H][64][d]
    float* kd;                 // [blocks][H][64][d]: exp(G_L - G_s) k_s
    float* U;                  // [blocks][H][64][E]: U, then u
    float* S;                  // [blocks][H][d][E]: what the block starts from
    float* decay;              // [blocks][H]: exp(G_L)
};
static inline long long db_floats(int n_tokens, int n_segs, int longest, int H, int d, int E) {
    return mb_blocks(n_tokens, n_segs, longest) * H * (2LL * DB_L * d + (long long)DB_L * E + (long long)d * E + 4) + 16;
}
static inline DBBuffers db_buffers(float* at, int n_tokens, int n_segs, int longest, int H, int d, int E) {
    const long long nb = mb_blocks(n_tokens, n_segs, longest) * H;
    DBBuffers b;
    b.W = at;
    b.kd = b.W + nb * DB_L * d;
    b.U = b.kd + nb * DB_L * d;
    b.S = b.U + nb * DB_L * E;
    b.decay = b.S + nb * d * E;
    return b;
}

// A block's rows of q or k as unit vectors times `scale` (a warp a row; zeros past nt), swizzled by chunks as mb_rows has them.
__device__ __forceinline__ void db_unit_rows(const float* src, long long stride, int nt, int d, float* dst, int dp, float scale) {
    const int lane = threadIdx.x & 31;
    for (int t = threadIdx.x >> 5; t < DB_L; t += DB_THREADS / 32) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t < nt && lane * 4 < d) v = *reinterpret_cast<const float4*>(src + (long long)t * stride + lane * 4);
        const float inv = scale / sqrtf(warp_sum(v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w) + 1e-6f);
        if (lane * 4 < dp) *reinterpret_cast<float4*>(dst + t * dp + ((lane ^ (t & 7)) << 2)) = make_float4(v.x * inv, v.y * inv, v.z * inv, v.w * inv);
    }
}
// G of a block's tokens in double and beta, by the CTA's first warp (past nt: the last G, and zero).  A token whose log g is an
// infinity, or below DB_LEAST, starts anew: the recurrence's factor exp(log g) is zero there.  It counts as DB_LEAST, whose exponential is zero
// too, so that differences of G between the tokens behind it stay what they are, where infinities would leave none.
constexpr float DB_LEAST = -1000.f;
struct DBTokens { double G[DB_L]; float beta[DB_L]; };
__device__ __forceinline__ void db_tokens(DBTokens& tk, const float* ba, size_t tok0, int nt, int h, int H, float A, float bias) {
    if (threadIdx.x >= 32) return;
    const int lane = threadIdx.x;
    double before = 0.0;
#pragma unroll
    for (int c = 0; c < DB_L; c += 32) {
        const int t = c + lane;
        const float* r = ba + (tok0 + (t < nt ? t : 0)) * 2 * H;
        const float log_g = A * mm_softplus(r[H + h] + bias);
        double G = t < nt ? (double)(log_g < DB_LEAST ? DB_LEAST : log_g) : 0.0;      // (a NaN stays one)
        tk.beta[t] = t < nt ? mm_sigmoid(r[h]) : 0.f;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double l = __shfl_up_sync(0xffffffffu, G, o);
            if (lane >= o) G += l;
        }
        G += before;
        tk.G[t] = G;
        before = __shfl_sync(0xffffffffu, G, 31);
    }
}
// out[r][e] = rows ty + 16 r of a times rows tx + 16 e of b, both [64][dp] swizzled.  A sum is four of every fourth entry, in runs of eight
// products that are added up when they are complete: one chain over all entries was off by half as much again as the recurrence's warp-wide sums.
__device__ __forceinline__ void db_product(const float* a, const float* b, int dp, int chunks, int tx, int ty, float (&out)[4][4]) {
    f32x2 acc[4][4];
    const f32x2 one = mm_pair(1.f, 1.f), zero = mm_pair(0.f, 0.f);
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
        for (int e = 0; e < 4; e++) acc[r][e] = zero;
    for (int c0 = 0; c0 < chunks; c0 += 8) {
        f32x2 lo[4][4], hi[4][4];
#pragma unroll
        for (int r = 0; r < 4; r++)
#pragma unroll
            for (int e = 0; e < 4; e++) lo[r][e] = hi[r][e] = zero;
        const int c1 = min(c0 + 8, chunks);
        for (int c = c0; c < c1; c++) {
            ulonglong2 x[4];
#pragma unroll
            for (int r = 0; r < 4; r++) { const int t = ty + 16 * r; x[r] = *reinterpret_cast<const ulonglong2*>(a + t * dp + ((c ^ (t & 7)) << 2)); }
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const int t = tx + 16 * e;
                const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(b + t * dp + ((c ^ (t & 7)) << 2));
#pragma unroll
                for (int r = 0; r < 4; r++) { lo[r][e] = mm_fma2(x[r].x, y.x, lo[r][e]); hi[r][e] = mm_fma2(x[r].y, y.y, hi[r][e]); }
            }
        }
#pragma unroll
        for (int r = 0; r < 4; r++)
#pragma unroll
            for (int e = 0; e < 4; e++) acc[r][e] = mm_fma2(one, mm_fma2(one, lo[r][e], hi[r][e]), acc[r][e]);
    }
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
        for (int e = 0; e < 4; e++) { const float2 v = mm_unpair(acc[r][e]); out[r][e] = v.x + v.y; }
}

// grid (blocks, heads).  c: [tokens, channels] float, q at 0 (G d), k at G d, v at 2 G d (H E); ba: [tokens, 2 H], b_raw | a_raw.
__global__ void __launch_bounds__(DB_THREADS, 2) delta_solve_kernel(const float* c, int channels, const float* ba, const float* __restrict__ a_log,
                                                                 const float* __restrict__ dt_bias, const MMSegment* __restrict__ segs, int n_segs,
                                                                 DBBuffers buf, int H, int G, int d, int E, int longest) {
    extern __shared__ __align__(16) float mm_smem[];
    __shared__ DBTokens tk;
    const MMBlock b = mm_find_block(segs, n_segs, blockIdx.x, DB_L, longest);
    pdl_launch_dependents();
    pdl_wait(KID_MATRIX_MEMORY);
    if (b.seg < 0) return;
    const MMSegment s = segs[b.seg];
    if (s.count <= longest) return;
    const int h = blockIdx.y, kh = h / (H / G), begin = b.tb * DB_L, nt = min(DB_L, s.count - begin), dp = (d + 31) & ~31;
    const size_t tok0 = (size_t)s.first + begin;
    const int cols = d + E;
    float* k_s = mm_smem;                        // [64][dp]
    float* A_s = k_s + DB_L * dp;                // [64][64]
    float* R_s = A_s + DB_L * DB_L;              // [64][cols]: the right sides, then the solutions
    const float* row = c + tok0 * channels;
    db_tokens(tk, ba, tok0, nt, h, H, -expf(a_log[h]), dt_bias[h]);
    db_unit_rows(row + (size_t)G * d + (size_t)kh * d, channels, nt, d, k_s, dp, 1.f);
    __syncthreads();
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    {
        float kk[4][4];
        db_product(k_s, k_s, dp, d / 4, tx, ty, kk);
#pragma unroll
        for (int r = 0; r < 4; r++)
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const int t = ty + 16 * r, o = tx + 16 * e;
                A_s[t * DB_L + o] = o < t ? mb_exp(tk.G[t] - tk.G[o]) * kk[r][e] : 0.f;
            }
    }
    const double GL = tk.G[DB_L - 1];
    float* kd = buf.kd + ((size_t)b.rank * H + h) * DB_L * d;
    for (int i = threadIdx.x; i < DB_L * d; i += DB_THREADS) {
        const int t = i / d, n = i % d;
        const float k = k_s[t * dp + (((n >> 2) ^ (t & 7)) << 2) + (n & 3)];
        R_s[t * cols + n] = mb_exp(tk.G[t]) * k;
        kd[i] = mb_exp(GL - tk.G[t]) * k;
    }
    for (int i = threadIdx.x; i < DB_L * E; i += DB_THREADS) {
        const int t = i / E, e = i % E;
        R_s[t * cols + d + e] = t < nt ? row[(size_t)t * channels + 2 * (size_t)G * d + (size_t)h * E + e] : 0.f;
    }
    if (threadIdx.x == 0) buf.decay[(size_t)b.rank * H + h] = mb_exp(GL);
    __syncthreads();
    // A thread a column, sixteen rows at a time: what the rows above them take off, in two sums each (of the even and of the odd rows), then what
    // they take off one another.  Both are formed apart from the right side, which is rounded once at its own size, as in the recurrence
    // (taken off one product at a time it was rounded sixteen times); beta comes last.
    float* W = buf.W + ((size_t)b.rank * H + h) * DB_L * d;
    float* U = buf.U + ((size_t)b.rank * H + h) * DB_L * E;
    for (int col = threadIdx.x; col < cols; col += DB_THREADS) {
        float* out = col < d ? W + col : U + (col - d);
        const int pitch = col < d ? d : E;
        for (int r0 = 0; r0 < DB_L; r0 += 16) {
            f32x2 s2[16];
#pragma unroll
            for (int t = 0; t < 16; t++) s2[t] = mm_pair(0.f, 0.f);
            for (int o = 0; o < r0; o += 4) {
                const f32x2 x0 = mm_pair(R_s[o * cols + col], R_s[(o + 1) * cols + col]), x1 = mm_pair(R_s[(o + 2) * cols + col], R_s[(o + 3) * cols + col]);
#pragma unroll
                for (int t = 0; t < 16; t++) {
                    const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(A_s + (r0 + t) * DB_L + o);
                    s2[t] = mm_fma2(a.x, x0, s2[t]);
                    s2[t] = mm_fma2(a.y, x1, s2[t]);
                }
            }
            float x[16];
#pragma unroll
            for (int t = 0; t < 16; t++) {
                const float* a = A_s + (r0 + t) * DB_L + r0;
                float in = 0.f;
#pragma unroll
                for (int o = 0; o < 16; o++)
                    if (o < t) in = fmaf(a[o], x[o], in);
                const float2 v = mm_unpair(s2[t]);
                x[t] = tk.beta[r0 + t] * (R_s[(r0 + t) * cols + col] - ((v.x + v.y) + in));
                out[(r0 + t) * pitch] = x[t];
            }
#pragma unroll
            for (int t = 0; t < 16; t++) R_s[(r0 + t) * cols + col] = x[t];
        }
    }
}

__device__ __forceinline__ void db_fetch16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

// grid (segments, heads, runs of 16 columns).  W S0: thread (token group of four, column group of four, quarter of the key
// entries); k^T u: thread (key entries of four, column group, half of the tokens); the shares are added in their order.
__global__ void __launch_bounds__(DB_THREADS) delta_states_kernel(const MMSegment* __restrict__ segs, int n_segs, float* state, long long state_stride,
                                                                  DBBuffers buf, int H, int d, int E, int longest) {
    extern __shared__ __align__(16) float mm_smem[];
    const MMSegment s = segs[blockIdx.x];
    int rank = 0;
    for (int i = 0; i < (int)blockIdx.x; i++) rank += segs[i].count > longest ? (segs[i].count + DB_L - 1) / DB_L : 0;
    pdl_launch_dependents();
    pdl_wait(KID_MATRIX_MEMORY);
    if (s.count <= longest) return;
    const int blocks = (s.count + DB_L - 1) / DB_L, h = blockIdx.y, c0 = blockIdx.z * DB_COLS, tid = threadIdx.x;
    const int wp = d + 4;                        // (a row's pitch: four more, so that neighbouring rows' chunks lie in other banks)
    float* W_s = mm_smem;                        // [2][64][wp]
    float* k_s = W_s + 2 * DB_L * wp;            // [2][64][d]
    float* S_s = k_s + 2 * DB_L * d;             // [d][16]
    float* u_s = S_s + d * DB_COLS;              // [64][16]
    float* share = u_s + DB_L * DB_COLS;         // [4][64][16], or [2][d][16]
    const int live = min(DB_COLS, E - c0);       // (a multiple of four)
    float* slot = state + (size_t)s.slot * state_stride + (size_t)h * d * E;
    for (int i = tid; i < d * DB_COLS; i += DB_THREADS) {
        const int n = i / DB_COLS, c = i % DB_COLS;
        S_s[i] = s.before > 0 && c < live ? slot[(size_t)n * E + c0 + c] : 0.f;
    }
    auto fetch = [&](int b) {
        const size_t at = ((size_t)(rank + b) * H + h) * DB_L * d;
        for (int i = tid; i < DB_L * d / 4; i += DB_THREADS) {
            const int t = i / (d / 4), n = i % (d / 4) * 4;
            db_fetch16(W_s + ((b & 1) * DB_L + t) * wp + n, buf.W + at + (size_t)t * d + n);
            db_fetch16(k_s + ((b & 1) * DB_L + t) * d + n, buf.kd + at + (size_t)t * d + n);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    fetch(0);
    for (int b = 0; b < blocks; b++) {
        const size_t bh = (size_t)(rank + b) * H + h;
        // this block's U and decay, and the next block's rows, are on their way while the products before them run
        float U4[4];
        const float dec = buf.decay[bh];
        float* Ub = buf.U + bh * DB_L * E + c0;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int i = tid + j * DB_THREADS, t = i / DB_COLS, c = i % DB_COLS;
            U4[j] = c < live ? Ub[(size_t)t * E + c] : 0.f;
        }
        if (b + 1 < blocks) fetch(b + 1); else asm volatile("cp.async.commit_group;\n" ::: "memory");
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        __syncthreads();
        float* Sb = buf.S + bh * d * E + c0;
        for (int i = tid; i < d * DB_COLS; i += DB_THREADS) {
            const int n = i / DB_COLS, c = i % DB_COLS;
            if (c < live) Sb[(size_t)n * E + c] = S_s[i];
        }
        {
            const int cg = tid & 3, tg = (tid >> 2) & 15, part = tid >> 6, per = ((d / 4 + 3) / 4) * 4, n0 = part * per, n1 = min(d, n0 + per);
            const float* W = W_s + (b & 1) * DB_L * wp;
            float acc[4][4];
#pragma unroll
            for (int r = 0; r < 4; r++)
#pragma unroll
                for (int e = 0; e < 4; e++) acc[r][e] = 0.f;
            for (int n = n0; n < n1; n += 4) {
                float4 w[4];
#pragma unroll
                for (int r = 0; r < 4; r++) w[r] = *reinterpret_cast<const float4*>(W + (tg + 16 * r) * wp + n);
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const float4 x = *reinterpret_cast<const float4*>(S_s + (n + j) * DB_COLS + cg * 4);
#pragma unroll
                    for (int r = 0; r < 4; r++) {
                        const float l = j == 0 ? w[r].x : j == 1 ? w[r].y : j == 2 ? w[r].z : w[r].w;
                        acc[r][0] = fmaf(l, x.x, acc[r][0]); acc[r][1] = fmaf(l, x.y, acc[r][1]);
                        acc[r][2] = fmaf(l, x.z, acc[r][2]); acc[r][3] = fmaf(l, x.w, acc[r][3]);
                    }
                }
            }
#pragma unroll
            for (int r = 0; r < 4; r++)
                *reinterpret_cast<float4*>(share + (part * DB_L + tg + 16 * r) * DB_COLS + cg * 4) = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int i = tid + j * DB_THREADS, t = i / DB_COLS, c = i % DB_COLS;
            float v = share[i];
#pragma unroll
            for (int p = 1; p < 4; p++) v += share[p * DB_L * DB_COLS + i];
            v = U4[j] - v;
            u_s[i] = v;
            if (c < live) Ub[(size_t)t * E + c] = v;
        }
        __syncthreads();
        for (int x = tid; x < (d / 4) * 8; x += DB_THREADS) {
            const int cg = x & 3, ng = (x >> 2) % (d / 4), part = x / d;
            const float* k = k_s + (b & 1) * DB_L * d + ng * 4;
            float acc[4][4];
#pragma unroll
            for (int r = 0; r < 4; r++)
#pragma unroll
                for (int e = 0; e < 4; e++) acc[r][e] = 0.f;
#pragma unroll 4
            for (int t = part * (DB_L / 2); t < (part + 1) * (DB_L / 2); t++) {
                const float4 kv = *reinterpret_cast<const float4*>(k + t * d);
                const float4 uv = *reinterpret_cast<const float4*>(u_s + t * DB_COLS + cg * 4);
                const float kk[4] = {kv.x, kv.y, kv.z, kv.w};
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    acc[r][0] = fmaf(kk[r], uv.x, acc[r][0]); acc[r][1] = fmaf(kk[r], uv.y, acc[r][1]);
                    acc[r][2] = fmaf(kk[r], uv.z, acc[r][2]); acc[r][3] = fmaf(kk[r], uv.w, acc[r][3]);
                }
            }
#pragma unroll
            for (int r = 0; r < 4; r++)
                *reinterpret_cast<float4*>(share + (part * d + ng * 4 + r) * DB_COLS + cg * 4) = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
        }
        __syncthreads();
        for (int i = tid; i < d * DB_COLS; i += DB_THREADS) S_s[i] = fmaf(dec, S_s[i], share[i] + share[d * DB_COLS + i]);
        __syncthreads();
    }
    for (int i = tid; i < d * DB_COLS; i += DB_THREADS) {
        const int n = i / DB_COLS, c = i % DB_COLS;
        if (c < live) slot[(size_t)n * E + c0 + c] = S_s[i];
    }
}

// grid (blocks, heads, column tiles).  A thread has tokens ty + 16 a, and keys tx + 16 b or the columns 4 tx .. 4 tx + 3.
__global__ void __launch_bounds__(DB_THREADS, 2) delta_outputs_kernel(const float* c, int channels, const float* ba, const float* __restrict__ a_log,
                                                                   const float* __restrict__ dt_bias, const MMSegment* __restrict__ segs, int n_segs,
                                                                   DBBuffers buf, float* __restrict__ y, int H, int G, int d, int E, int longest) {
    extern __shared__ __align__(16) float mm_smem[];
    __shared__ DBTokens tk;
    __shared__ float a_s[DB_L];
    const MMBlock b = mm_find_block(segs, n_segs, blockIdx.x, DB_L, longest);
    pdl_launch_dependents();
    pdl_wait(KID_MATRIX_MEMORY);
    if (b.seg < 0) return;
    const MMSegment s = segs[b.seg];
    if (s.count <= longest) return;
    const int h = blockIdx.y, kh = h / (H / G), c0 = blockIdx.z * DB_C, begin = b.tb * DB_L, nt = min(DB_L, s.count - begin), dp = (d + 31) & ~31;
    const size_t tok0 = (size_t)s.first + begin;
    float* q_s = mm_smem;                        // [64][dp]
    float* k_s = q_s + DB_L * dp;                // [64][dp]; then the state the block starts from, [d][64]
    float* u_s = k_s + (dp > DB_L ? DB_L * dp : DB_L * DB_L);       // [64][64]
    float* p_s = u_s + DB_L * DB_C;              // [64][64]
    const float* row = c + tok0 * channels;
    db_tokens(tk, ba, tok0, nt, h, H, -expf(a_log[h]), dt_bias[h]);
    db_unit_rows(row + (size_t)kh * d, channels, nt, d, q_s, dp, rsqrtf((float)d));
    db_unit_rows(row + (size_t)G * d + (size_t)kh * d, channels, nt, d, k_s, dp, 1.f);
    mb_rows(buf.U + ((size_t)b.rank * H + h) * DB_L * E + c0, E, nt, min(DB_C, E - c0), u_s, DB_C, 1.f, false);
    __syncthreads();
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4, chunks = d / 4;
    if (threadIdx.x < DB_L) a_s[threadIdx.x] = mb_exp(tk.G[threadIdx.x]);
    {
        float qk[4][4];
        db_product(q_s, k_s, dp, chunks, tx, ty, qk);
#pragma unroll
        for (int r = 0; r < 4; r++)
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const int t = ty + 16 * r, o = tx + 16 * e;
                p_s[t * DB_L + o] = o <= t ? mb_exp(tk.G[t] - tk.G[o]) * qk[r][e] : 0.f;
            }
    }
    __syncthreads();                             // the weights are there, the keys have been read
    const float* S = buf.S + ((size_t)b.rank * H + h) * d * E + c0;
    for (int i = threadIdx.x; i < d * (DB_C / 4); i += DB_THREADS) {
        const int n = i / (DB_C / 4), cc = i % (DB_C / 4) * 4;
        *reinterpret_cast<float4*>(k_s + n * DB_C + cc) = c0 + cc < E ? *reinterpret_cast<const float4*>(S + (size_t)n * E + cc) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __syncthreads();                             // the state is there
    // (sums of 16 products at most, added to the others when they are complete: short chains round less)
    f32x2 acc[4][2], run[4][2];
#pragma unroll
    for (int r = 0; r < 4; r++) acc[r][0] = acc[r][1] = run[r][0] = run[r][1] = mm_pair(0.f, 0.f);
    // (a weight of zero adds nothing: a later token's write may be an infinity)
    auto four = [&](const float4 (&left)[4], const float* right) {
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(right + j * DB_C + tx * 4);
#pragma unroll
            for (int r = 0; r < 4; r++) {
                const float l = j == 0 ? left[r].x : j == 1 ? left[r].y : j == 2 ? left[r].z : left[r].w;
                const f32x2 l2 = mm_pair(l, l);
                if (l != 0.f) {
                    run[r][0] = mm_fma2(l2, v.x, run[r][0]);
                    run[r][1] = mm_fma2(l2, v.y, run[r][1]);
                }
            }
        }
    };
    const f32x2 one = mm_pair(1.f, 1.f);
    auto settle = [&]() {
#pragma unroll
        for (int r = 0; r < 4; r++)
#pragma unroll
            for (int x = 0; x < 2; x++) { acc[r][x] = mm_fma2(one, run[r][x], acc[r][x]); run[r][x] = mm_pair(0.f, 0.f); }
    };
#pragma unroll 2
    for (int cc = 0; cc < chunks; cc++) {
        float4 q[4];
#pragma unroll
        for (int r = 0; r < 4; r++) { const int t = ty + 16 * r; q[r] = *reinterpret_cast<const float4*>(q_s + t * dp + ((cc ^ (t & 7)) << 2)); }
        four(q, k_s + cc * 4 * DB_C);
        if ((cc & 3) == 3 || cc == chunks - 1) settle();
    }
#pragma unroll
    for (int r = 0; r < 4; r++) {
        const float a = a_s[ty + 16 * r];
        acc[r][0] = mm_mul2(mm_pair(a, a), acc[r][0]);
        acc[r][1] = mm_mul2(mm_pair(a, a), acc[r][1]);
    }
#pragma unroll 2
    for (int k = 0; k < DB_L; k += 4) {
        float4 p[4];
#pragma unroll
        for (int r = 0; r < 4; r++) p[r] = *reinterpret_cast<const float4*>(p_s + (ty + 16 * r) * DB_L + k);
        four(p, u_s + k * DB_C);
        if ((k & 15) == 12) settle();
    }
#pragma unroll
    for (int r = 0; r < 4; r++) {
        const int t = ty + 16 * r;
        if (t >= nt || c0 + tx * 4 >= E) continue;
        const float2 x0 = mm_unpair(acc[r][0]), x1 = mm_unpair(acc[r][1]);
        *reinterpret_cast<float4*>(y + (tok0 + t) * H * E + (size_t)h * E + c0 + tx * 4) = make_float4(x0.x, x0.y, x1.x, x1.y);
    }
}

// grid (segments, runs of 256 channels): a longer segment's last taps - 1 inputs into the slot (oldest first), when the
// convolution of this step has read the ones before.  A longer segment has more tokens than taps.
template <typename T>
__global__ void __launch_bounds__(256) delta_conv_state_kernel(const T* u, int u_width, int conv_in_off, const MMSegment* __restrict__ segs, float* state,
                                                               long long state_stride, long long conv_off, int channels, int taps, int longest) {
    const MMSegment s = segs[blockIdx.x];
    pdl_launch_dependents();
    pdl_wait(KID_MATRIX_MEMORY);
    const int ch = blockIdx.y * 256 + threadIdx.x;
    if (s.count <= longest || ch >= channels) return;
    float* cs = state + (size_t)s.slot * state_stride + conv_off;
    for (int k = 0; k < taps - 1; k++) cs[(size_t)k * channels + ch] = to_f32(u[(size_t)(s.first + s.count - (taps - 1) + k) * u_width + conv_in_off + ch]);
}

// Whether segments of more than `longest` tokens take this path: keys of 32 entries or more (with 64 tokens over eight directions U and W S0 nearly
// cancel, and the writes come out 5 to 17 % further from 64-bit arithmetic than the recurrence's), whole vectors of four, and what delta_solve_kernel and
// delta_states_kernel keep in shared memory.
static inline size_t db_solve_smem(int d, int E) { return (size_t)(DB_L * ((d + 31) & ~31) + DB_L * DB_L + DB_L * (d + E)) * sizeof(float); }
static inline size_t db_states_smem(int d) {
    const int share = 4 * DB_L * DB_COLS > 2 * d * DB_COLS ? 4 * DB_L * DB_COLS : 2 * d * DB_COLS;
    return (size_t)(2 * DB_L * (d + 4) + 2 * DB_L * d + d * DB_COLS + DB_L * DB_COLS + share) * sizeof(float);
}
static inline bool db_takes(int channels, int d, int E, int max_segment_tokens, int longest) {
    return longest >= DB_L && max_segment_tokens > longest && d >= 32 && d % 4 == 0 && d <= DB_MAX_D && E % 4 == 0 && channels % 4 == 0 && db_solve_smem(d, E) <= 200 * 1024;
}

template <typename T>
static void launch_delta_blocks(const float* c, int channels, const float* ba, const float* a_log, const float* dt_bias, const T* u, int u_width,
                                const MMSegment* segs, int n_segs, float* state, long long state_stride, long long conv_off, int taps,
                                const DBBuffers& buf, float* y, int n_tokens, int H, int G, int d, int E, int longest, cudaStream_t stream) {
    const int dp = (d + 31) & ~31, blocks = n_tokens / DB_L + n_segs;
    const size_t solve = db_solve_smem(d, E), states = db_states_smem(d);
    const size_t outputs = (size_t)(DB_L * dp + (dp > DB_L ? DB_L * dp : DB_L * DB_L) + 2 * DB_L * DB_C) * sizeof(float);
    cudaFuncSetAttribute(delta_solve_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)solve);
    cudaFuncSetAttribute(delta_states_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)states);
    cudaFuncSetAttribute(delta_outputs_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)outputs);
    launch_chained(delta_solve_kernel, dim3(blocks, H), dim3(DB_THREADS), solve, stream, c, channels, ba, a_log, dt_bias, segs, n_segs, buf, H, G, d, E, longest);
    launch_chained(delta_states_kernel, dim3(n_segs, H, (E + DB_COLS - 1) / DB_COLS), dim3(DB_THREADS), states, stream, segs, n_segs, state, state_stride,
                   buf, H, d, E, longest);
    launch_chained(delta_outputs_kernel, dim3(blocks, H, (E + DB_C - 1) / DB_C), dim3(DB_THREADS), outputs, stream, c, channels, ba, a_log, dt_bias, segs,
                   n_segs, buf, y, H, G, d, E, longest);
    if (taps > 1)
        launch_chained(delta_conv_state_kernel<T>, dim3(n_segs, (channels + 255) / 256), dim3(256), 0, stream, u, u_width, 0, segs, state, state_stride,
                       conv_off, channels, taps, longest);
}
