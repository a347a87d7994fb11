// The matrix LSTM over a prompt's portion in blocks of 64 tokens that run AT THE SAME TIME (matrix_memory.cu has the recurrence
// token by token, for decoded tokens and short portions, and says what is computed).
//
// (The chunkwise form of the matrix LSTM: Beck et al., "xLSTM: Extended Long Short-Term Memory", 2024, and "Tiled Flash Linear Attention", 2025.)
// With the running maximum m known for every token, the recurrence is linear: S_t = a_t S_(t-1) + b_t k_t v_t^T with
// a_t = exp(f_t + m_(t-1) - m_t) and b_t = exp(i_t - m_t), both at most one.  With F the sum of f since a block's start and m0, S0
// what the block starts from, token t's numerator is
//     sum_{s <= t} exp(F_t - F_s + i_s - m_t) (q_t . k_s) v_s  +  exp(F_t + m0 - m_t) S0^T q_t
// and the normaliser's product likewise with one in the place of v_s: a block is a few small float products.
//   mlstm_gates_kernel          f, i and m of every token: a scan over (sum of f, maximum) in pairs, a head a CTA
//   mlstm_contributions_kernel  what a block adds to the state: sum_s exp(F_L - F_s + i_s - m_L) k_s v_s^T, and its decay
//   mlstm_starts_kernel         the state that every block starts from, block after block; the last one's end into the slot
//   mlstm_outputs_kernel        the sums above
// Sums of f and the exponents are formed in double (a block's sum may be a thousand times a difference within it); products and sums of values are float, as in the recurrence.  Nothing is divided by a decay.
//
// What bounds the recurrence is its chain (240 ns a token and head, 32 CTAs at work for one prompt); what bounds the blocks is
// the reads from shared memory behind their products.  1016 tokens beside 8 decoded ones, 4 heads of 128 x 256 (us, caches cold): the
// recurrence 244; these kernels 8 + 17 + 14 + 40, and 11 for the decoded tokens.  A segment that is not long goes through the recurrence
// all the same (kernels/ops.py, MLSTM_LONGEST).
#pragma once

#include "matrix_memory.cuh"

#define MB_L 64                // tokens a block
#define MB_C 64                // value columns a CTA
#define MB_THREADS 256
#define MB_MAX_D 256

struct MBBuffers {
    float* gates;              // [tokens][H][3]: f, i, m
    float* S;                  // [blocks of longer segments][H][d][E]: what the block adds, then what it starts from
    float* n;                  // [blocks][H][d], likewise
    float* decay;              // [blocks][H][2]: the block's decay, the m it starts from
};
// (longest: the tokens of the longest segment that goes token by token; MB_L at least)
static inline long long mb_blocks(int n_tokens, int n_segs, int longest) {
    const int longer = n_tokens / (longest + 1);
    return n_tokens / MB_L + (n_segs < longer ? n_segs : longer) + 1;
}
static inline long long mb_floats(int n_tokens, int n_segs, int longest, int H, int d, int E) {
    return mb_blocks(n_tokens, n_segs, longest) * H * ((long long)d * E + d + 4) + 3LL * n_tokens * H + 16;
}
static inline MBBuffers mb_buffers(float* at, int n_tokens, int n_segs, int longest, int H, int d, int E) {
    const long long nb = mb_blocks(n_tokens, n_segs, longest);
    MBBuffers b;
    b.S = at;                                              // (16-byte rows: d and E are multiples of four)
    b.n = b.S + nb * H * d * E;
    b.decay = b.n + nb * H * d;
    b.gates = b.decay + nb * H * 2;
    return b;
}

// grid (segments, heads)
__global__ void __launch_bounds__(MB_THREADS) mlstm_gates_kernel(const float* gates, const float* __restrict__ i_bias, const float* __restrict__ f_bias,
                                                                 float cap, const MMSegment* __restrict__ segs, const float* state,
                                                                 long long state_stride, MBBuffers buf, int H, int d, int E, int longest) {
    // eight warps scan 128 tokens each, then each takes what the warps before it left
    __shared__ double warp_F[MB_THREADS / 32], warp_M[MB_THREADS / 32], carry;
    const MMSegment s = segs[blockIdx.x];
    pdl_launch_dependents();
    pdl_wait(KID_MATRIX_MEMORY);
    if (s.count <= longest) return;
    const int h = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float bi = i_bias[h], bf = f_bias[h];
    double m = s.before > 0 ? (double)state[(size_t)s.slot * state_stride + (size_t)H * d * E + (size_t)H * d + h] : 0.0;
    for (int t0 = 0; t0 < s.count; t0 += 1024) {
        float2 g[4];
        double F[4], M[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int t = t0 + warp * 128 + j * 32 + lane;
            g[j] = make_float2(0.f, -CUDART_INF_F);
            if (t < s.count) {
                const float* r = gates + (size_t)(s.first + t) * 2 * H;
                g[j] = make_float2(mm_logsigmoid(cap * tanhf((r[H + h] + bf) / cap)), cap * tanhf((r[h] + bi) / cap));
            }
        }
        double Fw = 0.0, Mw = -CUDART_INF;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            F[j] = g[j].x; M[j] = g[j].y;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const double Fl = __shfl_up_sync(0xffffffffu, F[j], o), Ml = __shfl_up_sync(0xffffffffu, M[j], o);
                if (lane >= o) { M[j] = fmax(M[j], Ml + F[j]); F[j] += Fl; }
            }
            M[j] = fmax(M[j], Mw + F[j]); F[j] += Fw;
            Fw = __shfl_sync(0xffffffffu, F[j], 31); Mw = __shfl_sync(0xffffffffu, M[j], 31);
        }
        if (lane == 31) { warp_F[warp] = Fw; warp_M[warp] = Mw; }
        __syncthreads();
        for (int w = 0; w < warp; w++) m = fmax(m + warp_F[w], warp_M[w]);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int t = t0 + warp * 128 + j * 32 + lane;
            const double here = fmax(m + F[j], M[j]);
            if (t < s.count) {
                float* to = buf.gates + ((size_t)(s.first + t) * H + h) * 3;
                to[0] = g[j].x; to[1] = g[j].y; to[2] = (float)here;
            }
            if (warp == MB_THREADS / 32 - 1 && j == 3 && lane == 31) carry = here;
        }
        __syncthreads();
        m = carry;
    }
}

// exp(x), at most one, of an exponent in double: its rounding to float would be an error of 2^-24 of its size, so what the
// rounding left goes in as a factor.
__device__ __forceinline__ float mb_exp(double x) {
    const float hi = (float)x, e = expf(hi);
    return fmaf(e, (float)(x - (double)hi), e);
}

// What every thread of a block's CTA needs of its tokens: F and i in double, m (m0 behind the last), by the CTA's first warp.
struct MBTokens { double F[MB_L]; float i[MB_L], m[MB_L]; float m0; };
__device__ __forceinline__ void mb_tokens(MBTokens& tk, const MBBuffers& buf, size_t tok0, int nt, int h, int H, float m0) {
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        double before = 0.0;
#pragma unroll
        for (int c = 0; c < MB_L; c += 32) {
            const int t = c + lane;
            const float* g = buf.gates + ((tok0 + (t < nt ? t : 0)) * H + h) * 3;
            double F = t < nt ? (double)g[0] : 0.0;
            tk.i[t] = t < nt ? g[1] : 0.f;
            tk.m[t] = t < nt ? g[2] : 0.f;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const double l = __shfl_up_sync(0xffffffffu, F, o);
                if (lane >= o) F += l;
            }
            F += before;
            tk.F[t] = F;
            before = __shfl_sync(0xffffffffu, F, 31);
        }
        if (lane == 0) tk.m0 = m0;
    }
}
// rows of `width` entries (a multiple of four) of 64 tokens from src (row stride in entries) to shared memory, `pitch` floats a row,
// zeros for tokens past nt and columns past `width`; swz: 16-byte chunk c of row r at c ^ (r & 7)
template <typename T>
__device__ __forceinline__ void mb_rows(const T* src, long long stride, int nt, int width, float* dst, int pitch, float scale, bool swz) {
    const int chunks = pitch / 4;
    for (int i = threadIdx.x; i < MB_L * chunks; i += MB_THREADS) {
        const int t = i / chunks, c = i % chunks;
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        if (t < nt && c * 4 < width) head_quad_load(src + (long long)t * stride + c * 4, v);
        *reinterpret_cast<float4*>(dst + t * pitch + ((swz ? c ^ (t & 7) : c) << 2)) = make_float4(v[0] * scale, v[1] * scale, v[2] * scale, v[3] * scale);
    }
}

// grid (blocks, heads, column tiles).  A thread has 4 x 4 entries of the state's change at a time: a chunk of k by a chunk of v.
template <typename T>
__global__ void __launch_bounds__(MB_THREADS) mlstm_contributions_kernel(const T* u, int u_width, const MMSegment* __restrict__ segs, int n_segs,
                                                                         const float* state, long long state_stride, MBBuffers buf, int H, int d, int E, int longest) {
    extern __shared__ __align__(16) float mm_smem[];
    __shared__ MBTokens tk;
    __shared__ float w_s[MB_L];
    const MMBlock b = mm_find_block(segs, n_segs, blockIdx.x, MB_L, longest);
    pdl_launch_dependents();
    pdl_wait(KID_MATRIX_MEMORY);
    if (b.seg < 0) return;
    const MMSegment s = segs[b.seg];
    if (s.count <= longest) return;
    const int h = blockIdx.y, c0 = blockIdx.z * MB_C, begin = b.tb * MB_L, nt = min(MB_L, s.count - begin), dp = (d + 31) & ~31;
    const size_t tok0 = (size_t)s.first + begin;
    float* k_s = mm_smem;                        // [64][dp]
    float* v_s = k_s + MB_L * dp;                // [64][64]
    const float m0 = b.tb > 0 ? buf.gates[((tok0 - 1) * H + h) * 3 + 2]
                              : s.before > 0 ? state[(size_t)s.slot * state_stride + (size_t)H * d * E + (size_t)H * d + h] : 0.f;
    mb_tokens(tk, buf, tok0, nt, h, H, m0);
    const T* row = u + tok0 * u_width;
    mb_rows(row + (size_t)H * d + (size_t)h * d, u_width, nt, d, k_s, dp, 1.f, true);
    mb_rows(row + 2 * (size_t)H * d + (size_t)h * E + c0, u_width, nt, min(MB_C, E - c0), v_s, MB_C, 1.f, false);
    __syncthreads();
    if (threadIdx.x < MB_L) {
        const int t = threadIdx.x;
        w_s[t] = t < nt ? mb_exp(tk.F[nt - 1] - tk.F[t] + (double)tk.i[t] - (double)tk.m[nt - 1]) : 0.f;
    }
    __syncthreads();
    float* Sb = buf.S + ((size_t)b.rank * H + h) * d * E;
    const int n_chunks = d / 4;
    const int tx = threadIdx.x & 15;
    for (int cn = threadIdx.x >> 4; cn < n_chunks; cn += 32) {
        const bool two = cn + 16 < n_chunks;
        f32x2 acc[2][4][2];
#pragma unroll
        for (int z = 0; z < 2; z++)
#pragma unroll
            for (int r = 0; r < 4; r++) acc[z][r][0] = acc[z][r][1] = mm_pair(0.f, 0.f);
#pragma unroll 4
        for (int t = 0; t < MB_L; t++) {
            const float w = w_s[t];
            const float4 v = *reinterpret_cast<const float4*>(v_s + t * MB_C + tx * 4);
            const f32x2 v0 = mm_pair(v.x * w, v.y * w), v1 = mm_pair(v.z * w, v.w * w);
#pragma unroll
            for (int z = 0; z < 2; z++) {
                const int c = z && two ? cn + 16 : cn;
                const float4 k = *reinterpret_cast<const float4*>(k_s + t * dp + ((c ^ (t & 7)) << 2));
                const float kk[4] = {k.x, k.y, k.z, k.w};
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    const f32x2 k2 = mm_pair(kk[r], kk[r]);
                    acc[z][r][0] = mm_fma2(k2, v0, acc[z][r][0]);
                    acc[z][r][1] = mm_fma2(k2, v1, acc[z][r][1]);
                }
            }
        }
        if (c0 + tx * 4 < E)
#pragma unroll
            for (int z = 0; z < 2; z++) {
                if (z && !two) break;
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    const float2 x0 = mm_unpair(acc[z][r][0]), x1 = mm_unpair(acc[z][r][1]);
                    *reinterpret_cast<float4*>(Sb + (size_t)((cn + 16 * z) * 4 + r) * E + c0 + tx * 4) = make_float4(x0.x, x0.y, x1.x, x1.y);
                }
            }
    }
    if (blockIdx.z == 0) {
        for (int n = threadIdx.x; n < d; n += MB_THREADS) {
            float acc = 0.f;
            for (int t = 0; t < MB_L; t++) acc = fmaf(w_s[t], k_s[t * dp + (((n >> 2) ^ (t & 7)) << 2) + (n & 3)], acc);
            buf.n[((size_t)b.rank * H + h) * d + n] = acc;
        }
        if (threadIdx.x == 0) {
            float* to = buf.decay + ((size_t)b.rank * H + h) * 2;
            to[0] = mb_exp(tk.F[nt - 1] + (double)tk.m0 - (double)tk.m[nt - 1]);
            to[1] = tk.m0;
        }
    }
}

// grid (segments, heads, runs of 256 entries of S and n)
__global__ void __launch_bounds__(256) mlstm_starts_kernel(const MMSegment* __restrict__ segs, int n_segs, float* state, long long state_stride,
                                                           MBBuffers buf, int H, int d, int E, int longest) {
    const MMSegment s = segs[blockIdx.x];
    int rank = 0;
    for (int i = 0; i < (int)blockIdx.x; i++) rank += segs[i].count > longest ? (segs[i].count + MB_L - 1) / MB_L : 0;
    pdl_launch_dependents();
    pdl_wait(KID_MATRIX_MEMORY);
    if (s.count <= longest) return;
    const int blocks = (s.count + MB_L - 1) / MB_L, h = blockIdx.y;
    const long long i = blockIdx.z * 256LL + threadIdx.x, entries = (long long)d * E;
    if (i >= entries + d) return;
    float* slot = state + (size_t)s.slot * state_stride;
    float* end = i < entries ? slot + h * entries + i : slot + H * entries + (long long)h * d + (i - entries);
    float* x = i < entries ? buf.S + ((size_t)rank * H + h) * entries + i : buf.n + ((size_t)rank * H + h) * d + (i - entries);
    const size_t step = (size_t)H * (i < entries ? entries : d);
    const float* a = buf.decay + ((size_t)rank * H + h) * 2;
    float cur = s.before > 0 ? *end : 0.f;
    for (int b0 = 0; b0 < blocks; b0 += 8) {           // (eight blocks' loads leave before the first is used)
        float add[8], dec[8];
#pragma unroll
        for (int j = 0; j < 8; j++) {
            add[j] = b0 + j < blocks ? x[(b0 + j) * step] : 0.f;
            dec[j] = b0 + j < blocks ? a[(size_t)(b0 + j) * H * 2] : 0.f;
        }
#pragma unroll
        for (int j = 0; j < 8; j++) {
            if (b0 + j >= blocks) break;
            x[(b0 + j) * step] = cur;
            cur = fmaf(dec[j], cur, add[j]);
        }
    }
    *end = cur;
    if (i == 0) slot[H * entries + (long long)H * d + h] = buf.gates[((size_t)(s.first + s.count - 1) * H + h) * 3 + 2];
}

// grid (blocks, heads, column tiles).  A thread has tokens ty + 16 a, and keys tx + 16 b or the columns 4 tx .. 4 tx + 3.
template <typename T>
__global__ void __launch_bounds__(MB_THREADS) mlstm_outputs_kernel(const T* u, int u_width, const MMSegment* __restrict__ segs, int n_segs,
                                                                   MBBuffers buf, float* __restrict__ y, float* __restrict__ dn, int H, int d, int E,
                                                                   int longest) {
    extern __shared__ __align__(16) float mm_smem[];
    __shared__ MBTokens tk;
    __shared__ float a_s[MB_L];
    const MMBlock b = mm_find_block(segs, n_segs, blockIdx.x, MB_L, longest);
    pdl_launch_dependents();
    pdl_wait(KID_MATRIX_MEMORY);
    if (b.seg < 0) return;
    const MMSegment s = segs[b.seg];
    if (s.count <= longest) return;
    const int h = blockIdx.y, c0 = blockIdx.z * MB_C, begin = b.tb * MB_L, nt = min(MB_L, s.count - begin), dp = (d + 31) & ~31;
    const size_t tok0 = (size_t)s.first + begin;
    float* q_s = mm_smem;                        // [64][dp]
    float* k_s = q_s + MB_L * dp;                // [64][dp]; then the state the block starts from, [d][64]
    float* v_s = k_s + MB_L * dp;                // [64][64]
    float* p_s = v_s + MB_L * MB_C;              // [64][64]
    const bool fresh = b.tb == 0 && s.before <= 0;      // (the block starts from nothing)
    mb_tokens(tk, buf, tok0, nt, h, H, buf.decay[((size_t)b.rank * H + h) * 2 + 1]);
    const T* row = u + tok0 * u_width;
    mb_rows(row + (size_t)h * d, u_width, nt, d, q_s, dp, rsqrtf((float)d), true);
    mb_rows(row + (size_t)H * d + (size_t)h * d, u_width, nt, d, k_s, dp, 1.f, true);
    mb_rows(row + 2 * (size_t)H * d + (size_t)h * E + c0, u_width, nt, min(MB_C, E - c0), v_s, MB_C, 1.f, false);
    __syncthreads();
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4, chunks = d / 4;
    if (threadIdx.x < MB_L) {
        const int t = threadIdx.x;
        a_s[t] = t < nt && !fresh ? mb_exp(tk.F[t] + (double)tk.m0 - (double)tk.m[t]) : 0.f;
    }
    float sum[4];
    {
        f32x2 acc[4][4];
#pragma unroll
        for (int r = 0; r < 4; r++)
#pragma unroll
            for (int c = 0; c < 4; c++) acc[r][c] = mm_pair(0.f, 0.f);
#pragma unroll 2
        for (int c = 0; c < chunks; c++) {
            ulonglong2 q[4];
#pragma unroll
            for (int r = 0; r < 4; r++) { const int t = ty + 16 * r; q[r] = *reinterpret_cast<const ulonglong2*>(q_s + t * dp + ((c ^ (t & 7)) << 2)); }
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const int t = tx + 16 * e;
                const ulonglong2 k = *reinterpret_cast<const ulonglong2*>(k_s + t * dp + ((c ^ (t & 7)) << 2));
#pragma unroll
                for (int r = 0; r < 4; r++) { acc[r][e] = mm_fma2(q[r].x, k.x, acc[r][e]); acc[r][e] = mm_fma2(q[r].y, k.y, acc[r][e]); }
            }
        }
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const int t = ty + 16 * r;
            sum[r] = 0.f;
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const int k = tx + 16 * e;
                float p = 0.f;
                if (k <= t && t < nt) {
                    const float2 x = mm_unpair(acc[r][e]);
                    p = mb_exp(tk.F[t] - tk.F[k] + (double)tk.i[k] - (double)tk.m[t]) * (x.x + x.y);
                }
                sum[r] += p;
                p_s[t * MB_L + k] = p;
            }
        }
    }
    __syncthreads();                             // the weights are there, the keys have been read
    if (!fresh) {
        const float* S = buf.S + ((size_t)b.rank * H + h) * d * E + c0;
        for (int i = threadIdx.x; i < d * (MB_C / 4); i += MB_THREADS) {
            const int n = i / (MB_C / 4), c = i % (MB_C / 4) * 4;
            *reinterpret_cast<float4*>(k_s + n * MB_C + c) =
                c0 + c < E ? *reinterpret_cast<const float4*>(S + (size_t)n * E + c) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
    if (blockIdx.z == 0) {
        // the normaliser's product: a row's sixteen threads add their weights, and share out q . n
        const float* n0 = buf.n + ((size_t)b.rank * H + h) * d;
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const int t = ty + 16 * r;
            float qn = 0.f;
            if (!fresh) for (int n = tx; n < d; n += 16) qn = fmaf(q_s[t * dp + (((n >> 2) ^ (t & 7)) << 2) + (n & 3)], n0[n], qn);
            float v = fmaf(a_s[t], qn, sum[r]);
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (tx == 0 && t < nt) {
                float* to = dn + ((tok0 + t) * H + h) * 2;
                to[0] = v; to[1] = expf(-tk.m[t]);
            }
        }
    }
    __syncthreads();                             // the state is there
    f32x2 acc[4][2];
#pragma unroll
    for (int r = 0; r < 4; r++) acc[r][0] = acc[r][1] = mm_pair(0.f, 0.f);
    // four rows of `right` times four entries of `left` of each of this thread's tokens (a weight of zero adds nothing: a later
    // token's value may be an infinity)
    auto four = [&](const float4 (&left)[4], const float* right) {
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(right + j * MB_C + tx * 4);
#pragma unroll
            for (int r = 0; r < 4; r++) {
                const float l = j == 0 ? left[r].x : j == 1 ? left[r].y : j == 2 ? left[r].z : left[r].w;
                const f32x2 l2 = mm_pair(l, l);
                if (l != 0.f) {
                    acc[r][0] = mm_fma2(l2, v.x, acc[r][0]);
                    acc[r][1] = mm_fma2(l2, v.y, acc[r][1]);
                }
            }
        }
    };
    if (!fresh) {
#pragma unroll 2
        for (int c = 0; c < chunks; c++) {
            float4 q[4];
#pragma unroll
            for (int r = 0; r < 4; r++) { const int t = ty + 16 * r; q[r] = *reinterpret_cast<const float4*>(q_s + t * dp + ((c ^ (t & 7)) << 2)); }
            four(q, k_s + c * 4 * MB_C);
        }
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const float a = a_s[ty + 16 * r];
            acc[r][0] = mm_mul2(mm_pair(a, a), acc[r][0]);
            acc[r][1] = mm_mul2(mm_pair(a, a), acc[r][1]);
        }
    }
#pragma unroll 2
    for (int k = 0; k < MB_L; k += 4) {
        float4 p[4];
#pragma unroll
        for (int r = 0; r < 4; r++) p[r] = *reinterpret_cast<const float4*>(p_s + (ty + 16 * r) * MB_L + k);
        four(p, v_s + k * MB_C);
    }
#pragma unroll
    for (int r = 0; r < 4; r++) {
        const int t = ty + 16 * r;
        if (t >= nt || c0 + tx * 4 >= E) continue;
        const float2 x0 = mm_unpair(acc[r][0]), x1 = mm_unpair(acc[r][1]);
        *reinterpret_cast<float4*>(y + (tok0 + t) * H * E + (size_t)h * E + c0 + tx * 4) = make_float4(x0.x, x0.y, x1.x, x1.y);
    }
}

// Whether segments of more than `longest` tokens take this path: rows of whole vectors of four, keys that fit shared memory.
static inline bool mb_takes(const void* u, int u_width, int d, int E, int max_segment_tokens, int longest) {
    return longest >= MB_L && max_segment_tokens > longest && d % 4 == 0 && d <= MB_MAX_D && E % 4 == 0 && u_width % 4 == 0 && ((uintptr_t)u & 15) == 0;
}

template <typename T>
static void launch_mlstm_blocks(const T* u, int u_width, const float* gates, const float* i_bias, const float* f_bias, float cap,
                                const MMSegment* segs, int n_segs, float* state, long long state_stride, const MBBuffers& buf, float* y, float* dn,
                                int n_tokens, int H, int d, int E, int longest, cudaStream_t stream) {
    const int dp = (d + 31) & ~31, blocks = n_tokens / MB_L + n_segs, tiles = (E + MB_C - 1) / MB_C;
    const size_t smem_c = (size_t)(MB_L * dp + MB_L * MB_C) * sizeof(float);
    const size_t smem_o = (size_t)(2 * MB_L * dp + 2 * MB_L * MB_C) * sizeof(float);
    cudaFuncSetAttribute(mlstm_contributions_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_c);
    cudaFuncSetAttribute(mlstm_outputs_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_o);
    launch_chained(mlstm_gates_kernel, dim3(n_segs, H), dim3(MB_THREADS), 0, stream, gates, i_bias, f_bias, cap, segs, (const float*)state,
                   state_stride, buf, H, d, E, longest);
    launch_chained(mlstm_contributions_kernel<T>, dim3(blocks, H, tiles), dim3(MB_THREADS), smem_c, stream, u, u_width, segs, n_segs,
                   (const float*)state, state_stride, buf, H, d, E, longest);
    launch_chained(mlstm_starts_kernel, dim3(n_segs, H, (unsigned)(((long long)d * E + d + 255) / 256)), dim3(256), 0, stream, segs, n_segs, state,
                   state_stride, buf, H, d, E, longest);
    launch_chained(mlstm_outputs_kernel<T>, dim3(blocks, H, tiles), dim3(MB_THREADS), smem_o, stream, u, u_width, segs, n_segs, buf, y, dn, H, d, E, longest);
}
