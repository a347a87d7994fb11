// y[M, N] = x[M, K] . W[N, K]^T in float32 on the fifth-generation tensor cores.  The reference calls a library product
// (crates/pagedllm/src/model/layers.rs:27-35); in true float32 that runs on the CUDA cores.
//
// A float's 24 significant bits are three bfloat16 numbers' eight each, so x = x1 + x2 + x3 and W = w1 + w2 + w3 hold exactly
// (the split after the scheme of Dekker and of Ogita, Rump and Oishi, "Accurate sum and dot product", 2005: round, subtract, round what
// is left), a product of two parts is exact in the tensor cores, and x . W is the sum of the parts' products (without x3 w3,
// 2^-32 of the whole).  Weights that came from a bfloat16 file have w2 = w3 = 0: the tile's flags say so and those products are left
// out, at three instructions for what a bfloat16 product takes one.
//   Sums: the tensor cores add in float but cut off where a rounding would be, so a long sum there drifts towards zero.  A block of 64
// values of k therefore starts from zero, takes the small parts' products first and x1 w1 last (four instructions), and is then
// taken out of tensor memory and added in registers with rounding.
//   Not finite, or so large that a part would be infinite: the entries of such a row of x or of W (a flag each) are computed again by fused
// multiply-adds, as float arithmetic has them; so are those of a row with no value of 2^-100 or more, whose third parts
// would lose bits (what is below 2^-110 has some below bfloat16's least, 2^-133), and those whose sum is not finite: a first part is rounded up, and 1.9999 2^100
// by 2^27 is in float's range where the product of the first parts is not.  (A row of W of nothing but bfloat16's subnormal numbers is its own first part and stays: up to
// six bits fewer of its products are kept, as the tensor cores line them up by their leading zeros.)  Of W the splitting warps say which rows have values that three parts do not
// hold, and those are looked at once more, whole, behind the product (looked at by the splitting warps, which bound a product of few rows, 4096 x 12288 at 33 rows took
// 77 us and not 63).
//
// What bounds it: for many rows the bytes of x's parts on their way from L2 (6 a value and tile of W, against 8 instructions of
// tensor-core time), for few rows W's bytes and their splitting.  Hence tiles of 128 rows of W (the tensor cores' 128-row operand) by up to 256 rows
// of x, and K split over a cluster's CTAs where the tiles alone would leave SMs idle (partial tiles meet in shared memory, added in the order of
// k).  W comes by TMA as it lies, two or three blocks ahead: read by the splitting warps themselves, with eight 16-byte loads a thread under way,
// it came at 2.8 TB/s (4096 x 4096 at 32 rows 35.7 us, this way 26.4).
//
// Sixteen warps: 0-7 take the accumulators out of tensor memory and keep the sums (a lane a row of W); 8-11 split W's blocks
// and store the parts where the tensor cores read them (128-byte swizzle); 12 asks for the parts of x by TMA (a ring of one part of 64 values of k a
// place), 14 for W's blocks; 13 owns the tensor memory and issues.  Every wait is bounded: a thread that gives up raises
// a flag that the others see, all reach the cluster's barriers, and the status word says so (64).
#include <atomic>
#include <type_traits>

#include "tcgen05.cuh"

using namespace tc;

namespace {

constexpr int S_BM = 128, S_BK = 64;                 // rows of W a tile, values of k a block
constexpr int S_PART_W = S_BM * S_BK * 2;            // 16 KB: a part of a block of W
constexpr int S_W = 4 * S_PART_W;                    // the first part of two blocks, the second and the third of one
constexpr int S_TILE_W = S_BM * S_BK * 4;            // 32 KB: a block of W as it lies
constexpr int S_THREADS = 512;
constexpr int S_MAX_RING = 8, S_MAX_W = 3;
constexpr float S_LARGEST = 3.3895313e38f;           // the largest bfloat16: beyond it a part would be infinite
constexpr float S_SMALLEST = 7.8886091e-31f;         // 2^-100: what a third part loses (below 2^-133) of the values beside one of this size is nothing to a float

__device__ __forceinline__ uint32_t s_cluster_addr(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ float4 s_ld_cluster16(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];\n" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ int s_ld_cluster_int(uint32_t addr) {
    int v;
    asm volatile("ld.shared::cluster.s32 %0, [%1];\n" : "=r"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void tmem_ld16(uint32_t addr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(addr));
}
__device__ __forceinline__ float4 lds4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];\n" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void sts16(uint32_t addr, const uint32_t (&v)[4]) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};\n" ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
}

// Two floats to a pair of bfloat16, and what the pair leaves of them (exact).
__device__ __forceinline__ uint32_t part_of(float& a, float& b) {
    const uint32_t h = pack2(a, b);
    a -= __uint_as_float(h << 16);
    b -= __uint_as_float(h & 0xffff0000u);
    return h;
}
__device__ __forceinline__ bool too_large(float v) { return !(fabsf(v) <= S_LARGEST); }      // (NaN too)

// x [rows, K] to its parts [3][rows][K], and a flag for each row that holds a value the parts cannot.  A CTA a row, four values a thread
// and turn.
__global__ void __launch_bounds__(256) split_rows_kernel(const float* x, bf16* __restrict__ parts, int* __restrict__ odd_row, int rows, int K) {
    pdl_launch_dependents();
    pdl_wait(KID_GEMM);
    const int row = blockIdx.x;
    const float* src = x + (size_t)row * K;
    bf16* dst = parts + (size_t)row * K;
    const size_t plane = (size_t)rows * K;
    bool odd = false, large = false, some = false;
    for (int k = threadIdx.x * 4; k < K; k += blockDim.x * 4) {
        float4 v = *reinterpret_cast<const float4*>(src + k);
        odd |= too_large(v.x) | too_large(v.y) | too_large(v.z) | too_large(v.w);
        const float top = fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)));
        large |= top >= S_SMALLEST;
        some |= top > 0.f;
#pragma unroll
        for (int p = 0; p < 3; p++) {
            const uint32_t a = part_of(v.x, v.y), b = part_of(v.z, v.w);
            *reinterpret_cast<uint2*>(dst + p * plane + k) = make_uint2(a, b);
        }
    }
    const bool any_odd = __syncthreads_or(odd), any_large = __syncthreads_or(large), any = __syncthreads_or(some);
    if (threadIdx.x == 0) odd_row[row] = any_odd || (any && !any_large);
}

// The entry as float arithmetic has it, for values that cannot be split: by a warp (K is a multiple of eight).
__device__ __forceinline__ float plain_dot(const float* x, const float* w, int K, int lane) {
    float s = 0.f;
#pragma unroll 1
    for (int k = lane * 4; k < K; k += 128) {
        const float4 a = *reinterpret_cast<const float4*>(x + k), b = *reinterpret_cast<const float4*>(w + k);
        s = fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, s))));
    }
    return warp_sum(s);
}
// Whether three parts of a row are not the row: it has a value that no part can hold, or none beside which a lost bit is nothing.
__device__ __forceinline__ bool row_is_odd(const float* row, int K, int lane) {
    bool odd = false, large = false;
#pragma unroll 1
    for (int k = lane * 4; k < K; k += 128) {
        const float4 v = *reinterpret_cast<const float4*>(row + k);
        odd |= too_large(v.x) | too_large(v.y) | too_large(v.z) | too_large(v.w);
        large |= fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))) >= S_SMALLEST;
    }
    return __any_sync(0xffffffffu, odd) || !__any_sync(0xffffffffu, large);
}
__device__ __forceinline__ bool finite(float v) { return fabsf(v) <= CUDART_MAX_NORMAL_F; }

}  // namespace

// map_x: x's parts as [3][M][K], box 1 x ROWS x 64.  map_w: W as 16-bit halves [N][2 K], box 128 x 64 (32 values of k).
// Grid (tiles of W, splits of K, tiles of x), clusters of the splits.
template <int ROWS, int RING, int WRING, int MAX_SPLITS>
__global__ void __launch_bounds__(S_THREADS, 1) gemm_f32_tcgen05_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                                                                        const float* __restrict__ w, const float* x, const int* odd_row,
                                                                        float* __restrict__ y, int M, int N, int K, int* status) {
    constexpr int PART_X = ROWS * S_BK * 2;
    constexpr uint32_t TMEM_COLS = 2 * ROWS < 32 ? 32 : 2 * ROWS;
    constexpr int HALF = ROWS / 2;                     // columns of an accumulator (rows of x) a warp keeps
    static_assert(HALF % 16 == 0 && RING <= S_MAX_RING && WRING <= S_MAX_W, "whole loads from tensor memory; room for the barriers");
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t wparts = smem_u32(smem), wring = wparts + S_W, ring = wring + WRING * S_TILE_W;
    __shared__ __align__(8) unsigned long long bar_mem[2 * S_MAX_RING + 2 * S_MAX_W + 8];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_mem;
    __shared__ uint32_t odd_w[S_BM / 32], odd_all[S_BM / 32];      // the rows of W that three parts do not hold, a bit each: here, and in any share of k
    __shared__ volatile int need[2][4];                // which parts of a block of W hold anything (a warp's rows each): bit 1 the second, bit 2 the third
    volatile int* abort_flag = &abort_mem;
    const uint32_t xfull = smem_u32(bar_mem), xempty = xfull + 8 * S_MAX_RING, wfull = xempty + 8 * S_MAX_RING, wempty = wfull + 16,
                   accfull = wempty + 16, accempty = accfull + 16, sfull = accempty + 16, sempty = sfull + 8 * S_MAX_W;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int splits = gridDim.y, rank = blockIdx.y;
    const int k_blocks = (K + S_BK - 1) / S_BK;
    const int kb0 = k_blocks * rank / splits, n_kb = k_blocks * (rank + 1) / splits - kb0;
    const int n0 = blockIdx.x * S_BM, m0 = blockIdx.z * ROWS;

    if (threadIdx.x == 0) {
        for (int s = 0; s < RING; s++) {
            mbar_init(xfull + 8 * s, 1);
            mbar_init(xempty + 8 * s, 1);
        }
        for (int b = 0; b < WRING; b++) {
            mbar_init(sfull + 8 * b, 1);
            mbar_init(sempty + 8 * b, 4);
        }
        for (int b = 0; b < 2; b++) {
            mbar_init(wfull + 8 * b, 4);
            mbar_init(wempty + 8 * b, 1);
            mbar_init(accfull + 8 * b, 1);
            mbar_init(accempty + 8 * b, 8);
        }
        abort_mem = 0;
        for (int c = 0; c < S_BM / 32; c++) odd_w[c] = odd_all[c] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::);
        fence_async_smem();
    }
    if (warp == 13) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_slot)), "r"(TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    pdl_launch_dependents();

    float* part = reinterpret_cast<float*>(smem);      // [rows of x][rows of W], once the parts have been read
    if (warp >= 8) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 88;\n" ::);
        if (warp < 12) {
            // ---- W's parts: a warp's 32 rows of the tile; a lane and turn eight values of k of two rows, so that eight lanes
            //      (eight rows, one chunk of 16 bytes each) meet no bank twice, reading or writing -----------------------------
            const int cw = warp - 8;
            const uint32_t lane_row = (cw * 32 + (lane & 7)) * 128;
            const uint32_t from = lane_row + (((lane >> 3) * 2 ^ (lane & 7)) << 4);               // (the chunk behind it: ^ 16)
            const uint32_t to0 = lane_row + (((lane >> 3) ^ (lane & 7)) << 4), to1 = to0 ^ 64;    // (values 0 to 31 of the block, and 32 to 63)
            uint32_t lost = 0;                         // turns of which three parts leave something
            uint32_t filled = 0xfu;                    // turns (eight rows each) whose second and third part are not known to be zero
            for (int i = 0; i < n_kb; i++) {
                const int b = i & 1, ss = i % WRING;
                bool ok = (i < 2 || mbar_wait(wempty + 8 * b, ((i >> 1) - 1) & 1, abort_flag)) && mbar_wait(sfull + 8 * ss, (i / WRING) & 1, abort_flag);
                if (!__all_sync(0xffffffffu, ok)) break;
                const uint32_t src = wring + ss * S_TILE_W, dst = wparts + b * S_PART_W;
                int has = 0;
                bool alone = false;                    // the second and third part's memory is free
#pragma unroll
                for (int g = 0; g < 4; g++) {
                    float4 a[4];
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        a[2 * h] = lds4(src + h * (S_TILE_W / 2) + from + g * 1024);
                        a[2 * h + 1] = lds4(src + h * (S_TILE_W / 2) + (from ^ 16) + g * 1024);
                    }
                    uint32_t left = 0;
                    auto store = [&](uint32_t at) {    // a part of the sixteen values, and what it leaves of them
#pragma unroll
                        for (int h = 0; h < 2; h++) {
                            const uint32_t p[4] = {part_of(a[2 * h].x, a[2 * h].y), part_of(a[2 * h].z, a[2 * h].w),
                                                   part_of(a[2 * h + 1].x, a[2 * h + 1].y), part_of(a[2 * h + 1].z, a[2 * h + 1].w)};
                            sts16(at + (h ? to1 : to0) + g * 1024, p);
                        }
                        left = 0;
#pragma unroll
                        for (int e = 0; e < 4; e++)
                            left |= __float_as_uint(a[e].x) | __float_as_uint(a[e].y) | __float_as_uint(a[e].z) | __float_as_uint(a[e].w);
                    };
                    store(dst);
                    const bool any = __any_sync(0xffffffffu, left != 0);      // (what a part leaves of a value is +0 where it leaves nothing)
                    if (any || (filled >> g & 1)) {
                        if (!alone && i >= 1) ok = __all_sync(0xffffffffu, mbar_wait(wempty + 8 * (b ^ 1), ((i - 1) >> 1) & 1, abort_flag));
                        alone = true;
                        if (left) has |= 2;
                        store(wparts + 2 * S_PART_W);
                        if (left) has |= 4;
                        store(wparts + 3 * S_PART_W);
                        if (left) lost |= 1u << g;     // (so does what is not finite, and what is too large for a part)
                        filled = any ? filled | 1u << g : filled & ~(1u << g);
                    }
                }
                has = __reduce_or_sync(0xffffffffu, has);
                fence_async_smem();
                if (lane == 0) need[b][cw] = has;
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(sempty + 8 * ss);
                    mbar_arrive(wfull + 8 * b);
                }
                if (!ok) break;
            }
            uint32_t rows = 0;
#pragma unroll
            for (int g = 0; g < 4; g++) rows |= (lost >> g & 1) << (g * 8 + (lane & 7));
            rows = __reduce_or_sync(0xffffffffu, rows);
            if (lane == 0) odd_w[cw] = rows;
        } else if (warp == 12) {
            // ---- x's parts, the smallest first ---------------------------------------------------------------------
            pdl_wait(KID_GEMM_TC, lane == 0);
            int it = 0;
            bool ok = true;
            for (int i = 0; i < n_kb && ok; i++)
                for (int p = 2; p >= 0; p--, it++) {
                    const int s = it % RING;
                    if (it >= RING && !__all_sync(0xffffffffu, mbar_wait(xempty + 8 * s, ((it / RING) - 1) & 1, abort_flag))) { ok = false; break; }
                    if (elect_one()) {
                        mbar_expect_tx(xfull + 8 * s, PART_X);
                        tma_load_3d(ring + s * PART_X, &map_x, (kb0 + i) * S_BK, m0, p, xfull + 8 * s);
                    }
                }
            if (!ok) {
                // nothing may still be on its way into this CTA's memory when it leaves
                int ignored = 0;
                for (int j = it > RING ? it - RING : 0; j < it; j++) mbar_wait(xfull + 8 * (j % RING), (j / RING) & 1, &ignored);
            }
        } else if (warp == 14) {
            // ---- W as it lies: the first blocks go out beside the kernel before this one -----------------------------------
            bool ok = true;
            int i = 0;
            for (; i < n_kb; i++) {
                const int s = i % WRING;
                if (i >= WRING && !__all_sync(0xffffffffu, mbar_wait(sempty + 8 * s, ((i / WRING) - 1) & 1, abort_flag))) { ok = false; break; }
                if (elect_one()) {
                    mbar_expect_tx(sfull + 8 * s, S_TILE_W);
                    for (int h = 0; h < 2; h++)
                        tma_load_2d(wring + s * S_TILE_W + h * (S_TILE_W / 2), &map_w, ((kb0 + i) * 2 + h) * 64, n0, sfull + 8 * s);
                }
            }
            if (!ok) {
                int ignored = 0;
                for (int j = i > WRING ? i - WRING : 0; j < i; j++) mbar_wait(sfull + 8 * (j % WRING), (j / WRING) & 1, &ignored);
            }
        } else if (warp == 13) {
            // ---- issue ---------------------------------------------------------------------------------------------
            constexpr uint32_t idesc = instr_desc(S_BM, ROWS);
            const uint32_t one = elect_one() ? 1 : 0;
            int s = 0;
            uint32_t turn = 0;                         // of the ring
            bool ok = true;
            for (int i = 0; i < n_kb && ok; i++) {
                const int b = i & 1;
                ok = (i < 2 || mbar_wait(accempty + 8 * b, ((i >> 1) - 1) & 1, abort_flag)) && mbar_wait(wfull + 8 * b, (i >> 1) & 1, abort_flag);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                const int has = need[b][0] | need[b][1] | need[b][2] | need[b][3];
                const uint32_t acc = tmem + b * ROWS, w_lo = desc_lo(wparts + b * S_PART_W);
                const uint32_t w2_lo = desc_lo(wparts + 2 * S_PART_W), w3_lo = desc_lo(wparts + 3 * S_PART_W);
                auto products = [&](uint32_t wl, uint32_t xl, auto first) {      // 16 values of k = 32 bytes along the swizzled row
                    mma_ss_lo<!decltype(first)::value>(acc, wl, xl, idesc, one);
#pragma unroll
                    for (int j = 1; j < S_BK / 16; j++) mma_ss_lo<true>(acc, wl + 2 * j, xl + 2 * j, idesc, one);
                };
#pragma unroll
                for (int p = 2; p >= 0; p--) {
                    if (!__all_sync(0xffffffffu, mbar_wait(xfull + 8 * s, turn, abort_flag))) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t x_lo = desc_lo(ring + s * PART_X);
                    if (p == 2) {
                        // (the smallest product begins the sum; x3 w3 is left out)
                        if (has & 2) {
                            products(w2_lo, x_lo, std::true_type());
                            products(w_lo, x_lo, std::false_type());
                        } else products(w_lo, x_lo, std::true_type());
                    } else {
                        if (has & 4) products(w3_lo, x_lo, std::false_type());
                        if (has & 2) products(w2_lo, x_lo, std::false_type());
                        products(w_lo, x_lo, std::false_type());
                    }
                    mma_commit_one(xempty + 8 * s, one);
                    if (p == 0) {
                        mma_commit_one(wempty + 8 * b, one);
                        mma_commit_one(accfull + 8 * b, one);
                    }
                    if (++s == RING) { s = 0; turn ^= 1; }
                }
            }
            if (!ok) *abort_flag = 1;
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 168;\n" ::);
        pdl_wait(KID_GEMM_TC);                         // (the flags of x's rows are read below)
        float sum[HALF];
#pragma unroll
        for (int c = 0; c < HALF; c++) sum[c] = 0.f;
        const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
        const int c0 = (warp >> 2) * HALF;
        bool ok = true;
        for (int i = 0; i < n_kb; i++) {
            const int b = i & 1;
            if (!__all_sync(0xffffffffu, mbar_wait(accfull + 8 * b, (i >> 1) & 1, abort_flag))) { ok = false; break; }
            tc_fence_after();
            const uint32_t acc = tmem + lanes + b * ROWS + c0;
#pragma unroll
            for (int c = 0; c < HALF; c += 16) {
                uint32_t v[16];
                tmem_ld16(acc + c, v);
                tmem_wait_ld();
#pragma unroll
                for (int e = 0; e < 16; e++) {
                    sum[c + e] += __uint_as_float(v[e]);
                    asm volatile("" : "+f"(sum[c + e]));      // (added here: put off, the values of all loads would be held)
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(accempty + 8 * b);
        }
        if (ok) {
            // every product has been taken: the parts' memory is free for the partial sums
#pragma unroll
            for (int c = 0; c < HALF; c++) part[(c0 + c) * S_BM + (warp & 3) * 32 + lane] = sum[c];
        }
    }
    __syncwarp();
    tc_fence_before();
    if (splits > 1) asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    else __syncthreads();
    // ---- this CTA's share of the tile: four columns of a row of y a thread and turn, all splits' values asked for at once ----
    constexpr int UNITS = S_BM / 4;
    // (a thread asks for 32 rows' flags, and all wait for what these got: a read whose value nobody uses could be under way when that CTA leaves)
    uint32_t flags = 0;
    if (threadIdx.x < splits * (S_BM / 32)) flags = s_ld_cluster_int(s_cluster_addr(smem_u32(odd_w + threadIdx.x % (S_BM / 32)), threadIdx.x / (S_BM / 32)));
    if (flags) atomicOr(odd_all + threadIdx.x % (S_BM / 32), flags);
    const bool flagged = __syncthreads_or(flags != 0);
    bool again = flagged;
    const int live = (M - m0 < ROWS ? M - m0 : ROWS) * UNITS;
    for (int u = rank * S_THREADS + threadIdx.x; u < live; u += splits * S_THREADS) {
        const int m = m0 + u / UNITS, n = n0 + (u % UNITS) * 4;
        if (n >= N) continue;                          // (nothing is read that is not added and stored)
        float4 v[MAX_SPLITS];
#pragma unroll
        for (int p = 0; p < MAX_SPLITS; p++)
            if (p < splits) v[p] = s_ld_cluster16(s_cluster_addr(wparts + u * 16, p));
        float4 s = v[0];
#pragma unroll
        for (int p = 1; p < MAX_SPLITS; p++)
            if (p < splits) { s.x += v[p].x; s.y += v[p].y; s.z += v[p].z; s.w += v[p].w; }
        *reinterpret_cast<float4*>(y + (size_t)m * N + n) = s;
        again |= odd_row[m] != 0 || !(finite(s.x) && finite(s.y) && finite(s.z) && finite(s.w));
    }
    __syncwarp();
    // A CTA's shared memory stays until its peers have read it.  Every sum that a thread read from a peer went into a store to y above, every flag
    // into the barrier that told the threads of them, and the fence keeps those ahead of the arrival (rows_gemm_tcgen05.cu says more)
    if (splits > 1) asm volatile("fence.acq_rel.cta;\nbarrier.cluster.arrive.relaxed.aligned;\n" ::: "memory");
    // Behind the arrival (the peers need nothing more): the entries that cannot be summed in parts.  A warp's units are a row of x each turn.
    if (flagged) {
        for (int r = warp; r < S_BM; r += S_THREADS / 32)
            if ((odd_all[r / 32] >> (r % 32) & 1) && !row_is_odd(w + (size_t)(n0 + r) * K, K, lane) && lane == 0) atomicAnd(odd_all + r / 32, ~(1u << (r % 32)));
        __syncthreads();
    }
    if (__any_sync(0xffffffffu, again))
#pragma unroll 1
        for (int u = rank * S_THREADS + threadIdx.x; u < live; u += splits * S_THREADS) {
            const int m = m0 + u / UNITS, n = n0 + lane * 4;
            uint32_t which = 0;
            if (n < N) {
                const float4 s = *reinterpret_cast<const float4*>(y + (size_t)m * N + n);
                which = odd_row[m] ? 0xfu : (odd_all[lane / 8] >> (lane % 8 * 4) & 0xfu) | !finite(s.x) | !finite(s.y) << 1 | !finite(s.z) << 2 | !finite(s.w) << 3;
            }
#pragma unroll 1
            for (int e = 0; e < 4; e++)
#pragma unroll 1
                for (uint32_t todo = __ballot_sync(0xffffffffu, which >> e & 1); todo; todo &= todo - 1) {
                    const int owner = __ffs(todo) - 1, at = n0 + owner * 4 + e;
                    const float v = plain_dot(x + (size_t)m * K, w + (size_t)at * K, K, lane);
                    if (lane == owner) y[(size_t)m * N + at] = v;
                }
        }
    __syncwarp();
    if (splits > 1) asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    else __syncthreads();
    if (warp == 13) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(TMEM_COLS));
    }
    if (threadIdx.x == 0 && *abort_flag) atomicOr(status, 64);
}

// ---- host side ----------------------------------------------------------------------------------

// Whether this kernel takes the product.
PLLM_EXPORT int pllm_gemm_f32_tcgen05_supports(int M, int N, int K) {
    return M >= 1 && N >= 4 && N % 4 == 0 && K >= 64 && K % 8 == 0 && K <= 1 << 24 && (M + 31) / 32 <= 65535 && (long long)M * K <= 1LL << 31;
}

namespace {

template <int ROWS, int RING, int WRING>
constexpr size_t split_smem() {
    constexpr size_t parts = S_W + WRING * S_TILE_W + (size_t)RING * ROWS * S_BK * 2, sums = (size_t)ROWS * S_BM * 4;
    return (parts > sums ? parts : sums) + 1024;
}

template <int ROWS, int RING, int WRING, int MAX_SPLITS>
bool allow_split() {
    return cudaFuncSetAttribute(gemm_f32_tcgen05_kernel<ROWS, RING, WRING, MAX_SPLITS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)split_smem<ROWS, RING, WRING>()) == cudaSuccess;
}

// Clusters of ``size`` CTAs that run at the same time on the current device (asked once each; a cluster sits in one GPC): 0 where it is not to be known.
template <int ROWS, int RING, int WRING>
int most_clusters(int size) {
    constexpr int KNOWN = 64;
    static std::atomic<int> known[KNOWN][9];     // 1 + the clusters; 0: not asked yet
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    if (dev < KNOWN && known[dev][size].load() > 0) return known[dev][size].load() - 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(sm_count() / size, size);
    cfg.blockDim = dim3(S_THREADS);
    cfg.dynamicSmemBytes = split_smem<ROWS, RING, WRING>();
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = attr[0].val.clusterDim.z = 1;
    attr[0].val.clusterDim.y = size;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (!allow_split<ROWS, RING, WRING, 8>() || cudaOccupancyMaxActiveClusters(&n, gemm_f32_tcgen05_kernel<ROWS, RING, WRING, 8>, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;                                // (asked again next time)
    }
    if (dev < KNOWN) known[dev][size].store(n + 1);
    return n;
}

template <int ROWS, int RING, int WRING, int MAX_SPLITS>
int launch_split(const CUtensorMap& map, const CUtensorMap& map_w, const float* x, const float* w, const int* odd_row, float* y, int M, int N, int K,
                 int splits, int* status, cudaStream_t stream) {
    allow_split<ROWS, RING, WRING, MAX_SPLITS>();
    launch_chained_cluster_y(gemm_f32_tcgen05_kernel<ROWS, RING, WRING, MAX_SPLITS>, dim3((N + S_BM - 1) / S_BM, splits, (M + ROWS - 1) / ROWS),
                             dim3(S_THREADS), split_smem<ROWS, RING, WRING>(), stream, splits, map, map_w, w, x, odd_row, y, M, N, K, status);
    return launch_status();
}

template <int ROWS, int RING, int WRING>
int pick_split(const void* parts, const float* x, const float* w, const int* odd_row, float* y, int M, int N, int K, int splits, int* status,
               cudaStream_t stream) {
    CUtensorMap map, map_w;
    const long long d[3] = {K, M, 3}, st[2] = {2LL * K, 2LL * K * M}, dw[2] = {2LL * K, N}, sw[1] = {4LL * K};
    const int box[3] = {S_BK, ROWS, 1}, bw[2] = {64, S_BM};
    if (tensor_map(parts, 3, d, st, box, true, &map) != 0 || tensor_map(w, 2, dw, sw, bw, true, &map_w) != 0) return PLLM_ERR_SIZE;
    const long long tiles = (long long)((N + S_BM - 1) / S_BM) * ((M + ROWS - 1) / ROWS);
    const int k_blocks = (K + S_BK - 1) / S_BK;
    if (splits <= 0) {
        // The most CTAs to a tile's K that still run all at once, two blocks of k or more each: a second turn of them costs as much as the first
        // (512 x 1024 x 3072 with tiles of 256 rows, 16 tiles: eight CTAs each 38.8 us, six 26.0, four 29.6)
        splits = 1;
        for (int c = 8; c > 1 && splits == 1; c = c > 4 ? c - 2 : c - 1)
            if (tiles * c <= sm_count() && k_blocks / c >= 2 && tiles <= most_clusters<ROWS, RING, WRING>(c)) splits = c;
    }
    if (splits > 8 || splits > k_blocks) return PLLM_ERR_SIZE;
    if (splits == 1) return launch_split<ROWS, RING, WRING, 1>(map, map_w, x, w, odd_row, y, M, N, K, splits, status, stream);
    return launch_split<ROWS, RING, WRING, 8>(map, map_w, x, w, odd_row, y, M, N, K, splits, status, stream);
}

}  // namespace

// x: [M, K]; w: [N, K]; y: [M, N], all float; parts: [3, M, K] bfloat16 and odd_row: [M] int, both written here.  tile: rows of x a tile
// (32, 64, 128 or 256; 0: as the sizes ask), splits: CTAs that share a tile's K (0: as the sizes ask).
PLLM_EXPORT int pllm_gemm_f32_tcgen05(const float* x, const float* w, float* y, void* parts, int* odd_row, int M, int N, int K, int tile, int splits,
                                      int* status, cudaStream_t stream) {
    if (!pllm_gemm_f32_tcgen05_supports(M, N, K)) return PLLM_ERR_SIZE;
    if (((uintptr_t)x | (uintptr_t)w | (uintptr_t)y | (uintptr_t)parts) & 15) return PLLM_ERR_ALIGN;
    if (tile == 0) tile = M <= 32 ? 32 : (M <= 64 ? 64 : (M <= 128 ? 128 : 256));
    if (tile != 32 && tile != 64 && tile != 128 && tile != 256) return PLLM_ERR_SIZE;
    launch_chained(split_rows_kernel, dim3(M), dim3(K >= 1024 ? 256 : 128), 0, stream, x, (bf16*)parts, odd_row, M, K);
    if (const int e = launch_status()) return e;
    if (tile == 32) return pick_split<32, 6, 3>(parts, x, w, odd_row, y, M, N, K, splits, status, stream);
    if (tile == 64) return pick_split<64, 6, 3>(parts, x, w, odd_row, y, M, N, K, splits, status, stream);
    if (tile == 128) return pick_split<128, 4, 3>(parts, x, w, odd_row, y, M, N, K, splits, status, stream);
    return pick_split<256, 3, 2>(parts, x, w, odd_row, y, M, N, K, splits, status, stream);
}

PLLM_TRACE_EXPORT(gemm_f32_tcgen05)
