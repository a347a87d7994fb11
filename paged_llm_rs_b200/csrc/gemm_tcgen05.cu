// y[M, N] = x[M, K] . W[N, K]^T in bfloat16 with float accumulation on the fifth-generation
// tensor cores, for the many rows of a prompt portion: tcgen05.mma issued by one thread,
// operands staged in shared memory by TMA (cp.async.bulk.tensor, 128-byte swizzle), the
// accumulator in tensor memory, read back with tcgen05.ld for the epilogue.
//
// The reference calls a library product for every projection
// (crates/pagedllm/src/model/layers.rs:27-35) and a pass of its own for the gated
// activation (crates/pagedllm/src/model/layers.rs:93-99).  This kernel is the product with
// that activation in its epilogue: with GLU the weight is [gate rows | up rows] and a CTA
// multiplies 64 rows of each, so that y = silu(gate) * up leaves the kernel and the
// [M, 2N] intermediate is never written.
//
// The kernel is persistent: one CTA to an SM, each taking tiles of 128 x BN (BN = 256, or 128
// or 64 where the width asks for it) in turn, m fastest, so that the CTAs at work share W tiles in
// L2.  Six warps:
//   warp 4     producer: waits for a free stage, arms its barrier with the bytes to come and
//              issues the TMA loads, a lane each in one instruction (a prompt of 400 tokens at the 0.6B shape 1575 us from one lane in turn, 1547 this way) (a 128 x 64 tile of x, a BN x 64 tile of W; GLU: BN/2 rows
//              of gate and of up)
//   warp 5     allocates tensor memory (two accumulators of BN columns); waits for
//              a full stage and issues four tcgen05.mma (K = 16 each), then tcgen05.commit,
//              which frees the stage when those have read it; after a tile's last, a commit
//              to that accumulator's barrier.  All its lanes go through the loop and one of them
//              executes these instructions (tcgen05.cuh, mma_ss_lo): issued by a thread of its own, the 0.6B
//              shape's 2048-token step took 3071 us and the 8B shape's 4421, this way 3028 to 3039 and 4315 to 4337
//   warps 0-3  epilogue: wait for an accumulator, tcgen05.ld their 32 lanes (= rows) 32
//              columns at a time, convert, (activation,) store, hand the accumulator back;
//              the tensor cores are on the next tile meanwhile
// Every wait is bounded: a thread that gives up raises a flag that the others see, the
// CTA frees its tensor memory and leaves, and the status word says so (bit 64).
#include <atomic>

#include "tcgen05.cuh"

using namespace tc;

namespace {

constexpr int G_BM = 128, G_BK = 64;
constexpr int G_TILE_A = G_BM * G_BK * 2;           // 16 KB
constexpr int G_SMEM_TILES = 192 * 1024;            // what the stages may fill
constexpr int G_THREADS = 192;

}  // namespace

// The gated activations other than silu (common.cuh), with the fast exponential and division as the silu above.
__device__ __forceinline__ float glu_act_fast(int kind, float limit, float g, float u) {
    if (kind == GLU_RELU) return fmaxf(g, 0.f) * u;
    g = fminf(g, limit);
    u = fminf(fmaxf(u, -limit), limit);
    return __fdividef(g, 1.0f + __expf(-1.702f * g)) * (u + 1.0f);
}

// A lane's row of an accumulator to its place in y (null: past the last row), 32 columns at a time; ``taken`` is called when the last of
// them are in registers.
template <bool GLU, int BN, typename F>
__device__ __forceinline__ void tile_out(uint32_t acc, bf16* dst, int act, float limit, F taken) {
    constexpr int OUT_BN = GLU ? BN / 2 : BN;
#pragma unroll 2
    for (int c = 0; c < OUT_BN / 32; c++) {
        uint32_t v[32], out[16];
        tmem_ld32(acc + c * 32, v);
        if (GLU) {
            uint32_t u[32];
            tmem_ld32(acc + BN / 2 + c * 32, u);
            tmem_wait_ld();
#pragma unroll
            for (int k = 0; k < 16; k++) {
                // gate and up rounded as a product of their own would leave them, then the activation
                const float g0 = round_bf16(__uint_as_float(v[2 * k])), g1 = round_bf16(__uint_as_float(v[2 * k + 1]));
                const float u0 = round_bf16(__uint_as_float(u[2 * k])), u1 = round_bf16(__uint_as_float(u[2 * k + 1]));
                // (fast exponential and division: their error is far below the rounding to bfloat16,
                //  and the epilogue must keep pace with the tensor cores)
                if (act == GLU_SILU) out[k] = pack2(__fdividef(g0, 1.0f + __expf(-g0)) * u0, __fdividef(g1, 1.0f + __expf(-g1)) * u1);
                else out[k] = pack2(glu_act_fast(act, limit, g0, u0), glu_act_fast(act, limit, g1, u1));
            }
        } else {
            tmem_wait_ld();
            if (act == UNARY_NONE) {
#pragma unroll
                for (int k = 0; k < 16; k++) out[k] = pack2(__uint_as_float(v[2 * k]), __uint_as_float(v[2 * k + 1]));
            } else {
                // a one-argument activation of the product, rounded first as a product of its own would leave it
#pragma unroll
                for (int k = 0; k < 16; k++)
                    out[k] = pack2(unary_act(act, round_bf16(__uint_as_float(v[2 * k]))),
                                   unary_act(act, round_bf16(__uint_as_float(v[2 * k + 1]))));
            }
        }
        if (c == OUT_BN / 32 - 1) taken();
        if (dst) {
#pragma unroll
            for (int k = 0; k < 4; k++)
                *reinterpret_cast<uint4*>(dst + c * 32 + k * 8) = make_uint4(out[4 * k], out[4 * k + 1], out[4 * k + 2], out[4 * k + 3]);
        }
    }
}

// map_a: x [M, K], box 64 x 128.  map_b: W [rows, K], box 64 x BN (plain) or 64 x BN/2 (GLU).
// y: [M, n_out] bfloat16; n_out = N (plain) or N / 2 (GLU, W = [gate; up] of n_out rows each).
template <int EPI, int BN>
__global__ void __launch_bounds__(G_THREADS, 1) gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap map_a,
                                                                    const __grid_constant__ CUtensorMap map_b,
                                                                    bf16* __restrict__ y, int M, int n_out, int K,
                                                                    int* status, const int* tile_expert, int expert_rows,
                                                                    int act, float limit) {
    // Grouped form (tile_expert given): the rows of x are sorted by expert, every expert's rows padded to whole
    // tiles of 128; tile_expert[m tile] names the expert whose weights that tile multiplies (its rows of W start at
    // expert * expert_rows), or is negative for a tile past the last one in use, which every role skips alike.
    // The list is written by the kernel before this one: read after the wait for it, by plain loads.
    constexpr bool GLU = EPI == 1;
    constexpr int TILE_B = BN * G_BK * 2, STAGE = G_TILE_A + TILE_B;
    constexpr int STAGES = G_SMEM_TILES / STAGE;
    constexpr int OUT_BN = GLU ? BN / 2 : BN;            // columns of y a tile makes
    constexpr uint32_t TMEM_COLS = 2 * BN;               // two accumulators
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    // the tiles need 1024-byte alignment for the 128-byte swizzle
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t tiles = smem_u32(smem);
    unsigned char* ctl = smem + STAGES * STAGE;
    const uint32_t bars = smem_u32(ctl);                 // full[S], empty[S], acc_full[2], acc_empty[2]
    const uint32_t acc_full = bars + 8 * 2 * STAGES, acc_empty = acc_full + 16;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(ctl + 8 * (2 * STAGES + 4));
    volatile int* abort_flag = reinterpret_cast<volatile int*>(ctl + 8 * (2 * STAGES + 4) + 8);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tiles_m = (M + G_BM - 1) / G_BM, tiles_n = n_out / OUT_BN;
    const int n_tiles = tiles_m * tiles_n;
    const int k_blocks = (K + G_BK - 1) / G_BK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; s++) {
            mbar_init(bars + 8 * s, 1);
            mbar_init(bars + 8 * (STAGES + s), 1);
        }
        for (int b = 0; b < 2; b++) {
            mbar_init(acc_full + 8 * b, 1);
            mbar_init(acc_empty + 8 * b, 4);     // one arrival from each epilogue warp
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::);
        asm volatile("fence.proxy.async.shared::cta;\n" ::);
    }
    if (warp == 5) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_slot)), "r"(TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 4) {
        // ---- producer: a stage's requests go out by as many lanes in one instruction ---------------------
        pdl_wait(KID_GEMM_TC, lane == 0);     // x comes from the kernel before this one
        int s = 0;
        uint32_t turn = 1;                    // (the first turn of the ring finds its stages free)
        bool ok = true;
        for (int t = blockIdx.x; t < n_tiles && ok; t += gridDim.x) {
            const int m0 = (t % tiles_m) * G_BM, n0 = (t / tiles_m) * OUT_BN;
            int w_row0 = 0;
            if (tile_expert) {
                const int e = tile_expert[t % tiles_m];
                if (e < 0) continue;
                w_row0 = e * expert_rows;
            }
            // lane 0: rows of x; lane 1: W's (gate) rows; lane 2: the up rows
            const CUtensorMap* map = lane == 0 ? &map_a : &map_b;
            const int row = lane == 0 ? m0 : w_row0 + n0 + (lane == 2 ? n_out : 0);
            const uint32_t to = tiles + (lane == 0 ? 0 : G_TILE_A + (lane == 2 ? TILE_B / 2 : 0));
            for (int kb = 0; kb < k_blocks; kb++) {
                if (!__all_sync(0xffffffffu, mbar_wait(bars + 8 * (STAGES + s), turn, abort_flag))) { ok = false; break; }
                if (lane == 0) mbar_expect_tx(bars + 8 * s, STAGE);
                __syncwarp();
                if (lane < (GLU ? 3 : 2)) tma_load_2d(to + s * STAGE, map, kb * G_BK, row, bars + 8 * s);
                if (++s == STAGES) { s = 0; turn ^= 1; }
            }
        }
    } else if (warp == 5) {
        // ---- tensor-core issue ------------------------------------------------------------------
        constexpr uint32_t idesc = instr_desc(G_BM, BN);
        const uint32_t one = elect_one() ? 1 : 0;
        int i = 0, s = 0;
        uint32_t turn = 0;
        bool ok = true;
        if (tile_expert) asm volatile("griddepcontrol.wait;\n" ::: "memory");
        for (int t = blockIdx.x; t < n_tiles && ok; t += gridDim.x) {
            if (tile_expert && tile_expert[t % tiles_m] < 0) continue;
            const int b = i & 1;
            // the epilogue must have read this accumulator's last tile out
            if (i >= 2 && !__all_sync(0xffffffffu, mbar_wait(acc_empty + 8 * b, ((i >> 1) - 1) & 1, abort_flag))) { ok = false; break; }
            tc_fence_after();
            for (int kb = 0; kb < k_blocks; kb++) {
                if (!__all_sync(0xffffffffu, mbar_wait(bars + 8 * s, turn, abort_flag))) { ok = false; break; }
                tc_fence_after();
                const uint32_t a_lo = desc_lo(tiles + s * STAGE), b_lo = desc_lo(tiles + s * STAGE + G_TILE_A), d = tmem + b * BN;
                if (kb == 0) mma_ss_lo<false>(d, a_lo, b_lo, idesc, one);
                else mma_ss_lo<true>(d, a_lo, b_lo, idesc, one);
#pragma unroll
                for (int j = 1; j < G_BK / 16; j++) mma_ss_lo<true>(d, a_lo + 2 * j, b_lo + 2 * j, idesc, one);   // 16 values of k = 32 bytes along the swizzled row
                mma_commit_one(bars + 8 * (STAGES + s), one);      // the stage is free once these have read it
                if (++s == STAGES) { s = 0; turn ^= 1; }
            }
            if (ok) mma_commit_one(acc_full + 8 * b, one);         // this tile's accumulator is complete
            i++;
        }
    } else {
        // ---- epilogue: warp w owns lanes (rows) 32 w .. 32 w + 31 of the accumulators ---------------
        pdl_launch_dependents();
        int i = 0;
        if (tile_expert) asm volatile("griddepcontrol.wait;\n" ::: "memory");
        for (int t = blockIdx.x; t < n_tiles; t += gridDim.x) {
            if (tile_expert && tile_expert[t % tiles_m] < 0) continue;
            const int b = i & 1;
            const int m0 = (t % tiles_m) * G_BM, n0 = (t / tiles_m) * OUT_BN;
            if (!mbar_wait(acc_full + 8 * b, (i >> 1) & 1, abort_flag)) break;
            tc_fence_after();
            const int row = m0 + warp * 32 + lane;
            const uint32_t acc = tmem + ((uint32_t)(warp * 32) << 16) + b * BN;
            tile_out<GLU, BN>(acc, row < M ? y + (size_t)row * n_out + n0 : nullptr, act, limit, [&]() {
                // everything of this accumulator is in registers: the tensor cores may have it back
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(acc_empty + 8 * b);
            });
            i++;
        }
    }
    // ---- everyone meets; the allocating warp gives the tensor memory back ---------------------------
    tc_fence_before();
    __syncthreads();
    if (warp == 5) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(TMEM_COLS));
    }
    if (threadIdx.x == 0 && *abort_flag) atomicOr(status, 64);
}

// ---- the same with two CTAs to a tile of 256 x 256 -------------------------------------------------
// One CTA's product of 128 x 256 reads 12 KB of operands from shared memory for what the tensor cores do in the time of 8; a pair's
// reads half of W's tile each.  The roles are those above; the loads of both CTAs are counted by the leader's barriers, the
// leader's sixth warp issues for both, and its commits free the stages and hand over the accumulators in both.  Measured in captured
// steps with the gated product on pairs (us a step, one CTA a tile / pairs; the results are equal bit for bit): 0.6B shape, 2048 rows
// 3142 / 3118; 8B shape, 6 layers, 2048 rows 4548 / 4454, 512 rows 1897 / 1856.  The plain products stay with the library: on pairs
// the 0.6B step of 2048 rows takes 3149 with q/k/v, 3248 with o, 3271 with down (3067 to 3130 with none), the 8B one 4380, 4540 and
// 4555 (4386 to 4472).  Weights asked for ahead of the wait changed nothing here.
constexpr int P_STAGE = 2 * G_TILE_A;               // 128 rows of x and 128 of W, 32 KB
constexpr int P_STAGES = G_SMEM_TILES / P_STAGE;

template <int EPI>
__global__ void __launch_bounds__(G_THREADS, 1) gemm_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                                                                 bf16* __restrict__ y, int M, int n_out, int K, int* status, int act, float limit) {
    constexpr bool GLU = EPI == 1;
    constexpr int BN = 256, OUT_BN = GLU ? BN / 2 : BN;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t tiles = smem_u32(smem);
    unsigned char* ctl = smem + P_STAGES * P_STAGE;
    const uint32_t bars = smem_u32(ctl);                 // full[S] (the leader's), empty[S], acc_full[2], acc_empty[2] (the leader's)
    const uint32_t acc_full = bars + 8 * 2 * P_STAGES, acc_empty = acc_full + 16;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(ctl + 8 * (2 * P_STAGES + 4));
    volatile int* abort_flag = reinterpret_cast<volatile int*>(ctl + 8 * (2 * P_STAGES + 4) + 8);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = (int)cluster_rank(), pairs = gridDim.x / 2, pair = blockIdx.x / 2;
    const int tiles_m = (M + 2 * G_BM - 1) / (2 * G_BM), tiles_n = n_out / OUT_BN, n_tiles = tiles_m * tiles_n;
    const int k_blocks = (K + G_BK - 1) / G_BK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < P_STAGES; s++) {
            mbar_init(bars + 8 * s, 1);
            mbar_init(bars + 8 * (P_STAGES + s), 1);
        }
        for (int b = 0; b < 2; b++) {
            mbar_init(acc_full + 8 * b, 1);
            mbar_init(acc_empty + 8 * b, 8);     // one arrival from each epilogue warp of both CTAs
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::);
        fence_async_smem();
    }
    if (warp == 5) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_slot)), "r"(2 * BN));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::);
    }
    tc_fence_before();
    __syncthreads();
    pair_sync();                                 // both CTAs' barriers are ready
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 4) {
        pdl_wait(KID_GEMM_TC, lane == 0);        // x comes from the kernel before this one
        int s = 0;
        uint32_t turn = 1;
        bool ok = true;
        for (int t = pair; t < n_tiles && ok; t += pairs) {
            const int m0 = (t % tiles_m) * 2 * G_BM + rank * G_BM, n0 = (t / tiles_m) * OUT_BN;
            const int w_row = GLU ? rank * n_out + n0 : n0 + rank * (BN / 2);      // (the leader's half: gate rows; its peer's: up rows)
            const CUtensorMap* map = lane == 0 ? &map_a : &map_b;
            const int row = lane == 0 ? m0 : w_row;
            for (int kb = 0; kb < k_blocks; kb++) {
                if (!__all_sync(0xffffffffu, mbar_wait(bars + 8 * (P_STAGES + s), turn, abort_flag))) { ok = false; break; }
                if (rank == 0 && lane == 0) mbar_expect_tx(bars + 8 * s, 2 * P_STAGE);
                __syncwarp();
                if (lane < 2) tma_load_2d_pair(tiles + s * P_STAGE + lane * G_TILE_A, map, kb * G_BK, row, leader_addr(bars + 8 * s));
                if (++s == P_STAGES) { s = 0; turn ^= 1; }
            }
        }
    } else if (warp == 5) {
        if (rank == 0) {
            constexpr uint32_t idesc = instr_desc(2 * G_BM, BN);
            const uint32_t one = elect_one() ? 1 : 0;
            int i = 0, s = 0;
            uint32_t turn = 0;
            bool ok = true;
            for (int t = pair; t < n_tiles && ok; t += pairs) {
                const int b = i & 1;
                if (i >= 2 && !__all_sync(0xffffffffu, mbar_wait(acc_empty + 8 * b, ((i >> 1) - 1) & 1, abort_flag))) { ok = false; break; }
                tc_fence_after();
                for (int kb = 0; kb < k_blocks; kb++) {
                    if (!__all_sync(0xffffffffu, mbar_wait(bars + 8 * s, turn, abort_flag))) { ok = false; break; }
                    tc_fence_after();
                    const uint64_t a_desc = smem_desc(tiles + s * P_STAGE), b_desc = smem_desc(tiles + s * P_STAGE + G_TILE_A);
#pragma unroll
                    for (int j = 0; j < G_BK / 16; j++) mma_ss_pair(tmem + b * BN, a_desc + 2 * j, b_desc + 2 * j, idesc, (kb | j) ? 1u : 0u, one);
                    mma_commit_pair(bars + 8 * (P_STAGES + s), one);
                    if (++s == P_STAGES) { s = 0; turn ^= 1; }
                }
                if (ok) mma_commit_pair(acc_full + 8 * b, one);
                i++;
            }
        }
    } else {
        pdl_launch_dependents();
        int i = 0;
        for (int t = pair; t < n_tiles; t += pairs) {
            const int b = i & 1;
            const int m0 = (t % tiles_m) * 2 * G_BM + rank * G_BM, n0 = (t / tiles_m) * OUT_BN;
            if (!mbar_wait(acc_full + 8 * b, (i >> 1) & 1, abort_flag)) break;
            tc_fence_after();
            const int row = m0 + warp * 32 + lane;
            const uint32_t acc = tmem + ((uint32_t)(warp * 32) << 16) + b * BN;
            tile_out<GLU, BN>(acc, row < M ? y + (size_t)row * n_out + n0 : nullptr, act, limit, [&]() {
                // everything of this accumulator is in registers: the tensor cores may have it back
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(leader_addr(acc_empty + 8 * b));
            });
            i++;
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    pair_sync();                                 // neither CTA leaves while the other may still signal it, or use its memory
    if (warp == 5) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(2 * BN));
    }
    if (threadIdx.x == 0 && *abort_flag) atomicOr(status, 64);
}

// ---- host side ----------------------------------------------------------------------------------

// Whether this kernel takes the product (n_out: columns of y).
PLLM_EXPORT int pllm_gemm_tcgen05_supports(int M, int n_out, int K, int glu) {
    return M >= 1 && K >= 64 && K % 8 == 0 && n_out >= 64 && n_out % (glu ? 64 : 128) == 0;
}

namespace {


template <int EPI, int BN>
int launch_gemm(const void* x, const void* w, void* y, int M, int n_out, int K, int* status,
                cudaStream_t stream, const int* tile_expert = nullptr, int n_experts = 1, int act = GLU_SILU, float limit = 0.f) {
    constexpr bool GLU = EPI == 1;
    constexpr int OUT_BN = GLU ? BN / 2 : BN;
    constexpr int STAGE = G_TILE_A + BN * G_BK * 2, STAGES = G_SMEM_TILES / STAGE;
    CUtensorMap map_a, map_b;
    {
        const long long da[2] = {K, M}, db[2] = {K, (long long)n_experts * (GLU ? 2LL * n_out : n_out)}, st[1] = {2LL * K};
        const int ba[2] = {G_BK, G_BM}, bb[2] = {G_BK, OUT_BN};
        if (tensor_map(x, 2, da, st, ba, true, &map_a) != 0) return PLLM_ERR_SIZE;
        if (tensor_map(w, 2, db, st, bb, true, &map_b) != 0) return PLLM_ERR_SIZE;
    }
    const int g_sm_count = sm_count();
    const size_t smem = (size_t)STAGES * STAGE + 8 * (2 * STAGES + 4) + 16 + 1024;
    const int n_tiles = ((M + G_BM - 1) / G_BM) * (n_out / OUT_BN);
    const dim3 grid(n_tiles < g_sm_count ? n_tiles : g_sm_count);
    cudaFuncSetAttribute(gemm_tcgen05_kernel<EPI, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    launch_chained(gemm_tcgen05_kernel<EPI, BN>, grid, dim3(G_THREADS), smem, stream, map_a, map_b, (bf16*)y, M, n_out, K, status,
                   tile_expert, GLU ? 2 * n_out : n_out, act, limit);
    return launch_status();
}

constexpr size_t P_SMEM = (size_t)P_STAGES * P_STAGE + 8 * (2 * P_STAGES + 4) + 16 + 1024;

// The kernel's shared memory is allowed a device at a time, as every launcher here does it at each launch.
template <int EPI>
bool allow_pair() {
    return cudaFuncSetAttribute(gemm_pair_kernel<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)P_SMEM) == cudaSuccess;
}

// Pairs that run at the same time on the current device (asked once each): a pair sits in one GPC, so that it may be fewer than half of
// the SMs, and the tiles are dealt to those that do.  0: none, or not to be known, and the products are the one-CTA kernel's.
template <int EPI>
int most_pairs() {
    constexpr int KNOWN = 64;
    static std::atomic<int> known[KNOWN];        // 1 + the pairs of each device; 0: not asked yet
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    if (dev < KNOWN && known[dev].load() > 0) return known[dev].load() - 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * (sm_count() / 2));
    cfg.blockDim = dim3(G_THREADS);
    cfg.dynamicSmemBytes = P_SMEM;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (!allow_pair<EPI>() || cudaOccupancyMaxActiveClusters(&n, gemm_pair_kernel<EPI>, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;                                // (asked again next time)
    }
    n = n < sm_count() / 2 ? n : sm_count() / 2;
    if (dev < KNOWN) known[dev].store(n + 1);
    return n;
}

template <int EPI>
int launch_pair(const void* x, const void* w, void* y, int M, int n_out, int K, int* status, cudaStream_t stream, int act, float limit, int pairs) {
    constexpr bool GLU = EPI == 1;
    CUtensorMap map_a, map_b;
    {
        const long long da[2] = {K, M}, db[2] = {K, GLU ? 2LL * n_out : n_out}, st[1] = {2LL * K};
        const int box[2] = {G_BK, G_BM};
        if (tensor_map(x, 2, da, st, box, true, &map_a) != 0) return PLLM_ERR_SIZE;
        if (tensor_map(w, 2, db, st, box, true, &map_b) != 0) return PLLM_ERR_SIZE;
    }
    const int n_tiles = ((M + 2 * G_BM - 1) / (2 * G_BM)) * (n_out / (GLU ? 128 : 256));
    allow_pair<EPI>();
    launch_chained_cluster(gemm_pair_kernel<EPI>, dim3(2 * (n_tiles < pairs ? n_tiles : pairs)), dim3(G_THREADS), P_SMEM, stream, dim3(2, 1, 1), map_a,
                           map_b, (bf16*)y, M, n_out, K, status, act, limit);
    return launch_status();
}

}  // namespace

// x: [M, K]; w: [n_out, K], or with glu [2 n_out, K] = gate rows then up rows; y: [M, n_out]; all bfloat16.
// glu: 0 a plain product; positive: 1 + the gated activation's kind (common.cuh), with its limit; negative: minus a one-argument
// activation's kind (UNARY_*), applied to the plain product.
PLLM_EXPORT int pllm_gemm_tcgen05(const void* x, const void* w, void* y, int M, int n_out, int K, int glu, float limit, int* status,
                                  cudaStream_t stream) {
    const int unary = glu < 0 ? -glu : UNARY_NONE;
    if (glu < 0) glu = 0;
    if (!pllm_gemm_tcgen05_supports(M, n_out, K, glu) || unary > UNARY_RELU2 || glu > 1 + GLU_CLAMPED) return PLLM_ERR_SIZE;
    const int act = glu ? glu - 1 : unary;
    if (((uintptr_t)x | (uintptr_t)w | (uintptr_t)y) & 15) return PLLM_ERR_ALIGN;
    // tiles of 256 columns of W where the width divides into them and they still give every SM one
    const int tiles_m = (M + G_BM - 1) / G_BM;
    const int unit = glu ? 128 : 256;
    const bool wide = n_out % unit == 0 && (long long)tiles_m * (n_out / unit) >= sm_count();
    // pairs of CTAs where the tiles of 256 rows are not mostly padding and the device has room for a pair
    const int pairs = wide && (tiles_m % 2 == 0 || tiles_m >= 7) ? (glu ? most_pairs<1>() : most_pairs<0>()) : 0;
    if (pairs > 0)
        return glu ? launch_pair<1>(x, w, y, M, n_out, K, status, stream, act, limit, pairs)
                   : launch_pair<0>(x, w, y, M, n_out, K, status, stream, act, limit, pairs);
    // gated tiles of 32 columns where those of 64 leave more than half of the SMs idle (128 rows, 3072 x 1024: 10.4 -> 9.1 us; 250 rows, whose 192
    // tiles are two turns, a step of 1354 us -> 1418)
    if (glu && !wide && (long long)tiles_m * (n_out / 32) <= sm_count())
        return launch_gemm<1, 64>(x, w, y, M, n_out, K, status, stream, nullptr, 1, act, limit);
    if (glu)
        return wide ? launch_gemm<1, 256>(x, w, y, M, n_out, K, status, stream, nullptr, 1, act, limit)
                    : launch_gemm<1, 128>(x, w, y, M, n_out, K, status, stream, nullptr, 1, act, limit);
    return wide ? launch_gemm<0, 256>(x, w, y, M, n_out, K, status, stream, nullptr, 1, act)
                : launch_gemm<0, 128>(x, w, y, M, n_out, K, status, stream, nullptr, 1, act);
}

// The grouped form: x [M, K] holds the rows sorted by expert, each expert's rows padded to whole tiles of 128
// (M a multiple of 128, an upper bound); w [experts, n_out (glu: 2 n_out), K]; tile_expert [M / 128] on the device.
PLLM_EXPORT int pllm_gemm_tcgen05_grouped(const void* x, const void* w, void* y, int M, int n_out, int K, int glu, float limit,
                                          const int* tile_expert, int n_experts, int* status, cudaStream_t stream) {
    const int unary = glu < 0 ? -glu : UNARY_NONE;
    if (glu < 0) glu = 0;
    if (!pllm_gemm_tcgen05_supports(M, n_out, K, glu) || M % G_BM || n_experts < 1 || !tile_expert) return PLLM_ERR_SIZE;
    if (unary > UNARY_RELU2 || glu > 1 + GLU_CLAMPED) return PLLM_ERR_SIZE;
    const int act = glu ? glu - 1 : unary;
    if (((uintptr_t)x | (uintptr_t)w | (uintptr_t)y) & 15) return PLLM_ERR_ALIGN;
    const int tiles_m = M / G_BM;
    const int unit = glu ? 128 : 256;
    const bool wide = n_out % unit == 0 && (long long)tiles_m * (n_out / unit) >= sm_count();
    if (glu)
        return wide ? launch_gemm<1, 256>(x, w, y, M, n_out, K, status, stream, tile_expert, n_experts, act, limit)
                    : launch_gemm<1, 128>(x, w, y, M, n_out, K, status, stream, tile_expert, n_experts, act, limit);
    return wide ? launch_gemm<0, 256>(x, w, y, M, n_out, K, status, stream, tile_expert, n_experts, act)
                : launch_gemm<0, 128>(x, w, y, M, n_out, K, status, stream, tile_expert, n_experts, act);
}

PLLM_TRACE_EXPORT(gemm_tcgen05)
