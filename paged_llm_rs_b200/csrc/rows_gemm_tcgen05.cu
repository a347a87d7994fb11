// y[M, N] = x[M, K] . W[N, K]^T in bfloat16 with float accumulation for the rows of a decode step or of a short
// prompt (M <= 64), on the fifth-generation tensor cores with the WEIGHTS as the 128-row operand: a tile is 128
// rows of W against all rows of x, so that nothing is multiplied for padding but the last 16 rows' remainder.
// The reference calls a library product here (crates/pagedllm/src/model/layers.rs:27-35).
//
// What bounds it: the bytes of W (each read once; x is small and comes from L2), and for a small model's products
// (2 to 13 MB, 0.3 to 2 us at the copy bandwidth) the chain of one kernel after the other.  Hence
//   - W streams through a ring of TMA requests of 128 rows x 128 values of k (32 KB, 128-byte swizzle), and the ring's
//     first round goes out BEFORE the wait for the kernel before this one: for a small model that is all of the CTA's
//     weights, for a large one up to 28 MB of the next product's while the step is in its attention or its norms;
//   - K is split over the CTAs of a thread-block cluster where the tiles alone would leave SMs idle: each makes its
//     partial sums in tensor memory, puts them into its shared memory, and after one cluster barrier every CTA adds
//     a share of the tile over its peers' shared memory, in the order of k;
//   - two CTAs fit an SM, so that a tile's reduction, or the next kernel's weights, run beside another tile's loads.
// With GLU, W is [gate rows | up rows]: a CTA takes 64 rows of each, and act(gate, up) leaves the reduction.
//
// Measured on a B200 in captured decode steps at context 512 (us; before: skinny_gemm.cu up to 16 rows, the library's
// products, the activation's own pass and gemm_tcgen05.cu above): 6 layers of the 8B shape with the head, 8 / 16 / 32 / 64
// requests: 804 / 869 / 920 / 1045 -> 713 / 753 / 856 / 983; the 0.6B shape, 24 / 32 / 64 requests: 1561 / 1586 / 1747 -> 1285 / 1314 / 1713.
// Alone and back to back: the 8B shape's head (1.24 GB) at 8 rows 189 us (6.6 TB/s), its gate/up 35.0 (5.7), the library's
// head 213.  Where a product of 4 MB takes its 4 us (clocks of a CTA
// from the wait's end, 37 rows, eight CTAs a cluster): 1240 until x is there, 16 products until 2680, in shared memory at 3350, met at 4000, the
// peers' 17 KB read by 6530 (shared memory of another SM comes at some 12 bytes a clock), stored at 6770, gone at 7200.  With the warp's one lane
// issuing by predicate (tcgen05.cuh, mma_ss_lo) and not in a branch the 16 products take 1440 and not 1700: a prompt of 37 tokens 1102 -> 1075 us, 64
// requests 1720 -> 1687.  Asked for by each CTA from its own memory on, in turn: 0.7 % less, but a row's order of
// sums would follow its place in the step.  Sent to the CTA that adds them (st.async) instead of read by it: 1112 and 1730, the stores take as long as the reads.
//
// Ten warps: 0-7 take the accumulator out of tensor memory (a lane a row of W) and, with 8 and 9, add and store;
// warp 8 issues the loads, warp 9 owns the tensor memory and issues the tcgen05.mma.  Every wait is bounded: a thread
// that gives up raises a flag that the others see, all reach the cluster barriers, and the status word says so (64).
#include "tcgen05.cuh"

using namespace tc;

namespace {

constexpr int R_BM = 128, R_BK = 64;               // rows of W and values of k a tile (128 bytes a swizzled row)
constexpr int R_SK = 2 * R_BK;                     // values of k a stage: two tiles by one request
constexpr int R_TILE_W = R_BM * R_BK * 2;          // 16 KB
constexpr int R_THREADS = 320;                     // ten warps: 0-7 add and store too
constexpr int R_MAX_STAGES = 3;
constexpr int R_RING = 108 * 1024;                 // what a CTA's ring may fill (two CTAs an SM)
constexpr int R_MAX_ROWS = 64;

__device__ __forceinline__ void tmem_ld16(uint32_t addr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(addr));
}
__device__ __forceinline__ uint32_t cluster_addr(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ float4 ld_cluster16(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];\n" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory"); }

// four values of a row of y
__device__ __forceinline__ void store4(bf16* dst, float4 v) { *reinterpret_cast<uint2*>(dst) = make_uint2(pack2(v.x, v.y), pack2(v.z, v.w)); }
__device__ __forceinline__ void store4(float* dst, float4 v) { *reinterpret_cast<float4*>(dst) = v; }

}  // namespace

// map_w: W as [K / 64][N][64], box 2 x 128 x 64 (GLU: [K / 64][gate, up][n_out][64], box 2 x 2 x 64 x 64), so that a stage's two
// tiles land one behind the other by one request.  map_x: x as [K / 64][M][64], box 2 x rows x 64 (rows: M rounded up to 16;
// what lies past M or K arrives as zeros).  n_out: columns of y (GLU: W has 2 n_out rows).  Grid (tiles, splits), clusters of the splits.
template <bool GLU, int MAX_SPLITS, typename OutT>
__global__ void __launch_bounds__(R_THREADS, 2) rows_gemm_kernel(const __grid_constant__ CUtensorMap map_w,
                                                                 const __grid_constant__ CUtensorMap map_x, OutT* __restrict__ y,
                                                                 int M, int n_out, int K, int rows, int stages, uint32_t tmem_cols,
                                                                 int act, float limit, int* status) {
    constexpr int OUT_ROWS = GLU ? R_BM / 2 : R_BM;       // columns of y a tile makes
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    // (the tiles need 1024-byte alignment for the 128-byte swizzle; the offset is the same in every CTA of a cluster)
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const int tile_x = rows * R_BK * 2, stage = 2 * (R_TILE_W + tile_x);
    const uint32_t ring = smem_u32(smem);
    __shared__ __align__(8) unsigned long long bar_mem[2 * R_MAX_STAGES + 1];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_mem;
    volatile int* abort_flag = &abort_mem;
    const uint32_t full = smem_u32(bar_mem), empty = full + 8 * R_MAX_STAGES, done = full + 16 * R_MAX_STAGES;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int splits = gridDim.y, rank = blockIdx.y;
    // the splits take whole stages; the last stage of K may hold one tile only (what lies past K arrives as zeros)
    const int k_stages = (K + R_SK - 1) / R_SK;
    const int kb0 = k_stages * rank / splits, n_kb = k_stages * (rank + 1) / splits - kb0;
    const int row0 = blockIdx.x * OUT_ROWS;

    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; s++) {
            mbar_init(full + 8 * s, 1);
            mbar_init(empty + 8 * s, 1);
        }
        mbar_init(done, 1);
        abort_mem = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::);
        fence_async_smem();
    }
    if (warp == 9) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_slot)), "r"(tmem_cols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    // The next kernel's CTAs may take their places.  Only now that the tensor memory is this CTA's: a kernel that comes
    // early and takes it first would keep it until this one is over.
    pdl_launch_dependents();

    if (warp == 8) {
        const int first = n_kb < stages ? n_kb : stages;
        auto load_w = [&](int i, int s) {
            const uint32_t dst = ring + s * stage;
            mbar_expect_tx(full + 8 * s, stage);
            if (GLU) tma_load_4d(dst, &map_w, 0, row0, 0, (kb0 + i) * 2, full + 8 * s);
            else tma_load_3d(dst, &map_w, 0, row0, (kb0 + i) * 2, full + 8 * s);
        };
        auto load_x = [&](int i, int s) { tma_load_3d(ring + s * stage + 2 * R_TILE_W, &map_x, 0, 0, (kb0 + i) * 2, full + 8 * s); };
        for (int i = 0; i < first; i++)                     // the weights do not depend on the kernel before
            if (elect_one()) load_w(i, i);
        pdl_wait(KID_GEMM_TC, lane == 0);
        for (int i = 0; i < first; i++)
            if (elect_one()) load_x(i, i);
        int i = first;
        for (; i < n_kb; i++) {
            const int s = i % stages;
            if (!__all_sync(0xffffffffu, mbar_wait(empty + 8 * s, ((i / stages) - 1) & 1, abort_flag))) break;
            if (elect_one()) { load_w(i, s); load_x(i, s); }
        }
        if (i < n_kb) {
            // nothing may still be on its way into this CTA's memory when it leaves
            int ignored = 0;
            for (int j = i > stages ? i - stages : 0; j < i; j++) mbar_wait(full + 8 * (j % stages), (j / stages) & 1, &ignored);
        }
    } else if (warp == 9) {
        const uint32_t idesc = instr_desc(R_BM, rows), one = elect_one() ? 1 : 0;
        bool ok = true;
        int s = 0;
        uint32_t turn = 0;
        for (int i = 0; i < n_kb; i++) {
            if (!__all_sync(0xffffffffu, mbar_wait(full + 8 * s, turn, abort_flag))) { ok = false; break; }
            tc_fence_after();
            const uint32_t w_lo = desc_lo(ring + s * stage), x_lo = desc_lo(ring + s * stage + 2 * R_TILE_W), half = tile_x >> 4;
            if (i == 0) mma_ss_lo<false>(tmem, w_lo, x_lo, idesc, one);
            else mma_ss_lo<true>(tmem, w_lo, x_lo, idesc, one);
#pragma unroll
            for (int j = 1; j < R_BK / 16; j++) mma_ss_lo<true>(tmem, w_lo + 2 * j, x_lo + 2 * j, idesc, one);     // 16 values of k = 32 bytes along the swizzled row
#pragma unroll
            for (int j = 0; j < R_BK / 16; j++) mma_ss_lo<true>(tmem, w_lo + (R_TILE_W >> 4) + 2 * j, x_lo + half + 2 * j, idesc, one);
            mma_commit_one(i + 1 < n_kb ? empty + 8 * s : done, one);
            if (++s == stages) { s = 0; turn ^= 1; }
        }
        if (!ok) *abort_flag = 1;
    } else if (mbar_wait(done, 0, abort_flag)) {
        // every product has been taken: the ring's memory is free for the partial sums, part[row of x][row of W]
        // (warps w and w + 4 may read the same lanes of tensor memory: every other 16 rows of x each)
        tc_fence_after();
        float* part = reinterpret_cast<float*>(smem) + (warp & 3) * 32 + lane;
        const uint32_t acc = tmem + ((uint32_t)((warp & 3) * 32) << 16);
        for (int c = (warp >> 2) * 16; c < rows; c += 32) {
            uint32_t v[16];
            tmem_ld16(acc + c, v);
            tmem_wait_ld();
#pragma unroll
            for (int q = 0; q < 16; q++) part[(c + q) * R_BM] = __uint_as_float(v[q]);
        }
    }
    __syncwarp();
    tc_fence_before();
    if (splits > 1) { cluster_arrive(); cluster_wait(); } else __syncthreads();
    // ---- this CTA's share of the tile: four columns of a row of y a thread and turn, all splits' values asked for at
    //      once (they are a trip to another SM away) and added in the order of k -------------------------------------
    {
        constexpr int UNITS = OUT_ROWS / 4;
        constexpr int TURN = MAX_SPLITS * (GLU ? 2 : 1) <= 8 ? 2 : 1;      // units a thread has under way
        const int units = M * UNITS, step = splits * R_THREADS;
        for (int u0 = rank * R_THREADS + threadIdx.x; u0 < units; u0 += TURN * step) {
            float4 v[TURN][MAX_SPLITS], w[TURN][GLU ? MAX_SPLITS : 1];
#pragma unroll
            for (int h = 0; h < TURN; h++) {
                const int u = u0 + h * step;
                const uint32_t at = ring + ((u / UNITS) * R_BM + (u % UNITS) * 4) * 4;
                const bool in = u < units && row0 + (u % UNITS) * 4 < n_out;      // (nothing is read that is not added and stored)
#pragma unroll
                for (int p = 0; p < MAX_SPLITS; p++)
                    if (p < splits && in) {
                        const uint32_t from = MAX_SPLITS > 1 ? cluster_addr(at, p) : at;
                        v[h][p] = ld_cluster16(from);
                        if (GLU) w[h][p] = ld_cluster16(from + R_BM * 2);
                    }
            }
#pragma unroll
            for (int h = 0; h < TURN; h++) {
                const int u = u0 + h * step, m = u / UNITS, c = (u % UNITS) * 4;
                if (u >= units || row0 + c >= n_out) continue;
                float4 a = v[h][0], b = w[h][0];
#pragma unroll
                for (int p = 1; p < MAX_SPLITS; p++)
                    if (p < splits) {
                        a.x += v[h][p].x; a.y += v[h][p].y; a.z += v[h][p].z; a.w += v[h][p].w;
                        if (GLU) { b.x += w[h][p].x; b.y += w[h][p].y; b.z += w[h][p].z; b.w += w[h][p].w; }
                    }
                // (gate, up and what an activation reads are rounded as a product of their own would leave them)
                if (GLU) {
                    a.x = glu_act(act, limit, round_bf16(a.x), round_bf16(b.x));
                    a.y = glu_act(act, limit, round_bf16(a.y), round_bf16(b.y));
                    a.z = glu_act(act, limit, round_bf16(a.z), round_bf16(b.z));
                    a.w = glu_act(act, limit, round_bf16(a.w), round_bf16(b.w));
                } else if (act != UNARY_NONE) {
                    a.x = unary_act(act, round_bf16(a.x));
                    a.y = unary_act(act, round_bf16(a.y));
                    a.z = unary_act(act, round_bf16(a.z));
                    a.w = unary_act(act, round_bf16(a.w));
                }
                store4(y + (size_t)m * n_out + row0 + c, a);
            }
        }
    }
    // A CTA's shared memory stays until its peers have read it.  Every value that a thread read from a peer went into a store to y above (nothing
    // else is read), and the fence keeps those stores ahead of the arrival: what has been stored has been read.  An arrival that releases
    // does the same for 0.3 us more a product, since it also waits until the stores are seen (a prompt of 37 tokens at the 0.6B shape 1140 us, this way
    // 1098; 64 requests 1753 and 1716).  A read whose value is NOT used before the arrival would still be under way when the peer leaves.
    if (splits > 1) {
        __syncwarp();
        asm volatile("fence.acq_rel.cta;\nbarrier.cluster.arrive.relaxed.aligned;\n" ::: "memory");
        cluster_wait();
    } else __syncthreads();
    if (warp == 9) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(tmem_cols));
    }
    if (threadIdx.x == 0 && *abort_flag) atomicOr(status, 64);
}

// ---- host side ----------------------------------------------------------------------------------

// Whether this kernel takes the product (n_out: columns of y).
PLLM_EXPORT int pllm_rows_gemm_supports(int M, int n_out, int K) {
    return M >= 1 && M <= R_MAX_ROWS && K >= 64 && K % R_BK == 0 && n_out >= 64 && n_out % 8 == 0;
}

namespace {

template <bool GLU, int MAX_SPLITS, typename OutT>
int launch_rows(const void* x, const void* w, void* y, int M, int n_out, int K, int act, float limit, int splits, int* status,
                cudaStream_t stream) {
    const int rows = (M + 15) / 16 * 16, stage = 2 * (R_TILE_W + rows * R_BK * 2);
    const int tiles = (n_out + (GLU ? 63 : 127)) / (GLU ? 64 : 128), k_stages = (K + R_SK - 1) / R_SK;
    int stages = R_RING / stage;
    if (stages > R_MAX_STAGES) stages = R_MAX_STAGES;
    const int per = (k_stages + splits - 1) / splits;
    if (stages > per) stages = per;
    size_t smem = (size_t)stages * stage;
    if (smem < (size_t)rows * R_BM * 4) smem = (size_t)rows * R_BM * 4;       // (the partial sums)
    smem += 1024;
    uint32_t cols = 32;
    while (cols < (uint32_t)rows) cols *= 2;
    CUtensorMap map_w, map_x;
    {
        const long long dw[4] = {R_BK, n_out, GLU ? 2 : K / R_BK, K / R_BK}, sw[3] = {2LL * K, GLU ? 2LL * n_out * K : 2LL * R_BK, 2LL * R_BK};
        const int bw[4] = {R_BK, GLU ? 64 : R_BM, 2, 2};
        const long long dx[3] = {R_BK, M, K / R_BK}, sx[2] = {2LL * K, 2LL * R_BK};
        const int bx[3] = {R_BK, rows, 2};
        if (tensor_map(w, GLU ? 4 : 3, dw, sw, bw, true, &map_w) != 0 || tensor_map(x, 3, dx, sx, bx, true, &map_x) != 0) return PLLM_ERR_SIZE;
    }
    cudaFuncSetAttribute(rows_gemm_kernel<GLU, MAX_SPLITS, OutT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    launch_chained_cluster_y(rows_gemm_kernel<GLU, MAX_SPLITS, OutT>, dim3(tiles, splits), dim3(R_THREADS), smem, stream, splits, map_w, map_x,
                             (OutT*)y, M, n_out, K, rows, stages, cols, act, limit, status);
    return launch_status();
}

template <bool GLU, typename OutT>
int pick_splits(const void* x, const void* w, void* y, int M, int n_out, int K, int act, float limit, int splits, int* status, cudaStream_t stream) {
    const int tiles = (n_out + (GLU ? 63 : 127)) / (GLU ? 64 : 128), k_stages = (K + R_SK - 1) / R_SK;
    if (splits <= 0) {
        // K is halved while SMs would have no CTA and each split keeps two stages, and once more, to two CTAs an SM, where
        // each keeps four.  Decode steps of 24 to 64 requests with ONE product's splits changed (us a step, 1 / 2 / 4 / 8):
        // 0.6B shape q/k/v (32 tiles, 8 stages) 1767 / 1707 / 1713 / 1738, gate/up (48, 8) 1285 / 1239 / 1253 / -, down (8, 24)
        // - / - / 1255 / 1227; 8B shape, 8 requests: q/k/v (48, 32) 745 / 724 / 714 / 723, o (32, 32) - / 744 / 725 / 714,
        // gate/up (192, 32) 715 / 742 / 743 / 795, down (32, 96) - / 751 / 728 / 714.
        splits = 1;
        while (splits < 8 && ((tiles * splits * 2 <= sm_count() && k_stages / (splits * 2) >= 2) ||
                              (tiles * splits * 2 <= 2 * sm_count() && k_stages / (splits * 2) >= 4)))
            splits *= 2;
    }
    if (splits > 8 || splits > k_stages) return PLLM_ERR_SIZE;
    if (splits == 1) return launch_rows<GLU, 1, OutT>(x, w, y, M, n_out, K, act, limit, splits, status, stream);
    if (splits <= 4) return launch_rows<GLU, 4, OutT>(x, w, y, M, n_out, K, act, limit, splits, status, stream);
    return launch_rows<GLU, 8, OutT>(x, w, y, M, n_out, K, act, limit, splits, status, stream);
}

}  // namespace

// x: [M, K]; w: [n_out, K], or with glu [2 n_out, K] = gate rows then up rows; y: [M, n_out] bfloat16, or float with out_f32 (plain products).
// glu: 0 a plain product; positive: 1 + the gated activation's kind with its limit; negative: minus a one-argument activation's kind.
// splits: CTAs that share a tile's K (0: as the sizes ask).
PLLM_EXPORT int pllm_rows_gemm(const void* x, const void* w, void* y, int M, int n_out, int K, int glu, float limit, int out_f32, int splits,
                               int* status, cudaStream_t stream) {
    const int unary = glu < 0 ? -glu : UNARY_NONE;
    if (glu < 0) glu = 0;
    if (!pllm_rows_gemm_supports(M, n_out, K) || unary > UNARY_RELU2 || glu > 1 + GLU_CLAMPED || (glu && out_f32)) return PLLM_ERR_SIZE;
    if (((uintptr_t)x | (uintptr_t)w | (uintptr_t)y) & 15) return PLLM_ERR_ALIGN;
    if (glu) return pick_splits<true, bf16>(x, w, y, M, n_out, K, glu - 1, limit, splits, status, stream);
    return out_f32 ? pick_splits<false, float>(x, w, y, M, n_out, K, unary, limit, splits, status, stream)
                   : pick_splits<false, bf16>(x, w, y, M, n_out, K, unary, limit, splits, status, stream);
}

PLLM_TRACE_EXPORT(rows_gemm_tcgen05)
