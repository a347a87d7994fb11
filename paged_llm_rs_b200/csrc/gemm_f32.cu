// y[M, N] = x[M, K] . W[N, K]^T in true float32 on the CUDA cores: the float32 path's projections of few rows, or of some more into
// few columns (kernels/ops.py, gemm_f32_sizes).  The reference calls a library product (crates/pagedllm/src/model/layers.rs:27-35),
// whose tiles leave most of the chip idle there (256 rows, 1024 x 2048: 50 us, 21 of the 74 TFLOP/s).
//
// What bounds it: the multiply-adds from some 20 rows on (128 a clock and SM), the bytes of W below.  Hence
//   - both operands go to shared memory as they lie (K runs along the rows), 32 values of k a stage, three stages by
//     cp.async; a row's 16-byte chunks are stored at chunk ^ (row & 7), so that neither the copies nor the reads conflict;
//   - a thread makes TM x TN sums and reads four values of k of a row at once; a sum is kept as two, of the even and of the
//     odd k, so that fma.rn.f32x2 takes the operands as they were loaded (half the instructions of fmaf, whose issue
//     would otherwise compete with the loads from shared memory);
//   - the tile follows the rows of x: 128 x 64, 32 x 128 or 16 x 256 (the fewer rows, the more of W a CTA reads for them);
//   - K is split over a cluster's CTAs where the tiles alone would leave SMs idle; the partial tiles meet in shared memory
//     and are added in the order of k, so that a result does not depend on what ran where.
#include "common.cuh"

namespace {

constexpr int F_BK = 32, F_STAGES = 3, F_THREADS = 256;

__device__ __forceinline__ uint32_t f_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// 16 bytes into shared memory, or zeros
__device__ __forceinline__ void copy16(uint32_t dst, const float* src, bool live) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ void fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;\n" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ float halves(unsigned long long v) { return __uint_as_float((uint32_t)v) + __uint_as_float((uint32_t)(v >> 32)); }
__device__ __forceinline__ ulonglong2 lds16(uint32_t addr) {
    ulonglong2 v;
    asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];\n" : "=l"(v.x), "=l"(v.y) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ float f_ld_cluster(uint32_t addr, uint32_t rank) {
    uint32_t at;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(at) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];\n" : "=f"(v) : "r"(at) : "memory");
    return v;
}

}  // namespace

// Grid (tiles of N, tiles of M, splits of K), clusters of the splits.  K a multiple of 4.
template <int TM, int TN, int TY, int TX>
__global__ void __launch_bounds__(F_THREADS, 2) gemm_f32_kernel(const float* x, const float* __restrict__ w, float* __restrict__ y, int M, int N, int K) {
    static_assert(TY * TX == F_THREADS, "a thread to TM x TN sums");
    constexpr int BM = TM * TY, BN = TN * TX, STAGE = (BM + BN) * F_BK * 4;
    extern __shared__ __align__(128) unsigned char smem[];
    const uint32_t ring = f_smem(smem);
    const int tx = threadIdx.x % TX, ty = threadIdx.x / TX;
    const int n0 = blockIdx.x * BN, m0 = blockIdx.y * BM;
    const int splits = gridDim.z, rank = blockIdx.z;
    const int k_blocks = (K + F_BK - 1) / F_BK;
    const int kb0 = k_blocks * rank / splits, n_kb = k_blocks * (rank + 1) / splits - kb0;

    auto load_w = [&](int i) {
        const uint32_t base = ring + (i % F_STAGES) * STAGE + BM * F_BK * 4;
        const int k0 = (kb0 + i) * F_BK;
        for (int c = threadIdx.x; c < BN * 8; c += F_THREADS) {
            const int r = c >> 3, q = c & 7, k = k0 + q * 4;
            const bool live = n0 + r < N && k < K;
            copy16(base + r * 128 + ((q ^ (r & 7)) << 4), live ? w + (size_t)(n0 + r) * K + k : w, live);
        }
    };
    auto load_x = [&](int i) {
        const uint32_t base = ring + (i % F_STAGES) * STAGE;
        const int k0 = (kb0 + i) * F_BK;
        for (int c = threadIdx.x; c < BM * 8; c += F_THREADS) {
            const int r = c >> 3, q = c & 7, k = k0 + q * 4;
            const bool live = m0 + r < M && k < K;
            copy16(base + r * 128 + ((q ^ (r & 7)) << 4), live ? x + (size_t)(m0 + r) * K + k : x, live);
        }
    };
    unsigned long long acc[TM][TN];
#pragma unroll
    for (int a = 0; a < TM; a++)
#pragma unroll
        for (int b = 0; b < TN; b++) acc[a][b] = 0ull;

    // the weights do not depend on the kernel before this one; x does
    for (int i = 0; i < F_STAGES - 1 && i < n_kb; i++) load_w(i);
    pdl_launch_dependents();
    pdl_wait(KID_GEMM);
#pragma unroll
    for (int i = 0; i < F_STAGES - 1; i++) {
        if (i < n_kb) load_x(i);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    for (int i = 0; i < n_kb; i++) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(F_STAGES - 2) : "memory");
        __syncthreads();          // this stage is there for all, and the one that is loaded next has been read by all
        if (i + F_STAGES - 1 < n_kb) { load_w(i + F_STAGES - 1); load_x(i + F_STAGES - 1); }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        const uint32_t xs = ring + (i % F_STAGES) * STAGE, ws = xs + BM * F_BK * 4;
#pragma unroll
        for (int q = 0; q < F_BK / 4; q++) {
            ulonglong2 xv[TM];
#pragma unroll
            for (int a = 0; a < TM; a++) {
                const int r = ty + a * TY;
                xv[a] = lds16(xs + r * 128 + ((q ^ (r & 7)) << 4));
            }
#pragma unroll
            for (int b = 0; b < TN; b++) {
                const int r = tx + b * TX;
                const ulonglong2 wv = lds16(ws + r * 128 + ((q ^ (r & 7)) << 4));
#pragma unroll
                for (int a = 0; a < TM; a++) {
                    fma2(acc[a][b], xv[a].x, wv.x);
                    fma2(acc[a][b], xv[a].y, wv.y);
                }
            }
        }
    }
    if (splits == 1) {
#pragma unroll
        for (int a = 0; a < TM; a++)
#pragma unroll
            for (int b = 0; b < TN; b++) {
                const int m = m0 + ty + a * TY, n = n0 + tx + b * TX;
                if (m < M && n < N) y[(size_t)m * N + n] = halves(acc[a][b]);
            }
        return;
    }
    // ---- the splits' partial tiles: [row of x][row of W] in shared memory, each CTA adds a share of the rows ------------
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
    float* part = reinterpret_cast<float*>(smem);
#pragma unroll
    for (int a = 0; a < TM; a++)
#pragma unroll
        for (int b = 0; b < TN; b++) part[(ty + a * TY) * BN + tx + b * TX] = halves(acc[a][b]);
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    const int live = (M - m0 < BM ? M - m0 : BM) * BN;
    for (int u = rank * F_THREADS + threadIdx.x; u < live; u += splits * F_THREADS) {
        const int m = m0 + u / BN, n = n0 + u % BN;
        if (n >= N) continue;          // (nothing is read that is not added and stored)
        float v[8];
#pragma unroll
        for (int p = 0; p < 8; p++)
            if (p < splits) v[p] = f_ld_cluster(ring + u * 4, p);
        float s = v[0];
#pragma unroll
        for (int p = 1; p < 8; p++)
            if (p < splits) s += v[p];
        y[(size_t)m * N + n] = s;
    }
    // A CTA's shared memory stays until its peers have read it.  Every value that a thread read from a peer went into a store to y above, and the
    // fence keeps those stores ahead of the arrival (rows_gemm_tcgen05.cu says more)
    __syncwarp();
    asm volatile("fence.acq_rel.cta;\nbarrier.cluster.arrive.relaxed.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

// Whether this kernel takes the product.
PLLM_EXPORT int pllm_gemm_f32_supports(int M, int N, int K) { return M >= 1 && N >= 1 && K >= 4 && K % 4 == 0 && (M + 127) / 128 <= 65535; }

namespace {

template <int TM, int TN, int TY, int TX>
int launch_f32(const float* x, const float* w, float* y, int M, int N, int K, int splits, cudaStream_t stream) {
    constexpr int BM = TM * TY, BN = TN * TX;
    constexpr size_t smem = (size_t)F_STAGES * (BM + BN) * F_BK * 4;
    static_assert(smem >= (size_t)BM * BN * 4, "the partial tile lies where the stages were");
    const int k_blocks = (K + F_BK - 1) / F_BK;
    const long long tiles = (long long)((M + BM - 1) / BM) * ((N + BN - 1) / BN);
    if (splits <= 0) {
        // Two CTAs fit an SM.  The splits that leave the fewest places empty in the last turn of them, with four blocks of k or
        // more each; fewer where that is as good, since a split's partial sums cost a meeting.
        const long long places = 2LL * sm_count();
        double best = 0.0;
        splits = 1;
        for (int s = 1; s <= 8 && (s == 1 || k_blocks / s >= 4); s++) {
            const long long turns = (tiles * s + places - 1) / places;
            const double used = (double)(tiles * s) / (double)(turns * places);
            if (used > best * 1.1) { best = used; splits = s; }
        }
    }
    if (splits > 8 || splits > k_blocks) return PLLM_ERR_SIZE;
    cudaFuncSetAttribute(gemm_f32_kernel<TM, TN, TY, TX>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    launch_chained_cluster(gemm_f32_kernel<TM, TN, TY, TX>, dim3((N + BN - 1) / BN, (M + BM - 1) / BM, splits), dim3(F_THREADS), smem, stream,
                           dim3(1, 1, splits), x, w, y, M, N, K);
    return launch_status();
}

}  // namespace

// x: [M, K]; w: [N, K]; y: [M, N], all float.  tile: rows of x a tile (16, 32 or 128; 0: as the sizes ask), splits likewise.
PLLM_EXPORT int pllm_gemm_f32(const float* x, const float* w, float* y, int M, int N, int K, int tile, int splits, cudaStream_t stream) {
    if (!pllm_gemm_f32_supports(M, N, K)) return PLLM_ERR_SIZE;
    if (((uintptr_t)x | (uintptr_t)w) & 15) return PLLM_ERR_ALIGN;
    // (up to 64 rows, and 128 where W has few, two to four tiles of 32 rows rather than one of 128: 1024 x 2048 at 64 rows 22.9 us, 37.4)
    if (tile == 0) tile = M <= 16 ? 16 : (M <= 64 || (M <= 128 && N <= 1024) ? 32 : 128);
    if (tile == 16) return launch_f32<4, 4, 4, 64>(x, w, y, M, N, K, splits, stream);
    if (tile == 32) return launch_f32<4, 4, 8, 32>(x, w, y, M, N, K, splits, stream);
    if (tile == 128) return launch_f32<8, 4, 16, 16>(x, w, y, M, N, K, splits, stream);
    return PLLM_ERR_SIZE;
}

PLLM_TRACE_EXPORT(gemm_f32)
