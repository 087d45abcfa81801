// Y[M,N] = LayerNorm(A[M,K] @ W[K,N] + bias + residual) * gamma + beta for few rows: one 64 x 64, 64 x 128 or 128 x 128 tile per thread
// block, the thread blocks of a row block (N / BN of them, at most 16) form a cluster.
//
// gemm_ln.cu's 256-row blocks leave a few hundred rows to a handful of multiprocessors (128 rows x 768 columns: six); here 24 share
// them.  Main loop and the way of starting early are gemm_split.cu's.  Epilogue: one row and 64 columns per thread; x = accumulator +
// bias + residual goes back into tensor memory (fp32), 16 columns at a time; the thread's mean and centred sum of squares over its 64
// columns go into a table of the block, one bulk copy per peer brings the table to every other block of the cluster, and x, read
// again, is normalised with the merged statistics (parallel variance).  Statistics are fp32 and taken before any rounding to fp16.
// Measured (weights from HBM, back to back, K = N = 768, with residual): 128 rows 5.1 us, 1024 rows 7.8 us, where 128 x 256 tiles of one
// block each took 12.6 and 12.8.
#include <atomic>
#include "gemm_split.cuh"

namespace stof {
namespace {

constexpr int SL_MAX_CLUSTER = 16;               // thread blocks per row block; more than 8 need the non-portable cluster size

// merges (n_b, mean_b, m2_b) into (n_a, mean_a, m2_a): parallel variance (Chan et al.)
__device__ __forceinline__ void merge_row_stats(float& n_a, float& mean_a, float& m2_a, float n_b, float mean_b, float m2_b) {
    const float n = n_a + n_b;
    const float delta = mean_b - mean_a;
    const float f = __fdividef(n_b, n);                    // small whole numbers
    mean_a = fmaf(delta, f, mean_a);
    m2_a = m2_a + m2_b + delta * delta * n_a * f;
    n_a = n;
}

template <int BM, int BN>
__global__ void __launch_bounds__(SplitShape<BM, BN>::THREADS, 1)
gemm_split_ln_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, const __half* bias, const __half* residual,
                     long long ldr, const __half* gamma, const __half* beta, float eps, __half* c, long long ldc, int m, int k, int cluster, int stages,
                     int* status) {
    using Shape = SplitShape<BM, BN>;
    constexpr int EPI_WARPS = Shape::EPI_WARPS, PARTS = BN / 64;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    // stages | statistics of the row block: [block of the cluster][64-column part][row] {mean, centred sum of squares} | residual |
    // bias, gamma, beta | barriers
    float2* table = reinterpret_cast<float2*>(smem + stages * Shape::STAGE_BYTES);
    unsigned char* s_res = reinterpret_cast<unsigned char*>(table + cluster * PARTS * BM);
    unsigned char* s_vec = s_res + Shape::RESIDUAL_BYTES;
    uint64_t* bars = reinterpret_cast<uint64_t*>(s_vec + 3 * BN * 2);
    uint64_t *full = bars, *empty = bars + Shape::MAX_STAGES, *tfull = bars + 2 * Shape::MAX_STAGES, *received = tfull + 1;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(received + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = static_cast<int>(cluster_rank());
    const int m0 = static_cast<int>(blockIdx.x) / cluster * BM, n0 = rank * BN;
    const int kblocks = (k + S_BK - 1) / S_BK;
    const WaitCtx wctx{abort_flag, status};

    if (warp == EPI_WARPS + 1) {
        tmem_alloc(tmem_slot, BN);
        tmem_relinquish();
    } else if (warp == EPI_WARPS) {
        if (elect_one()) split_prefetch<BN>(map_a, map_w, n0, 0, kblocks, stages);
    } else if (threadIdx.x == 0) {
        *abort_flag = 0;
        for (int i = 0; i < stages; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        mbar_init(tfull, 1);
        mbar_init(received, 1);
        fence_mbar_init();
        mbar_arrive_expect_tx(received, static_cast<uint32_t>((cluster - 1) * PARTS * BM * 8));
    }
    tc_fence_before();
    __syncwarp();
    cluster_sync_all();                          // every block's barriers exist before a peer's copy reports to them
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    if (warp == EPI_WARPS) {
        split_produce<Shape, BN>(map_a, map_w, smem, full, empty, m0, n0, 0, kblocks, stages, wctx);
    } else if (warp == EPI_WARPS + 1) {
        split_multiply<Shape, BM, BN>(smem, full, empty, tfull, tmem_base, 0, kblocks, stages, wctx);
    } else {
        grid_dependency_wait();
        const uint4* s_bias = reinterpret_cast<const uint4*>(s_vec);
        stage_vector(s_vec, bias != nullptr ? bias + n0 : nullptr, BN, BN, 0u, 0);
        stage_vector(s_vec + 2 * BN, gamma != nullptr ? gamma + n0 : nullptr, BN, BN, 0x3C003C00u, 32);       // 1.0
        stage_vector(s_vec + 4 * BN, beta != nullptr ? beta + n0 : nullptr, BN, BN, 0u, 64);
        stage_residual<Shape>(s_res, residual, ldr, m0, n0, m, cluster * BN, 0, BM);
        const bool mute = failure_reported(status);
        copy_async_wait();
        epilogue_barrier<Shape::EPI_THREADS>();
        const int quarter = warp & 3, part = warp >> 2;
        const bool mine = BM == 128 || lane < 16;            // (a 64-row accumulator: 16 rows in the lower lanes of each quarter)
        const int lrow = BM == 128 ? quarter * 32 + lane : quarter * 16 + (lane & 15);
        const int row = m0 + lrow;
        const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + part * 64;
        mbar_wait_addr(smem_u32(tfull), 0, wctx, 2 * stages);
        tc_fence_after();
        // x = accumulator + bias + residual back into tensor memory; this thread's statistics over its 64 columns, 16 at a time
        float cnt = 0.f, mean = 0.f, m2 = 0.f;
#pragma unroll 1
        for (int g0 = 0; g0 < 8; g0 += 2) {
            uint32_t r[16];
            tmem_ld16(t_row + g0 * 8, r);
            tc_wait_ld();
            float2 sum2 = pk2(0.f, 0.f);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int g = part * 8 + g0 + h;
                const uint4 bu = s_bias[g], ru = *reinterpret_cast<const uint4*>(s_res + Shape::residual_at(lrow, g));
                const __half2 *bh = reinterpret_cast<const __half2*>(&bu), *rh = reinterpret_cast<const __half2*>(&ru);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    float2 x = pk2(__uint_as_float(r[8 * h + 2 * j]), __uint_as_float(r[8 * h + 2 * j + 1]));
                    x = add2(add2(x, __half22float2(bh[j])), __half22float2(rh[j]));
                    sum2 = add2(sum2, x);
                    r[8 * h + 2 * j] = __float_as_uint(x.x);
                    r[8 * h + 2 * j + 1] = __float_as_uint(x.y);
                }
            }
            tmem_st16(t_row + g0 * 8, r);
            const float mean_c = (sum2.x + sum2.y) * (1.0f / 16.0f);
            const float2 nm = pk2(-mean_c, -mean_c);
            float2 sq2 = pk2(0.f, 0.f);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float2 d = add2(pk2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1])), nm);
                sq2 = fma2(d, d, sq2);
            }
            merge_row_stats(cnt, mean, m2, 16.f, mean_c, sq2.x + sq2.y);
        }
        if (mine) table[(rank * PARTS + part) * BM + lrow] = make_float2(mean, m2);
        tc_wait_st();
        fence_proxy_async_smem();
        epilogue_barrier<Shape::EPI_THREADS>();                  // the block's own table is written
        if (static_cast<int>(threadIdx.x) < cluster && static_cast<int>(threadIdx.x) != rank) {
            const uint32_t own = smem_u32(table + rank * PARTS * BM), to = threadIdx.x;
            bulk_copy_to_peer(map_to_rank(own, to), own, PARTS * BM * 8, map_to_rank(smem_u32(received), to));
        }
        __syncwarp();
        mbar_wait_addr(smem_u32(received), 0, wctx, 2 * stages + 1);
        // The row's statistics, in the same order in every block.  All parts have 64 values: the mean of the means, and the parts'
        // squares about their own means plus 64 times the squares of those means about the common one
        float sum = 0.f;
#pragma unroll 4
        for (int p = 0; p < cluster * PARTS; ++p) sum += table[p * BM + lrow].x;
        mean = sum * (1.0f / static_cast<float>(cluster * PARTS));
        m2 = 0.f;
#pragma unroll 4
        for (int p = 0; p < cluster * PARTS; ++p) {
            const float2 t = table[p * BM + lrow];
            const float d = t.x - mean;
            m2 += fmaf(64.0f * d, d, t.y);
        }
        const float rstd = 1.0f / sqrtf(m2 * (1.0f / static_cast<float>(cluster * BN)) + eps);
        const float2 rstd2 = pk2(rstd, rstd), shift2 = pk2(-mean * rstd, -mean * rstd);
        const bool store = mine && row < m && !mute;
        __half* out = c + static_cast<size_t>(row) * ldc + n0;
#pragma unroll 1
        for (int g0 = 0; g0 < 8; g0 += 2) {
            uint32_t r[16];
            tmem_ld16(t_row + g0 * 8, r);
            tc_wait_ld();
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int g = part * 8 + g0 + h;
                const uint4 gu = s_bias[BN / 8 + g], bu = s_bias[BN / 4 + g];
                const __half2 *gh = reinterpret_cast<const __half2*>(&gu), *bh = reinterpret_cast<const __half2*>(&bu);
                uint32_t o[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    float2 y = fma2(pk2(__uint_as_float(r[8 * h + 2 * j]), __uint_as_float(r[8 * h + 2 * j + 1])), rstd2, shift2);
                    y = fma2(y, __half22float2(gh[j]), __half22float2(bh[j]));
                    o[j] = pack_half2(y.x, y.y);
                }
                if (store) *reinterpret_cast<uint4*>(out + 8 * g) = make_uint4(o[0], o[1], o[2], o[3]);
            }
        }
    }
    tc_fence_before();
    __syncwarp();
    cluster_sync_relaxed();                      // nobody leaves while a peer may still be reading out what it was sent from here
    tc_fence_after();
    if (warp == EPI_WARPS + 1) tmem_dealloc(tmem_base, BN);
}

template <int BM, int BN>
int launch_split_ln(const SplitLnCall& x, int* fits) {
    using Shape = SplitShape<BM, BN>;
    const int cluster = x.n / BN, row_blocks = (x.m + BM - 1) / BM;
    const int steps = (x.k + S_BK - 1) / S_BK;
    auto smem = [&](int stages) { return 1024 + static_cast<size_t>(stages) * Shape::STAGE_BYTES + static_cast<size_t>(x.n / 64) * BM * 8 + Shape::RESIDUAL_BYTES + 3 * BN * 2 + S_BAR_BYTES; };
    int stages = steps < Shape::MAX_STAGES ? steps : Shape::MAX_STAGES;
    while (stages > 1 && smem(stages) > S_SMEM_LIMIT) --stages;
    static std::atomic<bool> configured[64];     // per device; host threads may race here, every one of them stores the same value
    static std::atomic<int> resident[64][SL_MAX_CLUSTER + 1];
    int dev = 0;
    STOF_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        STOF_CUDA(cudaFuncSetAttribute(gemm_split_ln_kernel<BM, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, S_SMEM_LIMIT));
        STOF_CUDA(cudaFuncSetAttribute(gemm_split_ln_kernel<BM, BN>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    LaunchConfig lc(dim3(static_cast<unsigned>(row_blocks * cluster)), SplitShape<BM, BN>::THREADS, smem(stages), x.stream, static_cast<unsigned>(cluster));
    int clusters = (dev >= 0 && dev < 64) ? resident[dev][cluster].load() : 0;
    if (clusters == 0) {                         // how many clusters of this size the GPU holds at once, with a full ring of stages
        cudaLaunchConfig_t query = lc.cfg;
        query.dynamicSmemBytes = S_SMEM_LIMIT;
        query.attrs = &lc.attr[1];
        query.numAttrs = 1;
        if (cluster == 1) clusters = sm_count();
        else if (cudaOccupancyMaxActiveClusters(&clusters, gemm_split_ln_kernel<BM, BN>, &query) != cudaSuccess) {
            cudaGetLastError();
            clusters = 0;
        }
        if (clusters < 1) clusters = -1;         // clusters of this size do not run on this GPU
        if (dev >= 0 && dev < 64) resident[dev][cluster].store(clusters);
    }
    *fits = clusters >= row_blocks ? 1 : 0;
    if (*fits == 0) return STOF_OK;
    CUtensorMap ma;
    if (int rc = split_map_a<BM>(&ma, x.a, x.lda, x.m, x.k)) return rc;
    STOF_CUDA(cudaLaunchKernelEx(&lc.cfg, gemm_split_ln_kernel<BM, BN>, ma, *x.map_w, x.bias, x.residual, x.ldr, x.gamma, x.beta, x.eps, x.c, x.ldc,
                                 x.m, x.k, cluster, stages, x.status));
    return STOF_OK;
}

}  // namespace

int gemm_split_ln_dispatch(const SplitLnCall& x, int* done) {
    *done = 0;
    if (x.n % 64 == 0 && x.n / 64 <= SL_MAX_CLUSTER) {
        if (int rc = launch_split_ln<64, 64>(x, done)) return rc;
        if (*done != 0) return STOF_OK;
    }
    if (x.n % 128 == 0 && x.n / 128 <= SL_MAX_CLUSTER) {
        if (int rc = launch_split_ln<64, 128>(x, done)) return rc;
        if (*done != 0) return STOF_OK;
        if (int rc = launch_split_ln<128, 128>(x, done)) return rc;
    }
    return STOF_OK;
}

}  // namespace stof
