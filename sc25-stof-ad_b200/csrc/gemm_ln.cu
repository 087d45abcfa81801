// Y[M,N] = LayerNorm(A[M,K] @ W[K,N] + bias + residual) * gamma + beta, with the row statistics taken inside the GEMM's
// epilogue (tcgen05 cta_group::2 + TMEM + TMA), for N a multiple of 256 up to 1024.
//
// The main loop is gemm_pair.cu's: two thread blocks on neighbouring SMs multiply a 256 x 256 tile, each holding 128 rows of it and
// staging 128 of the 256 columns of W.  A LayerNorm row spans all N columns, so the N / 256 pairs that hold the column slices of the
// same 256 rows form a CLUSTER (2 to 8 blocks; block 2c + h owns rows h * 128 .. of column slice c) and exchange per-row partial
// statistics through distributed shared memory.  Persistent: cluster i walks the 256-row blocks i, i + clusters, ...
//   warp 16     TMA producer: A tile (128 rows x 64 k) and two 64 x 64 W boxes per stage, 4 stages of 32 KB, reported to the leader
//               of the pair (plain loads of this GPU's memory; every pair of the cluster fetches the A rows itself, from L2 after the first)
//   warp 17     leader of a pair: tcgen05.mma 256 x 256 x 16 into one of two 256-column fp32 accumulators
//   warps 0-15  epilogue, one row (tensor-memory lane) and 64 columns per thread, x = accumulator + bias + residual held in registers:
//               the accumulator is handed back as soon as it has been read; the residual tile was put into the warp's slab by a TMA
//               load issued when the slab came free, and into L2 a row block earlier.  Mean and centred sum of squares over the 64
//               columns are merged over the four warps of a row through shared memory, one of them sends the block's result to each
//               block of the cluster that holds the same rows (st.async, counted by that block's "partials complete" barrier), and
//               once all N / 256 results have arrived x is normalised, scaled, shifted, packed to fp16 over the residual in the slab
//               and written with a TMA store.
// What bounds it: the main loop from K = 1024 on, below that the epilogue.  With 8 epilogue warps of 128 columns each, x written back to
// tensor memory, the residual loaded row by row (16 of every 2048 bytes per request) and releasing remote arrives, a row block of 128 took
// 11 to 16 us whatever K was.  With residual, K = N = 768: 32768 rows 100 -> 49 us, 8192 24.1 -> 19.3; K = N = 1024: 32768 rows 133 -> 78 us.
// (At 18 warps the cap is 96 registers; 56 bytes are spilled and 104 read back.)
// The statistics are fp32 and taken before any rounding to fp16 (the unfused path rounds the GEMM output first).
// Both tables and the "partials complete" barriers are double-buffered like the accumulators: a block may run at most one row block
// ahead of its peers, because it cannot complete row block t + 1 before every peer has contributed to it; a peer's warps contribute
// to t + 1 only behind a barrier of the four warps of the row, which every one of them reaches after it has read what it needs of t.
// All blocks of a cluster meet at a cluster barrier before they leave: nobody frees shared memory a peer may still write.
#include <cstdlib>
#include <atomic>
#include "gemm_split.h"
#include "stof_ptx.cuh"

namespace stof {
namespace {

constexpr int L_BM = 128, L_BN = 256, L_BK = 64;      // per block: 128 rows x 256 columns of the pair's 256 x 256 tile
constexpr int L_STAGES = 4;
constexpr int L_A_BYTES = L_BM * L_BK * 2;            // 16 KB
constexpr int L_B_BYTES = L_BK * (L_BN / 2) * 2;      // 16 KB: this block's 128 of the 256 W columns
constexpr int L_STAGE_BYTES = L_A_BYTES + L_B_BYTES;
constexpr int L_PARTS = L_BN / 64;                    // epilogue warps per 32 rows
constexpr int L_EPI_WARPS = 4 * L_PARTS;
constexpr int L_THREADS = (L_EPI_WARPS + 2) * 32;
constexpr int L_TMEM_COLS = 512;
constexpr int L_SLAB_BYTES = 32 * 64 * 2;
constexpr int L_MAX_SLICES = 4;                       // N <= 1024
constexpr int L_VEC_BYTES = 3 * L_BN * 4;             // bias, gamma, beta of the block's columns, as fp32
constexpr int L_LOCAL_BYTES = 2 * L_PARTS * L_BM * 8;          // [accumulator][64-column part][row] {mean, centred sum of squares}
constexpr int L_TABLE_BYTES = 2 * L_MAX_SLICES * L_BM * 8;     // [accumulator][column slice][row]
constexpr size_t L_SMEM = 1024 + static_cast<size_t>(L_STAGES) * L_STAGE_BYTES + L_EPI_WARPS * L_SLAB_BYTES + L_VEC_BYTES + L_LOCAL_BYTES +
                          L_TABLE_BYTES + 512;

enum { LB_FULL = 0, LB_EMPTY = L_STAGES, LB_TFULL = 2 * L_STAGES, LB_TEMPTY = 2 * L_STAGES + 2, LB_PART = 2 * L_STAGES + 4,
       LB_RES = 2 * L_STAGES + 6, LB_COUNT = LB_RES + L_EPI_WARPS };

// 8 bytes into a block of the cluster, reported to that block's mbarrier: unlike a store followed by an arrive that releases at
// cluster scope, which waited 3000 cycles for whatever else the thread had under way, it costs the sender nothing
__device__ __forceinline__ void st_async_f32x2(uint32_t cluster_addr, float a, float b, uint32_t bar_cluster_addr) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];" ::"r"(cluster_addr), "f"(a), "f"(b),
                 "r"(bar_cluster_addr)
                 : "memory");
}
// `count` parts of a row, PART_N values each: mean of the means, and the parts' squares about their own means plus PART_N times
// the squares of those means about the common one
template <int PART_N>
__device__ __forceinline__ float2 merge_parts(const float2* parts, int count) {
    float sum = 0.f, m2 = 0.f;
    for (int i = 0; i < count; ++i) sum += parts[i * L_BM].x;
    const float mean = sum / static_cast<float>(count);
    for (int i = 0; i < count; ++i) {
        const float2 t = parts[i * L_BM];
        const float d = t.x - mean;
        m2 += fmaf(static_cast<float>(PART_N) * d, d, t.y);
    }
    return make_float2(mean, m2);
}

__global__ void __launch_bounds__(L_THREADS, 1)
gemm_ln_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_c,
               const __grid_constant__ CUtensorMap map_r, const __half* bias, int has_residual, const __half* gamma, const __half* beta, float eps,
               int m, int n, int k, int slices, int* status) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    unsigned char* slabs = smem + L_STAGES * L_STAGE_BYTES;          // one 4 KB slab per epilogue warp, 1024-aligned
    unsigned char* s_vec = slabs + L_EPI_WARPS * L_SLAB_BYTES;
    float2* local = reinterpret_cast<float2*>(s_vec + L_VEC_BYTES);
    float2* table = reinterpret_cast<float2*>(reinterpret_cast<unsigned char*>(local) + L_LOCAL_BYTES);
    uint64_t* bars = reinterpret_cast<uint64_t*>(reinterpret_cast<unsigned char*>(table) + L_TABLE_BYTES);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + LB_COUNT);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = static_cast<int>(cluster_rank()), size = 2 * slices;
    const int slice = rank >> 1, half = rank & 1;
    const bool leader = half == 0;
    const int cluster_id = blockIdx.x / size, clusters = gridDim.x / size;
    const int tiles_m = (m + 2 * L_BM - 1) / (2 * L_BM);
    const int kblocks = (k + L_BK - 1) / L_BK;
    const int n0 = slice * L_BN;
    const WaitCtx wctx{abort_flag, status};

    if (threadIdx.x == 0) {
        *abort_flag = 0;
        for (int i = 0; i < L_STAGES; ++i) {
            mbar_init(&bars[LB_FULL + i], 1);                 // the leader's: its own arrive.expect_tx; bytes from both blocks of the pair
            mbar_init(&bars[LB_EMPTY + i], 1);                // a commit of the leader, in both blocks
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&bars[LB_TFULL + i], 1);                // a commit of the leader, in both blocks
            mbar_init(&bars[LB_TEMPTY + i], 2 * L_EPI_WARPS); // the leader's: the epilogue warps of both blocks
            mbar_init(&bars[LB_PART + i], 1);                 // one local arrive.expect_tx; the bytes of all column slices
        }
        for (int i = 0; i < L_EPI_WARPS; ++i) mbar_init(&bars[LB_RES + i], 1);
        fence_mbar_init();
    }
    if (warp == L_EPI_WARPS + 1) {
        tmem_alloc_pair(tmem_slot, L_TMEM_COLS);
        tmem_relinquish_pair();
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();                                       // every block's barriers exist before any remote store, copy or arrive
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    grid_dependency_wait();
    grid_launch_dependents();

    if (warp == L_EPI_WARPS) {
        // ------------------------------------------------------------------ TMA producer (both blocks of a pair)
        if (elect_one()) {
            tma_prefetch_desc(&map_a);
            tma_prefetch_desc(&map_w);
            int it = 0;
            for (int rb = cluster_id; rb < tiles_m; rb += clusters) {
                const int m0 = rb * (2 * L_BM) + half * L_BM;
                const int w0 = n0 + half * (L_BN / 2);
                for (int kb = 0; kb < kblocks; ++kb, ++it) {
                    const int s = it % L_STAGES;
                    const uint32_t ph = (it / L_STAGES) & 1;
                    mbar_wait(&bars[LB_EMPTY + s], ph ^ 1, wctx, LB_EMPTY + s);
                    if (leader) mbar_arrive_expect_tx(&bars[LB_FULL + s], 2 * L_STAGE_BYTES);
                    const uint32_t full = map_to_rank(smem_u32(&bars[LB_FULL + s]), static_cast<uint32_t>(rank & ~1));
                    unsigned char* a_dst = smem + s * L_STAGE_BYTES;
                    unsigned char* b_dst = a_dst + L_A_BYTES;
                    tma_load_2d_pair(a_dst, &map_a, full, kb * L_BK, m0);
#pragma unroll
                    for (int j = 0; j < L_BN / 128; ++j)
                        tma_load_2d_pair(b_dst + j * (L_BK * 64 * 2), &map_w, full, w0 + 64 * j, kb * L_BK);
                }
            }
        }
    } else if (warp == L_EPI_WARPS + 1) {
        // ------------------------------------------------------------------ MMA issuer (leader of a pair)
        if (leader && elect_one()) {
            constexpr uint32_t idesc = make_idesc_f16(2 * L_BM, L_BN, /*b_mn_major=*/true);
            const uint32_t peer = static_cast<uint32_t>(rank + 1);
            int it = 0, tile = 0;
            for (int rb = cluster_id; rb < tiles_m; rb += clusters, ++tile) {
                const int acc = tile & 1;
                const uint32_t acc_ph = (tile >> 1) & 1;
                mbar_wait(&bars[LB_TEMPTY + acc], acc_ph ^ 1, wctx, LB_TEMPTY + acc);
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + acc * L_BN;
                for (int kb = 0; kb < kblocks; ++kb, ++it) {
                    const int s = it % L_STAGES;
                    const uint32_t ph = (it / L_STAGES) & 1;
                    mbar_wait(&bars[LB_FULL + s], ph, wctx, LB_FULL + s);
                    tc_fence_after();
                    const uint32_t a_addr = smem_u32(smem + s * L_STAGE_BYTES);
                    const uint32_t b_addr = a_addr + L_A_BYTES;
#pragma unroll
                    for (int kk = 0; kk < L_BK / 16; ++kk) {
                        const uint64_t a_desc = make_smem_desc_sw128(a_addr + kk * 32, 16, 1024);
                        const uint64_t b_desc = make_smem_desc_sw128(b_addr + kk * 2048, L_BK * 64 * 2, 1024);
                        mma_f16_ss_pair(d_tmem, a_desc, b_desc, idesc, (kb > 0 || kk > 0) ? 1u : 0u);
                    }
                    tc_commit_pair(smem_u32(&bars[LB_EMPTY + s]));
                    tc_commit_pair(map_to_rank(smem_u32(&bars[LB_EMPTY + s]), peer));
                }
                tc_commit_pair(smem_u32(&bars[LB_TFULL + acc]));
                tc_commit_pair(map_to_rank(smem_u32(&bars[LB_TFULL + acc]), peer));
            }
        }
    } else {
        // ------------------------------------------------------------------ epilogue (all blocks)
        const int quarter = warp & 3, part = warp >> 2;
        const int lrow = quarter * 32 + lane;                 // row inside the block's 128 = tensor-memory lane
        const int col0 = n0 + part * 64;
        unsigned char* slab = slabs + warp * L_SLAB_BYTES;
        unsigned char* slab_row = slab + lane * 128;
        uint64_t* res_bar = &bars[LB_RES + warp];
        const float inv_n = 1.0f / static_cast<float>(n);
        const bool mute = failure_reported(status);
        auto request_residual = [&](int rb) {                 // one lane: the warp's 32 x 64 piece, rows beyond the matrix as zeros
            mbar_arrive_expect_tx(res_bar, L_SLAB_BYTES);
            tma_load_2d(slab, &map_r, res_bar, col0, rb * (2 * L_BM) + half * L_BM + quarter * 32);
        };
        if (has_residual && lane == 0 && cluster_id < tiles_m) request_residual(cluster_id);
        if (threadIdx.x < 3 * L_BN / 2) {                     // the block's columns of the three vectors
            const int v = threadIdx.x / (L_BN / 2), i = threadIdx.x % (L_BN / 2);
            const __half* src = v == 0 ? bias : (v == 1 ? gamma : beta);
            const float none = v == 1 ? 1.0f : 0.0f;
            reinterpret_cast<float2*>(s_vec)[threadIdx.x] =
                src != nullptr ? __half22float2(*reinterpret_cast<const __half2*>(src + n0 + 2 * i)) : make_float2(none, none);
        }
        asm volatile("bar.sync 5, %0;" ::"n"(L_EPI_WARPS * 32) : "memory");
        const float4* v_bias = reinterpret_cast<const float4*>(s_vec) + part * 16;
        const float4 *v_gamma = v_bias + L_BN / 4, *v_beta = v_gamma + L_BN / 4;
        int tile = 0;
        for (int rb = cluster_id; rb < tiles_m; rb += clusters, ++tile) {
            const int acc = tile & 1;
            const uint32_t acc_ph = (tile >> 1) & 1;
            const int row0 = rb * (2 * L_BM) + half * L_BM + quarter * 32;
            float2 x[32];
            if (has_residual && lane == 0 && rb + clusters < tiles_m) tma_prefetch_2d(&map_r, col0, row0 + clusters * (2 * L_BM));
            mbar_wait(&bars[LB_TFULL + acc], acc_ph, wctx, LB_TFULL + acc);
            tc_fence_after();
            {
                const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + acc * L_BN + part * 64;
                uint32_t r0[32], r1[32];
                tmem_ld32(t_row, r0);
                tmem_ld32(t_row + 32, r1);
                tc_wait_ld();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {                              // the accumulator has been read: hand it back to the leader's MMA warp
                    if (leader) mbar_arrive(&bars[LB_TEMPTY + acc]);
                    else remote_arrive_cta(map_to_rank(smem_u32(&bars[LB_TEMPTY + acc]), static_cast<uint32_t>(rank - 1)));
                }
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    x[i] = pk2(__uint_as_float(r0[2 * i]), __uint_as_float(r0[2 * i + 1]));
                    x[16 + i] = pk2(__uint_as_float(r1[2 * i]), __uint_as_float(r1[2 * i + 1]));
                }
            }
            if (has_residual) {
                mbar_wait(res_bar, static_cast<uint32_t>(tile & 1), wctx, LB_RES);
            } else {
                if (lane == 0) tma_store_wait_read();         // the slab's previous store has been read out
                __syncwarp();
            }
            // x = accumulator + bias + residual; mean and centred sum of squares over this thread's 64 columns
            float2 sum_a = pk2(0.f, 0.f), sum_b = pk2(0.f, 0.f);
#pragma unroll
            for (int g = 0; g < 8; ++g) {
                uint4 ru = make_uint4(0u, 0u, 0u, 0u);
                if (has_residual) ru = *reinterpret_cast<const uint4*>(slab_row + ((g ^ (lane & 7)) << 4));
                const __half2* rh = reinterpret_cast<const __half2*>(&ru);
#pragma unroll
                for (int j = 0; j < 4; j += 2) {
                    const float4 b = v_bias[2 * g + j / 2];
                    float2 &v0 = x[4 * g + j], &v1 = x[4 * g + j + 1];
                    v0 = add2(add2(v0, pk2(b.x, b.y)), __half22float2(rh[j]));
                    v1 = add2(add2(v1, pk2(b.z, b.w)), __half22float2(rh[j + 1]));
                    sum_a = add2(sum_a, v0);
                    sum_b = add2(sum_b, v1);
                }
            }
            sum_a = add2(sum_a, sum_b);
            const float mean_p = (sum_a.x + sum_a.y) * (1.0f / 64.0f);
            const float2 nm = pk2(-mean_p, -mean_p);
            float2 sq_a = pk2(0.f, 0.f), sq_b = pk2(0.f, 0.f);
#pragma unroll
            for (int i = 0; i < 32; i += 2) {
                const float2 da = add2(x[i], nm), db = add2(x[i + 1], nm);
                sq_a = fma2(da, da, sq_a);
                sq_b = fma2(db, db, sq_b);
            }
            sq_a = add2(sq_a, sq_b);
            // the four warps of these rows merge theirs, then warp `part` brings the block's result to column slice `part`
            float2* mine = local + acc * L_PARTS * L_BM + lrow;
            if (threadIdx.x == 0) mbar_arrive_expect_tx(&bars[LB_PART + acc], static_cast<uint32_t>(slices * L_BM * 8));
            mine[part * L_BM] = make_float2(mean_p, sq_a.x + sq_a.y);
            asm volatile("bar.sync %0, %1;" ::"r"(1 + quarter), "n"(L_PARTS * 32) : "memory");
            if (part < slices) {
                const float2 t = merge_parts<64>(mine, L_PARTS);
                const uint32_t to = static_cast<uint32_t>(2 * part + half);
                st_async_f32x2(map_to_rank(smem_u32(table + (acc * L_MAX_SLICES + slice) * L_BM + lrow), to), t.x, t.y,
                               map_to_rank(smem_u32(&bars[LB_PART + acc]), to));
            }
            mbar_wait_cluster(&bars[LB_PART + acc], acc_ph, wctx, LB_PART + acc);
            const float2 stat = merge_parts<L_BN>(table + acc * L_MAX_SLICES * L_BM + lrow, slices);
            const float rstd = 1.0f / sqrtf(stat.y * inv_n + eps);
            const float2 rstd2 = pk2(rstd, rstd), shift2 = pk2(-stat.x * rstd, -stat.x * rstd);
#pragma unroll
            for (int g = 0; g < 8; ++g) {
                uint32_t o[4];
#pragma unroll
                for (int j = 0; j < 4; j += 2) {
                    const float4 ga = v_gamma[2 * g + j / 2], be = v_beta[2 * g + j / 2];
                    const float2 y0 = fma2(fma2(x[4 * g + j], rstd2, shift2), pk2(ga.x, ga.y), pk2(be.x, be.y));
                    const float2 y1 = fma2(fma2(x[4 * g + j + 1], rstd2, shift2), pk2(ga.z, ga.w), pk2(be.z, be.w));
                    o[j] = pack_half2(y0.x, y0.y);
                    o[j + 1] = pack_half2(y1.x, y1.y);
                }
                *reinterpret_cast<uint4*>(slab_row + ((g ^ (lane & 7)) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
                if (row0 < m && !mute) {
                    tma_store_2d(&map_c, slab, col0, row0);           // rows beyond the matrix are clipped by the tensor map
                    tma_store_commit();
                }
                if (has_residual && rb + clusters < tiles_m) {
                    tma_store_wait_read();
                    request_residual(rb + clusters);
                }
            }
        }
        if (lane == 0) tma_store_wait_all();
    }
    // no block leaves while a peer may still write its table, signal one of its barriers, read its shared memory or write its tensor memory
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();
    if (warp == L_EPI_WARPS + 1) {
        tc_fence_after();
        tmem_dealloc_pair(tmem_base, L_TMEM_COLS);
    }
}

// How many clusters of 2 * slices blocks the GPU keeps resident at once (the SMs of a cluster lie in one processing cluster of the
// chip, so fewer than SMs / cluster size may fit: 74, 33, 22 and 15 of 2, 4, 6 and 8 blocks), cached per device and cluster size.
int resident_clusters(int slices, int* clusters) {
    static std::atomic<int> resident[64][L_MAX_SLICES + 1];      // host threads may race here, every one of them stores the same value
    int dev = 0;
    STOF_CUDA(cudaGetDevice(&dev));
    *clusters = (dev >= 0 && dev < 64) ? resident[dev][slices].load() : 0;
    if (*clusters != 0) return STOF_OK;
    STOF_CUDA(cudaFuncSetAttribute(gemm_ln_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(L_SMEM)));
    const int size = 2 * slices;
    LaunchConfig lc(dim3(static_cast<unsigned>((sm_count() / size) * size)), L_THREADS, L_SMEM, nullptr, static_cast<unsigned>(size));
    lc.cfg.attrs = &lc.attr[1];                          // the cluster dimension alone
    lc.cfg.numAttrs = 1;
    STOF_CUDA(cudaOccupancyMaxActiveClusters(clusters, gemm_ln_kernel, &lc.cfg));
    if (*clusters < 1) {
        set_error("gemm+layernorm: no cluster of %d thread blocks fits on this GPU", size);
        return STOF_E_LIMIT;
    }
    if (dev >= 0 && dev < 64) resident[dev][slices].store(*clusters);
    return STOF_OK;
}

// Beyond K = 2048: is one kernel faster than the GEMM followed by the LayerNorm kernel?  It saves the LayerNorm pass, but clusters of 6
// and 8 blocks leave 16 and 28 SMs idle and its rounds are of whole row blocks.  A 256 x 256 tile of a pair of blocks and a 128 x 256
// tile of one block take the same time per 64 of K, 0.4 us; a LayerNorm pass takes that long per 300,000 elements.  Measured with
// residual, one kernel / two: K = 3072, N = 768: 4096 rows 27.3 / 28.8 us (1 round / 1), 6144 44.1 / 31.9 (2 / 1), 8192 45.4 / 48.6
// (2 / 2), 32768 134 / 142 (6 / 6); K = 4096, N = 1024: 2816 rows 32.6 / 33.2 (1 / 1), 8192 79.4 / 65.8 (3 / 2), 32768 237 / 225 (9 / 7).
// Where the GEMM alone would run on small tiles it stays ahead: K = 3072, N = 768: 3072 rows 26.6 / 21.8.
// Up to K = 2048 it is one kernel whatever the time: two kernels round the sums to fp16 before the statistics, and rows with a common
// offset of 60 and a spread of 0.5 then come out 3.7e-2 off, against 2e-3 (K = N = 1024: 2048 rows 14.2 us against 12.4, 4096 rows 19.8
// against 19.1).  Beyond, two kernels have been the form of these shapes from the start.
bool one_kernel_wins(int m, int n, int k, bool residual, int clusters) {
    if (((m + 127LL) / 128) * ((n + 127LL) / 128) <= sm_count()) return false;
    const long long rounds = ((m + 255LL) / 256 + clusters - 1) / clusters;
    const long long extra = rounds - gemm_rounds(m, n, k, residual ? STOF_EPI_BIAS_RESIDUAL : STOF_EPI_BIAS);
    return extra * ((k + 63) / 64) * 300000 <= static_cast<long long>(m) * n;
}

}  // namespace
}  // namespace stof

using namespace stof;

// Declared in include/stof_b200.h.  Shapes that neither fused kernel covers (N not a multiple of 256, or beyond 1024), and those beyond
// K = 2048 that two kernels are faster for, run as the GEMM with the bias + residual epilogue followed by the row LayerNorm kernel in place.
// STOF_B200_GEMM_LN=fused / split overrides.
extern "C" int stof_gemm_bias_residual_layernorm(const void* a, long long lda, const void* w, long long ldw, const void* bias,
                                                 const void* residual, long long ldr, const void* gamma, const void* beta, float eps,
                                                 void* c, long long ldc, int m, int n, int k, int* status_dev, void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    STOF_REQUIRE(a && w && c, "gemm+layernorm: null operand");
    STOF_REQUIRE(m >= 0 && n > 0 && k > 0, "gemm+layernorm: bad shape m=%d n=%d k=%d", m, n, k);
    STOF_REQUIRE(n % 8 == 0 && k % 8 == 0, "gemm+layernorm: n=%d and k=%d must be multiples of 8", n, k);
    STOF_REQUIRE(lda % 8 == 0 && ldw % 8 == 0 && ldc % 8 == 0, "gemm+layernorm: leading dimensions must be multiples of 8 elements");
    STOF_REQUIRE(lda >= k && ldw >= n && ldc >= n, "gemm+layernorm: leading dimension smaller than the row length");
    STOF_REQUIRE(aligned16(a) && aligned16(w) && aligned16(c) && aligned16(bias) && aligned16(residual) && aligned16(gamma) && aligned16(beta),
                 "gemm+layernorm: pointers must be 16-byte aligned");
    STOF_REQUIRE(!residual || (ldr % 8 == 0 && ldr >= n), "gemm+layernorm: residual row stride must be a multiple of 8, >= n");
    if (m == 0) return STOF_OK;
    static const int mode = [] {
        const char* e = std::getenv("STOF_B200_GEMM_LN");
        return e == nullptr ? 0 : (e[0] == 'f' ? 1 : (e[0] == 's' ? 2 : 0));
    }();
    const int slices = n / L_BN;
    const bool covered = n % L_BN == 0 && slices <= L_MAX_SLICES && mode != 2;
    CUtensorMap mw;
    if (covered) {
        const uint64_t dims[2] = {static_cast<uint64_t>(n), static_cast<uint64_t>(k)};
        const uint64_t strides[1] = {static_cast<uint64_t>(ldw) * 2};
        const uint32_t box[2] = {64, L_BK};
        if (int rc = make_tensor_map_f16(&mw, w, 2, dims, strides, box)) return rc;
    }
    // few rows; beyond K = 2048 a row block's few thread blocks walk K longer than the split GEMM and a LayerNorm pass take
    if (covered && mode == 0 && k <= 2048) {
        int done = 0;
        const int rc = gemm_split_ln_dispatch({a, lda, &mw, static_cast<const __half*>(bias), static_cast<const __half*>(residual), ldr,
                                               static_cast<const __half*>(gamma), static_cast<const __half*>(beta), eps, static_cast<__half*>(c), ldc, m, n,
                                               k, status_dev, stream}, &done);
        if (rc != STOF_OK || done != 0) return rc;
    }
    int clusters = 0;
    if (covered)
        if (int rc = resident_clusters(slices, &clusters)) return rc;
    // (over A itself only in one kernel: nothing is written before all blocks of a row block have multiplied)
    if (!covered || (mode != 1 && k > 2048 && a != c && !one_kernel_wins(m, n, k, residual != nullptr, clusters))) {
        int rc = residual ? stof_gemm_bias_act(a, lda, w, ldw, bias, residual, ldr, c, ldc, m, n, k, STOF_EPI_BIAS_RESIDUAL, status_dev, stream_)
                          : stof_gemm_bias_act(a, lda, w, ldw, bias, nullptr, 0, c, ldc, m, n, k, STOF_EPI_BIAS, status_dev, stream_);
        if (rc != STOF_OK) return rc;
        return stof_bias_residual_layernorm(c, ldc, nullptr, nullptr, 0, gamma, beta, eps, c, ldc, m, n, status_dev, stream_);
    }
    CUtensorMap ma, mc, mr;
    {
        const uint64_t dims[2] = {static_cast<uint64_t>(k), static_cast<uint64_t>(m)};
        const uint64_t strides[1] = {static_cast<uint64_t>(lda) * 2};
        const uint32_t box[2] = {L_BK, L_BM};
        if (int rc = make_tensor_map_f16(&ma, a, 2, dims, strides, box)) return rc;
    }
    {
        const uint64_t dims[2] = {static_cast<uint64_t>(n), static_cast<uint64_t>(m)};
        const uint64_t strides[1] = {static_cast<uint64_t>(ldc) * 2};
        const uint32_t box[2] = {64, 32};
        if (int rc = make_tensor_map_f16(&mc, c, 2, dims, strides, box)) return rc;
    }
    if (residual != nullptr) {
        const uint64_t dims[2] = {static_cast<uint64_t>(n), static_cast<uint64_t>(m)};
        const uint64_t strides[1] = {static_cast<uint64_t>(ldr) * 2};
        const uint32_t box[2] = {64, 32};
        if (int rc = make_tensor_map_f16(&mr, residual, 2, dims, strides, box)) return rc;
    } else {
        mr = mc;                                     // never read
    }
    const int tiles_m = (m + 2 * L_BM - 1) / (2 * L_BM), size = 2 * slices;
    if (clusters > tiles_m) clusters = tiles_m;
    LaunchConfig lc(dim3(static_cast<unsigned>(clusters * size)), L_THREADS, L_SMEM, stream, static_cast<unsigned>(size));
    STOF_CUDA(cudaLaunchKernelEx(&lc.cfg, gemm_ln_kernel, ma, mw, mc, mr, static_cast<const __half*>(bias), residual != nullptr ? 1 : 0,
                                 static_cast<const __half*>(gamma), static_cast<const __half*>(beta), eps, m, n, k, slices, status_dev));
    return STOF_OK;
}
