// C[M,N] = epilogue(A[M,K] @ W[K,N] + bias) for shapes with few output tiles: small tiles, and the contraction of a tile cut
// over the thread blocks of a cluster.
//
// At a few hundred rows the 128 x 256 tiles of the one-block kernel leave most of the GPU idle (128 rows x 768 columns: three
// tiles) and each of the few thread blocks then walks all of K alone: 48 steps of 64 at K = 3072, 22 us.  What a launch of this
// size takes is latency - getting started, the first tile's way from HBM, the last tile's way out - so this kernel is made for it:
//   * tiles of 64 x 64, 128 x 64 or 128 x 128, one per thread block, K cut over a cluster of S = 1, 2 or 4 blocks
//   * nearly all of a block's operands in flight at once (up to 192 KB of stages of 128 along K; a stage of 64 spent more time
//     asking whether it had landed, some 180 cycles, than multiplying)
//   * the kernel starts under the tail of the one before it, and has its weight tiles brought into L2 ahead of the dependency wait
//   * a short epilogue (gemm_split.cuh)
//   warps 0-3 (0-7 at BN = 128)   epilogue
//   the warp after them           TMA producer
//   the last one                  MMA issuer: tcgen05.mma BM x BN x 16 into a BN-column fp32 accumulator in tensor memory
// Epilogue, one row and 64 columns per thread (a 64-row accumulator lies in the lower 16 lanes of each quarter of tensor memory):
//               S = 1: tensor memory -> bias, activation or residual -> fp16 -> global
//               S > 1: tensor memory -> fp32 partial tile in shared memory (over the stages, idle by then).  Block r of the cluster
//               finishes rows r * BM / S ..: every block sends each peer that peer's rows with one bulk copy into the peer's
//               receive buffer, which reports to the peer's barrier (reading them there with loads took 1300 - 3200 cycles, and
//               two more cluster barriers).  No atomics, no workspace in global memory, and the order of the sum is fixed.
// Measured (weights from HBM, back to back, against the one-block kernel): 128 rows 768 -> 768 columns 8.1 -> 3.6 us, 768 -> 3072
// 8.4 -> 4.0 us, 3072 -> 768 19.9 -> 5.9 us; more beside the dispatch in gemm_tc.cu.
#include <atomic>
#include "gemm_split.cuh"
#include "stof_epilogue.cuh"

namespace stof {
namespace {

template <int BM, int BN>
struct SplitSmem {
    using Shape = SplitShape<BM, BN>;
    static constexpr int PITCH = BN + 4;                            // floats per row of the partial tile: 16 bytes off a power of two
    static constexpr int PARTIAL_BYTES = BM * PITCH * 4;
    // stages or partial tile | the peers' parts of this block's rows | residual | bias | barriers
    __host__ __device__ static int received_at(int stages) {
        return stages * Shape::STAGE_BYTES > PARTIAL_BYTES ? stages * Shape::STAGE_BYTES : PARTIAL_BYTES;
    }
    __host__ __device__ static int part_bytes(int split) { return BM / split * PITCH * 4; }       // one peer's part
    __host__ __device__ static int residual_at(int stages, int split) { return received_at(stages) + (split - 1) * part_bytes(split); }
    __host__ __device__ static int bias_at(int stages, int split, bool residual) { return residual_at(stages, split) + (residual ? Shape::RESIDUAL_BYTES : 0); }
    __host__ __device__ static int bars_at(int stages, int split, bool residual) { return bias_at(stages, split, residual) + BN * 2; }
    static size_t bytes(int stages, int split, bool residual) { return 1024 + static_cast<size_t>(bars_at(stages, split, residual)) + S_BAR_BYTES; }
    static int stages(int steps, int split, bool residual) {
        int n = steps < Shape::MAX_STAGES ? steps : Shape::MAX_STAGES;
        while (n > 1 && bytes(n, split, residual) > S_SMEM_LIMIT) --n;
        return n;
    }
};

// bias and activation or residual on 8 columns, packed to fp16
template <int EPI>
__device__ __forceinline__ uint4 finish8(float2 (&v)[4], const uint4& bias, const uint4& residual) {
    const __half2 *bh = reinterpret_cast<const __half2*>(&bias), *rh = reinterpret_cast<const __half2*>(&residual);
    uint32_t o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        v[j] = add2(v[j], __half22float2(bh[j]));
        if (EPI == STOF_EPI_BIAS_GELU_ERF) v[j] = gelu_erf2(v[j]);
        else if (EPI == STOF_EPI_BIAS_GELU_TANH) v[j] = gelu_tanh2(v[j]);
        else if (EPI == STOF_EPI_BIAS_RELU) v[j] = make_float2(fmaxf(v[j].x, 0.0f), fmaxf(v[j].y, 0.0f));
        else if (EPI == STOF_EPI_BIAS_RESIDUAL) v[j] = add2(v[j], __half22float2(rh[j]));
        o[j] = pack_half2(v[j].x, v[j].y);
    }
    return make_uint4(o[0], o[1], o[2], o[3]);
}

template <int EPI, int BM, int BN>
__global__ void __launch_bounds__(SplitShape<BM, BN>::THREADS, 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, const __half* bias,
                  const __half* residual, long long ldr, __half* c, long long ldc, int m, int n, int k, int split, int stages, int* status) {
    using Shape = SplitShape<BM, BN>;
    using Smem = SplitSmem<BM, BN>;
    constexpr bool RES = EPI == STOF_EPI_BIAS_RESIDUAL;
    constexpr int EPI_WARPS = Shape::EPI_WARPS;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    unsigned char *s_res = smem + Smem::residual_at(stages, split), *s_bias = smem + Smem::bias_at(stages, split, RES);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Smem::bars_at(stages, split, RES));
    uint64_t *full = bars, *empty = bars + Shape::MAX_STAGES, *tfull = bars + 2 * Shape::MAX_STAGES, *received = tfull + 1;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(received + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = split > 1 ? static_cast<int>(cluster_rank()) : 0;
    const int tile = blockIdx.x / split;
    // neighbouring tiles walk down the rows of one weight column block first: they share its weight tiles
    const int tiles_m = (m + BM - 1) / BM;
    const int m0 = (tile % tiles_m) * BM, n0 = (tile / tiles_m) * BN;
    const int kblocks = (k + S_BK - 1) / S_BK;
    const int kb0 = kblocks * rank / split, kb1 = kblocks * (rank + 1) / split;
    const WaitCtx wctx{abort_flag, status};

    if (warp == EPI_WARPS + 1) {
        tmem_alloc(tmem_slot, BN);
        tmem_relinquish();
    } else if (warp == EPI_WARPS) {
        if (elect_one()) split_prefetch<BN>(map_a, map_w, n0, kb0, kb1, stages);
    } else if (threadIdx.x == 0) {
        *abort_flag = 0;
        for (int i = 0; i < stages; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        mbar_init(tfull, 1);
        mbar_init(received, 1);
        fence_mbar_init();
        if (split > 1) mbar_arrive_expect_tx(received, static_cast<uint32_t>((split - 1) * Smem::part_bytes(split)));
    }
    tc_fence_before();
    if (split > 1) {
        __syncwarp();
        cluster_sync_all();                      // every block's barriers exist before a peer's copy reports to them
    } else {
        __syncthreads();
    }
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == EPI_WARPS) {
        split_produce<Shape, BN>(map_a, map_w, smem, full, empty, m0, n0, kb0, kb1, stages, wctx);
    } else if (warp == EPI_WARPS + 1) {
        split_multiply<Shape, BM, BN>(smem, full, empty, tfull, tmem_base, kb0, kb1, stages, wctx);
    } else {
        grid_dependency_wait();
        const int rows = BM / split, row_lo = rank * rows;        // the rows this block finishes
        stage_vector(s_bias, bias != nullptr ? bias + n0 : nullptr, n - n0, BN, 0u, 0);
        if (RES) stage_residual<Shape>(s_res, residual, ldr, m0, n0, m, n, row_lo, rows);
        const bool mute = failure_reported(status);
        copy_async_wait();
        epilogue_barrier<Shape::EPI_THREADS>();
        const int quarter = warp & 3, part = warp >> 2;
        const bool mine = BM == 128 || lane < 16;
        const int lrow = BM == 128 ? quarter * 32 + lane : quarter * 16 + (lane & 15);
        const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + part * 64;
        mbar_wait_addr(smem_u32(tfull), 0, wctx, 2 * stages);
        tc_fence_after();
        if (split == 1) {
            const int row = m0 + lrow;
            const bool live = mine && row < m && !mute;
            __half* out = c + static_cast<size_t>(row) * ldc + n0;
#pragma unroll 1
            for (int g0 = part * 8; g0 < part * 8 + 8; g0 += 2) {
                uint32_t r[16];
                tmem_ld16(t_row + (g0 & 7) * 8, r);
                tc_wait_ld();
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int g = g0 + h;
                    float2 v[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) v[j] = pk2(__uint_as_float(r[8 * h + 2 * j]), __uint_as_float(r[8 * h + 2 * j + 1]));
                    uint4 res = make_uint4(0u, 0u, 0u, 0u);
                    if (RES) res = *reinterpret_cast<const uint4*>(s_res + Shape::residual_at(lrow, g));
                    const uint4 o = finish8<EPI>(v, reinterpret_cast<const uint4*>(s_bias)[g], res);
                    if (live && n0 + 8 * g < n) *reinterpret_cast<uint4*>(out + 8 * g) = o;
                }
            }
        } else {
            // a row of the partial tile, 16 bytes at a time; the pitch keeps eight lanes on different banks
            float* own = reinterpret_cast<float*>(smem);
            float* prow = own + lrow * Smem::PITCH + part * 64;
#pragma unroll 1
            for (int c0 = 0; c0 < 64; c0 += 16) {
                uint32_t r[16];
                tmem_ld16(t_row + c0, r);
                tc_wait_ld();
                if (mine)
#pragma unroll
                    for (int i = 0; i < 4; ++i) *reinterpret_cast<uint4*>(prow + c0 + 4 * i) = make_uint4(r[4 * i], r[4 * i + 1], r[4 * i + 2], r[4 * i + 3]);
            }
            const float* parts = reinterpret_cast<const float*>(smem + Smem::received_at(stages));
            const int part_floats = Smem::part_bytes(split) / 4;
            fence_proxy_async_smem();
            epilogue_barrier<Shape::EPI_THREADS>();                  // the partial tile is written
            if (static_cast<int>(threadIdx.x) < split && static_cast<int>(threadIdx.x) != rank) {
                // this block's part comes at place `rank`, or rank - 1 behind the receiver's own
                const int to = static_cast<int>(threadIdx.x), place = rank < to ? rank : rank - 1;
                bulk_copy_to_peer(map_to_rank(smem_u32(parts + place * part_floats), static_cast<uint32_t>(to)), smem_u32(own + to * part_floats),
                                  static_cast<uint32_t>(Smem::part_bytes(split)), map_to_rank(smem_u32(received), static_cast<uint32_t>(to)));
            }
            __syncwarp();
            mbar_wait_addr(smem_u32(received), 0, wctx, 2 * stages + 1);
            // output pieces of 8 columns, eight or sixteen neighbouring threads to a row
#pragma unroll 1
            for (int i = threadIdx.x; i < rows * Shape::CHUNKS; i += Shape::EPI_THREADS) {
                const int lr = i / Shape::CHUNKS, g = i % Shape::CHUNKS, row = m0 + row_lo + lr;
                const int at = lr * Smem::PITCH + 8 * g;
                float2 v[4] = {};
#pragma unroll 1
                for (int p = 0; p < split; ++p) {
                    const float* from = (p == rank ? own + rank * part_floats : parts + (p < rank ? p : p - 1) * part_floats) + at;
                    const float4 x = *reinterpret_cast<const float4*>(from), y = *reinterpret_cast<const float4*>(from + 4);
                    v[0] = add2(v[0], pk2(x.x, x.y));
                    v[1] = add2(v[1], pk2(x.z, x.w));
                    v[2] = add2(v[2], pk2(y.x, y.y));
                    v[3] = add2(v[3], pk2(y.z, y.w));
                }
                uint4 res = make_uint4(0u, 0u, 0u, 0u);
                if (RES) res = *reinterpret_cast<const uint4*>(s_res + Shape::residual_at(row_lo + lr, g));
                const uint4 o = finish8<EPI>(v, reinterpret_cast<const uint4*>(s_bias)[g], res);
                if (row < m && n0 + 8 * g < n && !mute) *reinterpret_cast<uint4*>(c + static_cast<size_t>(row) * ldc + n0 + 8 * g) = o;
            }
        }
    }
    tc_fence_before();
    // A block has waited for all that its peers send it, but a peer may still be reading out what this one sends from here
    if (split > 1) {
        __syncwarp();
        cluster_sync_relaxed();
    } else {
        __syncthreads();
    }
    tc_fence_after();
    if (warp == EPI_WARPS + 1) tmem_dealloc(tmem_base, BN);
}

template <int EPI, int BM, int BN>
int launch_split(const SplitCall& x) {
    using Smem = SplitSmem<BM, BN>;
    constexpr bool RES = EPI == STOF_EPI_BIAS_RESIDUAL;
    static std::atomic<bool> configured[64];     // per device; host threads may race here, every one of them stores the same value
    int dev = 0;
    STOF_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        STOF_CUDA(cudaFuncSetAttribute(gemm_split_kernel<EPI, BM, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, S_SMEM_LIMIT));
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    CUtensorMap ma;
    if (int rc = split_map_a<BM>(&ma, x.a, x.lda, x.m, x.k)) return rc;
    const int tiles = ((x.m + BM - 1) / BM) * ((x.n + BN - 1) / BN);
    const int steps = ((x.k + S_BK - 1) / S_BK + x.split - 1) / x.split;
    const int stages = Smem::stages(steps, x.split, RES);
    LaunchConfig lc(dim3(static_cast<unsigned>(tiles * x.split)), SplitShape<BM, BN>::THREADS, Smem::bytes(stages, x.split, RES), x.stream,
                    static_cast<unsigned>(x.split));
    STOF_CUDA(cudaLaunchKernelEx(&lc.cfg, gemm_split_kernel<EPI, BM, BN>, ma, *x.map_w, x.bias, x.residual, x.ldr, x.c, x.ldc, x.m, x.n, x.k, x.split,
                                 stages, x.status));
    return STOF_OK;
}

template <int BM, int BN>
int dispatch_split(const SplitCall& x) {
    switch (x.epilogue) {
        case STOF_EPI_BIAS: return launch_split<STOF_EPI_BIAS, BM, BN>(x);
        case STOF_EPI_BIAS_GELU_ERF: return launch_split<STOF_EPI_BIAS_GELU_ERF, BM, BN>(x);
        case STOF_EPI_BIAS_GELU_TANH: return launch_split<STOF_EPI_BIAS_GELU_TANH, BM, BN>(x);
        case STOF_EPI_BIAS_RELU: return launch_split<STOF_EPI_BIAS_RELU, BM, BN>(x);
        default: return launch_split<STOF_EPI_BIAS_RESIDUAL, BM, BN>(x);
    }
}

}  // namespace

int gemm_split_dispatch(const SplitCall& x, int bm, int bn) {
    if (bm == 64) return dispatch_split<64, 64>(x);
    if (bn == 64) return dispatch_split<128, 64>(x);
    return dispatch_split<128, 128>(x);
}

}  // namespace stof
