// C[M,N] = epilogue(A[M,K] @ W[K,N] + bias) on the sm_100a tensor cores (tcgen05 + TMEM + TMA).
//
// Persistent kernel, one thread block per SM, 128 x 256 output tiles, K in steps of 64:
//   warp 8      TMA producer: A tile (128 rows x 64 k, K-major) and four 64 x 64 W boxes (k rows x 64 n,
//               i.e. N-major as the weights lie in memory) per stage, 4 stages of 48 KB
//   warp 9      MMA issuer: 4 tcgen05.mma (128 x 256 x 16) per stage into one of two 256-column fp32
//               accumulators in tensor memory; tcgen05.commit releases the stage / publishes the tile
//   warps 0-7   epilogue: tcgen05.ld 64 columns at a time, + bias, optional GELU (erf or tanh form, evaluated on
//               packed fp32 pairs) or + residual (prefetched into registers before the accumulator is ready),
//               fp16 pack into a swizzled shared-memory slab, TMA store; runs under the next tile's main loop
// Weights are consumed in their (K, N) row-major layout through an MN-major shared-memory
// descriptor, so no transposed copy is ever made.
#include <cstdlib>
#include <atomic>
#include "gemm_split.h"
#include "stof_ptx.cuh"
#include "stof_epilogue.cuh"

namespace stof {
namespace {

constexpr int G_BM = 128, G_BN = 256, G_BK = 64;
constexpr int G_STAGES = 4;
constexpr int G_A_BYTES = G_BM * G_BK * 2;            // 16 KB
constexpr int G_B_BYTES = G_BK * G_BN * 2;            // 32 KB
constexpr int G_STAGE_BYTES = G_A_BYTES + G_B_BYTES;  // 48 KB
constexpr int G_EPI_WARPS = 8;
constexpr int G_THREADS = (G_EPI_WARPS + 2) * 32;
constexpr int G_TMEM_COLS = 512;
constexpr int G_SLAB_BYTES = 32 * 64 * 2;                // per epilogue warp: 32 rows x 64 columns of fp16 (TMA store source)
constexpr size_t G_SMEM = 1024 + static_cast<size_t>(G_STAGES) * G_STAGE_BYTES + G_EPI_WARPS * G_SLAB_BYTES + 256;

enum { BAR_FULL = 0, BAR_EMPTY = G_STAGES, BAR_TFULL = 2 * G_STAGES, BAR_TEMPTY = 2 * G_STAGES + 2, BAR_COUNT = 2 * G_STAGES + 4 };

template <int EPI>
__global__ void __launch_bounds__(G_THREADS, 1)
gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_c,
            const __half* bias, const __half* residual, long long ldr, int m, int n, int k, int* status) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    unsigned char* slabs = smem + G_STAGES * G_STAGE_BYTES;          // one 4 KB slab per epilogue warp, 1024-aligned
    uint64_t* bars = reinterpret_cast<uint64_t*>(slabs + G_EPI_WARPS * G_SLAB_BYTES);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + BAR_COUNT);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tiles_n = (n + G_BN - 1) / G_BN, tiles_m = (m + G_BM - 1) / G_BM;
    const int num_tiles = tiles_m * tiles_n;
    const int kblocks = (k + G_BK - 1) / G_BK;
    const WaitCtx wctx{abort_flag, status};

    if (threadIdx.x == 0) {
        *abort_flag = 0;
        for (int i = 0; i < G_STAGES; ++i) {
            mbar_init(&bars[BAR_FULL + i], 1);
            mbar_init(&bars[BAR_EMPTY + i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&bars[BAR_TFULL + i], 1);
            mbar_init(&bars[BAR_TEMPTY + i], G_EPI_WARPS);
        }
        fence_mbar_init();
    }
    if (warp == G_EPI_WARPS + 1) {
        tmem_alloc(tmem_slot, G_TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    grid_dependency_wait();
    grid_launch_dependents();

    if (warp == G_EPI_WARPS) {
        // ------------------------------------------------------------------ TMA producer
        if (elect_one()) {
            tma_prefetch_desc(&map_a);
            tma_prefetch_desc(&map_w);
            int it = 0;
            for (int t = blockIdx.x; t < num_tiles; t += gridDim.x) {
                const int m0 = (t / tiles_n) * G_BM, n0 = (t % tiles_n) * G_BN;
                for (int kb = 0; kb < kblocks; ++kb, ++it) {
                    const int s = it % G_STAGES;
                    const uint32_t ph = (it / G_STAGES) & 1;
                    mbar_wait(&bars[BAR_EMPTY + s], ph ^ 1, wctx, BAR_EMPTY + s);
                    unsigned char* a_dst = smem + s * G_STAGE_BYTES;
                    unsigned char* b_dst = a_dst + G_A_BYTES;
                    mbar_arrive_expect_tx(&bars[BAR_FULL + s], G_STAGE_BYTES);
                    tma_load_2d(a_dst, &map_a, &bars[BAR_FULL + s], kb * G_BK, m0);
#pragma unroll
                    for (int j = 0; j < G_BN / 64; ++j)
                        tma_load_2d(b_dst + j * (G_BK * 64 * 2), &map_w, &bars[BAR_FULL + s], n0 + 64 * j, kb * G_BK);
                }
            }
        }
    } else if (warp == G_EPI_WARPS + 1) {
        // ------------------------------------------------------------------ MMA issuer
        if (elect_one()) {
            constexpr uint32_t idesc = make_idesc_f16(G_BM, G_BN, /*b_mn_major=*/true);
            int it = 0, local = 0;
            for (int t = blockIdx.x; t < num_tiles; t += gridDim.x, ++local) {
                const int acc = local & 1;
                const uint32_t acc_ph = (local >> 1) & 1;
                mbar_wait(&bars[BAR_TEMPTY + acc], acc_ph ^ 1, wctx, BAR_TEMPTY + acc);
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + acc * G_BN;
                for (int kb = 0; kb < kblocks; ++kb, ++it) {
                    const int s = it % G_STAGES;
                    const uint32_t ph = (it / G_STAGES) & 1;
                    mbar_wait(&bars[BAR_FULL + s], ph, wctx, BAR_FULL + s);
                    tc_fence_after();
                    const uint32_t a_addr = smem_u32(smem + s * G_STAGE_BYTES);
                    const uint32_t b_addr = a_addr + G_A_BYTES;
#pragma unroll
                    for (int kk = 0; kk < G_BK / 16; ++kk) {
                        const uint64_t a_desc = make_smem_desc_sw128(a_addr + kk * 32, 16, 1024);
                        const uint64_t b_desc = make_smem_desc_sw128(b_addr + kk * 2048, G_BK * 64 * 2, 1024);
                        mma_f16_ss(d_tmem, a_desc, b_desc, idesc, (kb > 0 || kk > 0) ? 1u : 0u);
                    }
                    tc_commit(&bars[BAR_EMPTY + s]);
                }
                tc_commit(&bars[BAR_TFULL + acc]);
            }
        }
    } else {
        // ------------------------------------------------------------------ epilogue
        const int quarter = warp & 3, half_n = warp >> 2;
        unsigned char* slab = slabs + warp * G_SLAB_BYTES;
        const bool mute = failure_reported(status);
        int local = 0;
        for (int t = blockIdx.x; t < num_tiles; t += gridDim.x, ++local) {
            const int acc = local & 1;
            const uint32_t acc_ph = (local >> 1) & 1;
            const int m0 = (t / tiles_n) * G_BM, n0 = (t % tiles_n) * G_BN;
            const int row0 = m0 + quarter * 32;
            const int row = row0 + lane;
            const int colbase = n0 + half_n * (G_BN / 2);
            // the residual does not depend on the accumulator: its loads are in flight while the tile's MMAs finish
            uint4 res[2][8];
            if (EPI == STOF_EPI_BIAS_RESIDUAL) {
#pragma unroll
                for (int ch = 0; ch < 2; ++ch)
#pragma unroll
                    for (int g = 0; g < 8; ++g) {
                        const int col = colbase + ch * 64 + g * 8;
                        res[ch][g] = (row < m && col < n) ? __ldca(reinterpret_cast<const uint4*>(residual + static_cast<size_t>(row) * ldr + col))
                                                          : make_uint4(0u, 0u, 0u, 0u);
                    }
            }
            mbar_wait(&bars[BAR_TFULL + acc], acc_ph, wctx, BAR_TFULL + acc);
            tc_fence_after();
            const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + acc * G_BN + half_n * (G_BN / 2);
#pragma unroll
            for (int ch = 0; ch < 2; ++ch) {
                // requested ahead of the accumulator: coherent loads stay where they stand, and each would be waited for below (8192 x 3072,
                // K = 768, GELU: 35.4 us there, 30.6 here; the residual form spills 96 bytes by it, at the same time)
                uint4 bu[8];
#pragma unroll
                for (int g = 0; g < 8; ++g) {
                    const int col = colbase + ch * 64 + 8 * g;
                    bu[g] = bias != nullptr && col < n ? __ldca(reinterpret_cast<const uint4*>(bias + col)) : make_uint4(0u, 0u, 0u, 0u);
                }
                uint32_t r0[32], r1[32];
                tmem_ld32(t_row + ch * 64, r0);
                tmem_ld32(t_row + ch * 64 + 32, r1);
                tc_wait_ld();
                if (ch == 1) {
                    // both chunks of this accumulator half are in registers: hand the accumulator back to the MMA warp
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&bars[BAR_TEMPTY + acc]);
                }
                const int col0 = colbase + ch * 64;
                if (col0 < n && row0 < m) {
                    if (lane == 0) tma_store_wait_read();             // the slab's previous store has been read out
                    __syncwarp();
#pragma unroll
                    for (int g = 0; g < 8; ++g) {                     // 8 columns = one 16-byte chunk of the output row
                        const uint32_t* src = (g < 4) ? &r0[8 * g] : &r1[8 * (g - 4)];
                        float2 v[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j) v[j] = pk2(__uint_as_float(src[2 * j]), __uint_as_float(src[2 * j + 1]));
                        if (bias != nullptr) {
                            const __half2* bh = reinterpret_cast<const __half2*>(&bu[g]);
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                const float2 f = __half22float2(bh[j]);
                                v[j] = add2(v[j], pk2(f.x, f.y));
                            }
                        }
                        if (EPI == STOF_EPI_BIAS_GELU_ERF) {
#pragma unroll
                            for (int j = 0; j < 4; ++j) v[j] = gelu_erf2(v[j]);
                        } else if (EPI == STOF_EPI_BIAS_GELU_TANH) {
#pragma unroll
                            for (int j = 0; j < 4; ++j) v[j] = gelu_tanh2(v[j]);
                        } else if (EPI == STOF_EPI_BIAS_RELU) {
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                float x0, x1;
                                upk2(v[j], x0, x1);
                                v[j] = pk2(fmaxf(x0, 0.0f), fmaxf(x1, 0.0f));
                            }
                        } else if (EPI == STOF_EPI_BIAS_RESIDUAL) {
                            const __half2* rh = reinterpret_cast<const __half2*>(&res[ch][g]);
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                const float2 f = __half22float2(rh[j]);
                                v[j] = add2(v[j], pk2(f.x, f.y));
                            }
                        }
                        uint4 o;
                        float lo, hi;
                        upk2(v[0], lo, hi); o.x = pack_half2(lo, hi);
                        upk2(v[1], lo, hi); o.y = pack_half2(lo, hi);
                        upk2(v[2], lo, hi); o.z = pack_half2(lo, hi);
                        upk2(v[3], lo, hi); o.w = pack_half2(lo, hi);
                        *reinterpret_cast<uint4*>(slab + lane * 128 + ((g ^ (lane & 7)) << 4)) = o;
                    }
                    fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0 && !mute) {
                        tma_store_2d(&map_c, slab, col0, row0);       // rows / columns beyond the matrix are clipped by the tensor map
                        tma_store_commit();
                    }
                }
            }
        }
        if (lane == 0) tma_store_wait_all();
    }
    tc_fence_before();
    __syncthreads();
    if (warp == G_EPI_WARPS + 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, G_TMEM_COLS);
    }
}

template <int EPI>
int launch(const CUtensorMap& ma, const CUtensorMap& mw, const CUtensorMap& mc, const __half* bias, const __half* residual, long long ldr,
           int m, int n, int k, int* status, cudaStream_t stream) {
    static std::atomic<bool> configured[64];     // per device; host threads may race here, every one of them stores the same value
    int dev = 0;
    STOF_CUDA(cudaGetDevice(&dev));
    if (dev >= 0 && dev < 64 && !configured[dev]) {
        STOF_CUDA(cudaFuncSetAttribute(gemm_kernel<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(G_SMEM)));
        configured[dev] = true;
    }
    const int tiles = ((m + G_BM - 1) / G_BM) * ((n + G_BN - 1) / G_BN);
    int grid = sm_count();
    if (grid > tiles) grid = tiles;
    LaunchConfig lc(dim3(static_cast<unsigned>(grid)), G_THREADS, G_SMEM, stream);
    STOF_CUDA(cudaLaunchKernelEx(&lc.cfg, gemm_kernel<EPI>, ma, mw, mc, bias, residual, ldr, m, n, k, status));
    return STOF_OK;
}

}  // namespace

// the two-block (cta_group::2) kernel, gemm_pair.cu
int gemm_pair_dispatch(const CUtensorMap& ma, const CUtensorMap& mw, const CUtensorMap& mc, const __half* bias, const __half* residual,
                       long long ldr, int m, int n, int k, int epilogue, int* status, cudaStream_t stream);
namespace {
// 0 = one-block kernel, 1 = two-block kernel, -1 = by shape.  STOF_B200_GEMM_PAIR overrides (read once).
int pair_mode() {
    static const int mode = [] {
        const char* e = std::getenv("STOF_B200_GEMM_PAIR");
        return (e != nullptr && (e[0] == '0' || e[0] == '1')) ? e[0] - '0' : -1;
    }();
    return mode;
}
// Pairs of blocks on 256 x 256 tiles once every pair of SMs gets at least two of them; small problems keep 128 x 256 tiles.
// The residual epilogue at K <= 1024 outlasts the main loop in both kernels; measured per shape (K = N = 1024 and 768,
// bias + residual): 16384 rows one-block +3 %, 65536 rows equal within 1.5 %, 262144 rows two-block +3 % - so that case
// moves to the two-block kernel only from 16 tiles per pair of SMs on.
bool takes_pairs(int m, int n, int k, int epilogue) {
    const int mode = pair_mode();
    if (mode >= 0) return mode == 1;
    const long long tiles256 = ((m + 255LL) / 256) * ((n + 255LL) / 256), pairs = sm_count() / 2;
    const bool short_residual = epilogue == STOF_EPI_BIAS_RESIDUAL && k <= 1024;
    return tiles256 >= (short_residual ? 16LL : 2LL) * pairs;
}

bool overlap(const void* p, long long p_bytes, const void* q, long long q_bytes) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(p), b = reinterpret_cast<uintptr_t>(q);
    return a < b + static_cast<uintptr_t>(q_bytes) && b < a + static_cast<uintptr_t>(p_bytes);
}
}  // namespace

// Tiles of 256 columns that the busiest multiprocessor (or pair) walks in the GEMM kernel that a shape gets, small tiles apart
long long gemm_rounds(int m, int n, int k, int epilogue) {
    const bool pairs = takes_pairs(m, n, k, epilogue);
    const long long rows = pairs ? 256 : 128, workers = pairs ? sm_count() / 2 : sm_count();
    return (((m + rows - 1) / rows) * ((n + 255LL) / 256) + workers - 1) / workers;
}
}  // namespace stof

using namespace stof;

extern "C" int stof_gemm_bias_act(const void* a, long long lda, const void* w, long long ldw, const void* bias, const void* residual,
                                  long long ldr, void* c, long long ldc, int m, int n, int k, int epilogue, int* status_dev,
                                  void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    STOF_REQUIRE(a && w && c, "gemm: null operand");
    STOF_REQUIRE(m >= 0 && n > 0 && k > 0, "gemm: bad shape m=%d n=%d k=%d", m, n, k);
    STOF_REQUIRE(n % 8 == 0 && k % 8 == 0, "gemm: n=%d and k=%d must be multiples of 8", n, k);
    STOF_REQUIRE(lda % 8 == 0 && ldw % 8 == 0 && ldc % 8 == 0, "gemm: leading dimensions must be multiples of 8 elements");
    STOF_REQUIRE(lda >= k && ldw >= n && ldc >= n, "gemm: leading dimension smaller than the row length");
    STOF_REQUIRE(aligned16(a) && aligned16(w) && aligned16(c) && aligned16(bias) && aligned16(residual), "gemm: pointers must be 16-byte aligned");
    STOF_REQUIRE(epilogue >= STOF_EPI_BIAS && epilogue <= STOF_EPI_BIAS_RELU, "gemm: unknown epilogue %d", epilogue);
    if (epilogue == STOF_EPI_BIAS_RESIDUAL)
        STOF_REQUIRE(residual && ldr % 8 == 0 && ldr >= n, "gemm: residual epilogue needs a residual with a row stride multiple of 8, >= n");
    if (m == 0) return STOF_OK;

    CUtensorMap ma, mw;
    {
        const uint64_t dims[2] = {static_cast<uint64_t>(k), static_cast<uint64_t>(m)};
        const uint64_t strides[1] = {static_cast<uint64_t>(lda) * 2};
        const uint32_t box[2] = {G_BK, G_BM};
        if (int rc = make_tensor_map_f16(&ma, a, 2, dims, strides, box)) return rc;
    }
    {
        const uint64_t dims[2] = {static_cast<uint64_t>(n), static_cast<uint64_t>(k)};
        const uint64_t strides[1] = {static_cast<uint64_t>(ldw) * 2};
        const uint32_t box[2] = {64, G_BK};
        if (int rc = make_tensor_map_f16(&mw, w, 2, dims, strides, box)) return rc;
    }
    const __half *bp = static_cast<const __half*>(bias), *rp = static_cast<const __half*>(residual);
    if (pair_mode() < 0) {
        // Few tiles: the smallest tiles that still all run at once, with K cut in two or four where it is long and that still fits
        // (gemm_split.cu; a second wave of these one-tile blocks costs more than the 128 x 256 tiles of the kernel below).
        // Measured, weights from HBM, this kernel against the 128 x 256 one: K = 768: 128 rows x 768 columns 64 x 64 3.6 / 8.1 us,
        // 512 x 2304 128 x 64 5.1 / 8.2, 1000 x 2304 128 x 128 7.1 / 8.2, 512 x 3072 128 x 128 6.8 / 8.3; K = 3072, 768 columns:
        // 128 rows 64 x 64 in two parts 5.9 / 19.9, 512 rows 64 x 64 8.1 / 19.7, 1000 rows 128 x 64 10.6 / 19.5.
        // C over A is sound where one block reads a row of A and writes it, after its last product: with tiles as wide as the matrix.
        // (Up to 256 columns the kernel below has such tiles.)
        const bool over_a = overlap(a, ((m - 1LL) * lda + k) * 2, c, ((m - 1LL) * ldc + n) * 2);
        const int sms = sm_count();
        constexpr int SHAPES[3][2] = {{64, 64}, {128, 64}, {128, 128}};
        for (const auto& t : SHAPES) {
            const long long tiles = static_cast<long long>((m + t[0] - 1) / t[0]) * ((n + t[1] - 1) / t[1]);
            if (tiles > sms) continue;
            if (over_a && n > t[1]) continue;
            int split = 1;
            if (k >= 2048 && 2 * tiles <= sms) split = 2;
            if (k >= 4096 && 4 * tiles <= sms) split = 4;
            return gemm_split_dispatch({a, lda, &mw, bp, rp, ldr, static_cast<__half*>(c), ldc, m, n, k, split, epilogue, status_dev, stream}, t[0], t[1]);
        }
    }
    CUtensorMap mc;
    {
        const uint64_t dims[2] = {static_cast<uint64_t>(n), static_cast<uint64_t>(m)};
        const uint64_t strides[1] = {static_cast<uint64_t>(ldc) * 2};
        const uint32_t box[2] = {64, 32};
        if (int rc = make_tensor_map_f16(&mc, c, 2, dims, strides, box)) return rc;
    }
    if (takes_pairs(m, n, k, epilogue)) return gemm_pair_dispatch(ma, mw, mc, bp, rp, ldr, m, n, k, epilogue, status_dev, stream);
    switch (epilogue) {
        case STOF_EPI_BIAS: return launch<STOF_EPI_BIAS>(ma, mw, mc, bp, rp, ldr, m, n, k, status_dev, stream);
        case STOF_EPI_BIAS_GELU_ERF: return launch<STOF_EPI_BIAS_GELU_ERF>(ma, mw, mc, bp, rp, ldr, m, n, k, status_dev, stream);
        case STOF_EPI_BIAS_GELU_TANH: return launch<STOF_EPI_BIAS_GELU_TANH>(ma, mw, mc, bp, rp, ldr, m, n, k, status_dev, stream);
        case STOF_EPI_BIAS_RELU: return launch<STOF_EPI_BIAS_RELU>(ma, mw, mc, bp, rp, ldr, m, n, k, status_dev, stream);
        default: return launch<STOF_EPI_BIAS_RESIDUAL>(ma, mw, mc, bp, rp, ldr, m, n, k, status_dev, stream);
    }
}
