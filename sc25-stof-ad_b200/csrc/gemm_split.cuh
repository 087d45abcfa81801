// What the GEMM kernels for few output tiles have in common (gemm_split.cu, gemm_split_ln.cu): shapes, the TMA producer and the
// MMA issuer of one BM x BN tile over K steps kb0 .. kb1 - 1 of 128.
#pragma once
#include "gemm_split.h"
#include "stof_ptx.cuh"

namespace stof {
namespace {

constexpr int S_BK = 128;                       // two 64-wide swizzle atoms per stage
constexpr int S_STAGE_MEMORY = 192 * 1024;
constexpr int S_BAR_BYTES = 512;
constexpr int S_SMEM_LIMIT = 227 * 1024;

template <int BM, int BN>
struct SplitShape {
    static constexpr int EPI_WARPS = 4 * (BN / 64);                 // four for each 64 columns: one row and 64 columns per thread
    static constexpr int EPI_THREADS = 32 * EPI_WARPS;
    static constexpr int THREADS = EPI_THREADS + 64;
    static constexpr int A_ATOM = BM * 128;                         // BM rows of 64 fp16
    static constexpr int B_ATOM = 64 * 128;                         // 64 k rows of 64 fp16
    static constexpr int A_BYTES = 2 * A_ATOM;
    static constexpr int STAGE_BYTES = A_BYTES + 2 * (BN / 64) * B_ATOM;
    static constexpr int MAX_STAGES = S_STAGE_MEMORY / STAGE_BYTES;
    static constexpr int CHUNKS = BN / 8;                           // 16-byte pieces per row of the output tile
    static constexpr int RESIDUAL_BYTES = BM * BN * 2;
    // where row r, piece g of the residual tile lies in its copy in shared memory: eight rows that read one piece meet eight banks
    __device__ __forceinline__ static int residual_at(int r, int g) { return (r * CHUNKS + (g ^ (r & 7))) * 16; }
};

// The epilogues run once per launch, on instructions that come from L2 as they are needed (some three bytes a cycle: 64 columns
// unrolled took 5000 cycles before the first store).  So they are short loops over 16 columns, and what they read beside the
// accumulator - bias, gamma, beta, the residual tile - is put into shared memory while the products run.
//
// Asynchronous 16-byte copy global -> shared; zeros where `valid` is false
__device__ __forceinline__ void copy_async16(uint32_t dst, const void* src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16u : 0u) : "memory");
}
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Epilogue threads, from thread `first` on: `count` fp16 values (a multiple of 8) of a row vector, or `fill` (two fp16) where there is none
__device__ __forceinline__ void stage_vector(unsigned char* dst, const __half* src, int valid, int count, uint32_t fill, int first) {
    const int g = static_cast<int>(threadIdx.x) - first;
    if (g < 0 || g >= count / 8) return;
    if (src != nullptr) copy_async16(smem_u32(dst) + 16 * g, 8 * g < valid ? src + 8 * g : src, 8 * g < valid);
    else reinterpret_cast<uint4*>(dst)[g] = make_uint4(fill, fill, fill, fill);
}
// Rows row_lo .. row_lo + rows - 1 of the residual tile (tile-local row numbers)
template <class Shape>
__device__ __forceinline__ void stage_residual(unsigned char* dst, const __half* residual, long long ldr, int m0, int n0, int m, int n, int row_lo, int rows) {
    const uint32_t d = smem_u32(dst);
#pragma unroll 1
    for (int i = threadIdx.x; i < rows * Shape::CHUNKS; i += Shape::EPI_THREADS) {
        const int r = row_lo + i / Shape::CHUNKS, g = i % Shape::CHUNKS;
        const bool valid = residual != nullptr && m0 + r < m && n0 + 8 * g < n;
        if (residual != nullptr) copy_async16(d + Shape::residual_at(r, g), valid ? residual + static_cast<size_t>(m0 + r) * ldr + n0 + 8 * g : residual, valid);
        else *reinterpret_cast<uint4*>(dst + Shape::residual_at(r, g)) = make_uint4(0u, 0u, 0u, 0u);
    }
}
template <int THREADS>
__device__ __forceinline__ void epilogue_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(THREADS) : "memory"); }

// shared memory of this block -> shared memory of a block of the cluster, completion on that block's mbarrier
__device__ __forceinline__ void bulk_copy_to_peer(uint32_t dst_cluster, uint32_t src, uint32_t bytes, uint32_t bar_cluster) {
    asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst_cluster), "r"(src), "r"(bytes),
                 "r"(bar_cluster)
                 : "memory");
}

// Producer warp: loads the operands of the tile
template <class Shape, int BN>
__device__ __forceinline__ void split_produce(const CUtensorMap& map_a, const CUtensorMap& map_w, unsigned char* smem, uint64_t* full, uint64_t* empty,
                                              int m0, int n0, int kb0, int kb1, int stages, const WaitCtx& wctx) {
    const bool issue = elect_one();
    const uint32_t full0 = smem_u32(full), empty0 = smem_u32(empty), smem0 = smem_u32(smem);
    auto load_w = [&](int kb, int s) {
        const uint32_t bar = full0 + 8 * s, dst = smem0 + s * Shape::STAGE_BYTES + Shape::A_BYTES;
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int j = 0; j < BN / 64; ++j)
                tma_load_2d_addr(dst + (h * (BN / 64) + j) * Shape::B_ATOM, &map_w, bar, n0 + 64 * j, kb * S_BK + 64 * h);
    };
    auto load_a = [&](int kb, int s) {
        const uint32_t bar = full0 + 8 * s, dst = smem0 + s * Shape::STAGE_BYTES;
#pragma unroll
        for (int h = 0; h < 2; ++h) tma_load_2d_addr(dst + h * Shape::A_ATOM, &map_a, bar, kb * S_BK + 64 * h, m0);
    };
    grid_dependency_wait();
    grid_launch_dependents();
    const int first = min(kb1 - kb0, stages);
    if (issue)
        for (int i = 0; i < first; ++i) {
            mbar_arrive_expect_tx_addr(full0 + 8 * i, Shape::STAGE_BYTES);
            load_w(kb0 + i, i);
            load_a(kb0 + i, i);
        }
    int s = 0;
    uint32_t phase = 0;
    for (int kb = kb0 + first; kb < kb1; ++kb) {
        mbar_wait_addr(empty0 + 8 * s, phase, wctx, stages + s);
        if (issue) {
            mbar_arrive_expect_tx_addr(full0 + 8 * s, Shape::STAGE_BYTES);
            load_w(kb, s);
            load_a(kb, s);
        }
        if (++s == stages) { s = 0; phase ^= 1u; }
    }
}

// Issuer warp: the tile's products.  The whole warp walks the loop and one lane issues, so that descriptors and addresses
// stay warp-uniform; a ring position by division (a run-time number of stages) or generic pointers doubled the time of a step.
template <class Shape, int BM, int BN>
__device__ __forceinline__ void split_multiply(unsigned char* smem, uint64_t* full, uint64_t* empty, uint64_t* tfull, uint32_t tmem_base, int kb0,
                                               int kb1, int stages, const WaitCtx& wctx) {
    constexpr uint32_t idesc = make_idesc_f16(BM, BN, /*b_mn_major=*/true);
    const bool issue = elect_one();
    const uint32_t full0 = smem_u32(full), empty0 = smem_u32(empty);
    const uint64_t a_desc0 = make_smem_desc_sw128(smem_u32(smem), 16, 1024);
    const uint64_t b_desc0 = make_smem_desc_sw128(smem_u32(smem) + Shape::A_BYTES, Shape::B_ATOM, 1024);
    int s = 0;
    uint32_t phase = 0, acc = 0;
    for (int kb = kb0; kb < kb1; ++kb) {
        mbar_wait_addr(full0 + 8 * s, phase, wctx, s);
        tc_fence_after();
        const uint64_t off = static_cast<uint64_t>(s * (Shape::STAGE_BYTES >> 4));
        if (issue) {
#pragma unroll
            for (int kk = 0; kk < S_BK / 16; ++kk) {
                const int h = kk / 4, q = kk % 4;
                mma_f16_ss(tmem_base, a_desc0 + off + h * (Shape::A_ATOM >> 4) + q * 2, b_desc0 + off + h * ((BN / 64) * Shape::B_ATOM >> 4) + q * 128,
                           idesc, acc);
                acc = 1;
            }
            tc_commit_addr(empty0 + 8 * s);
        }
        if (++s == stages) { s = 0; phase ^= 1u; }
    }
    if (issue) tc_commit_addr(smem_u32(tfull));
    grid_dependency_wait();
}

// Ahead of the dependency wait, by one thread: descriptors, and the block's first weight tiles into L2.  (Loading them for good
// there, where a caller knows that nothing just wrote them, gained nothing in an encoder: 365 us a pass either way.)
template <int BN>
__device__ __forceinline__ void split_prefetch(const CUtensorMap& map_a, const CUtensorMap& map_w, int n0, int kb0, int kb1, int stages) {
    tma_prefetch_desc(&map_a);
    tma_prefetch_desc(&map_w);
    for (int kb = kb0; kb < kb1 && kb < kb0 + stages; ++kb)
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int j = 0; j < BN / 64; ++j) tma_prefetch_2d(&map_w, n0 + 64 * j, kb * S_BK + 64 * h);
}

// Host: the A map (boxes of BM rows x 64)
template <int BM>
int split_map_a(CUtensorMap* map, const void* a, long long lda, int m, int k) {
    const uint64_t dims[2] = {static_cast<uint64_t>(k), static_cast<uint64_t>(m)};
    const uint64_t strides[1] = {static_cast<uint64_t>(lda) * 2};
    const uint32_t box[2] = {64, BM};
    return make_tensor_map_f16(map, a, 2, dims, strides, box);
}

}  // namespace
}  // namespace stof
