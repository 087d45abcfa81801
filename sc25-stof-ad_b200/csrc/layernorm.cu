// y = LayerNorm(x + bias + residual) * gamma + beta over rows of fp16, fp32 statistics (HBM-bound).
//
// One warp per row or pair of rows, persistent over rows.  A row is read once (through a shared-memory ring fed by bulk copies, two
// further groups of the warp in flight), held in registers as packed fp32 pairs, reduced with warp shuffles (mean, then the centred
// sum of squares, biased variance as src/triton_template/add_layernorm.py:33-55 and F.layer_norm do), and written once
// with 128-bit stores; bias, gamma and beta of a lane's columns stay in registers across rows.  Rows longer than 2048 elements are
// re-read from cache for the second and third sweep instead of being held in registers.
#include "stof_host.h"
#include "stof_ptx.cuh"

#include <cuda_fp16.h>

namespace stof {
namespace {

constexpr int LN_WARPS = 8;
constexpr int LN_BLOCKS_PER_SM = 4;
constexpr int LN_STAGES = 3;

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

template <int N>
__device__ __forceinline__ void warp_sums(float (&v)[N]) {        // N sums at once, their steps interleaved
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int i = 0; i < N; ++i) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
}

__device__ __forceinline__ void load8(const __half* p, float (&f)[8]) {
    const uint4 u = *reinterpret_cast<const uint4*>(p);
    const __half2* h = reinterpret_cast<const __half2*>(&u);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 t = __half22float2(h[i]);
        f[2 * i] = t.x;
        f[2 * i + 1] = t.y;
    }
}

__device__ __forceinline__ void add8(const __half* p, float (&f)[8]) {
    float t[8];
    load8(p, t);
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] += t[i];
}

__device__ __forceinline__ void store8(__half* p, const float (&f)[8]) {
    uint4 u;
    __half2* h = reinterpret_cast<__half2*>(&u);
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = __floats2half2_rn(f[2 * i], f[2 * i + 1]);
    *reinterpret_cast<uint4*>(p) = u;
}

// NCHUNK: 16-byte chunks held per lane and row (hidden <= NCHUNK * 256); NCHUNK == 0 selects the re-reading variant.
// ROWS: rows a warp normalises at a time.  Persistent: each warp walks groups of ROWS rows.  Rows (and residual rows) arrive through a
// per-warp ring of LN_STAGES shared-memory buffers filled by 1-D bulk copies, so that two further groups per warp are always in flight
// and the kernel keeps enough bytes outstanding to cover the HBM latency without spending registers on it.
// What bounds it: HBM and, one row at a time, the issue slots and the two reductions (590 instructions a row, 16 warps on an SM,
// 2.7 TB/s at 32768 x 1024 from HBM).  Two rows at a time share the conversion of bias, gamma and beta (held as fp16 in registers: as
// fp32 they alone took 64) and overlap their reductions: from HBM, 32768 rows of 768 28 -> 19 us (5.2 TB/s), of 1024 45 -> 27 us,
// 8192 rows of 768 9.5 -> 8.0 us.  Two blocks on an SM matter more than the last registers (hidden 768: 23 us with one of 152; at
// hidden 1024 two rows spill 48 bytes at the cap of 128).
template <int NCHUNK, int ROWS>
__global__ void __launch_bounds__(LN_WARPS * 32, 2)
layernorm_kernel(const __half* x, long long ldx, const __half* bias, const __half* residual,
                 long long ldr, const __half* gamma, const __half* beta, float eps, __half* y,
                 long long ldy, int rows, int hidden, int* status) {
    extern __shared__ __align__(128) unsigned char ln_smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int warps_total = gridDim.x * LN_WARPS;
    int row = blockIdx.x * LN_WARPS + warp;                // (a group of ROWS rows, in the variants that hold rows in registers)
    grid_dependency_wait();
    grid_launch_dependents();
    const int groups = (rows + ROWS - 1) / ROWS;
    if (row >= groups) return;
    const int nchunks = hidden >> 3;
    const float inv_n = 1.0f / static_cast<float>(hidden);

    if constexpr (NCHUNK > 0) {
        const uint32_t row_bytes = static_cast<uint32_t>(hidden) * 2u;
        const uint32_t part_bytes = ROWS * row_bytes, slot_bytes = residual ? 2u * part_bytes : part_bytes;
        uint64_t* bars = reinterpret_cast<uint64_t*>(ln_smem) + warp * LN_STAGES;
        unsigned char* ring = ln_smem + LN_WARPS * LN_STAGES * 8 + static_cast<size_t>(warp) * LN_STAGES * slot_bytes;
        if (lane == 0) {
            for (int s = 0; s < LN_STAGES; ++s) mbar_init(&bars[s], 1);
            fence_mbar_init();
        }
        __syncwarp();
        auto issue = [&](int group, int s) {               // lane 0 only
            unsigned char* dst = ring + static_cast<size_t>(s) * slot_bytes;
            const int first = group * ROWS, count = min(ROWS, rows - first);
            mbar_arrive_expect_tx(&bars[s], static_cast<uint32_t>(count) * (residual ? 2u * row_bytes : row_bytes));
            for (int i = 0; i < count; ++i) {
                const int r = rows - 1 - (first + i);      // rows are visited from the last to the first (see the launcher)
                bulk_load_1d(dst + i * row_bytes, x + static_cast<size_t>(r) * ldx, row_bytes, &bars[s]);
                if (residual) bulk_load_1d(dst + part_bytes + i * row_bytes, residual + static_cast<size_t>(r) * ldr, row_bytes, &bars[s]);
            }
        };
        if (lane == 0) {
#pragma unroll
            for (int s = 0; s < LN_STAGES - 1; ++s)
                if (row + s * warps_total < groups) issue(row + s * warps_total, s);
        }
        // 8 halves -> 4 packed fp32 pairs
        auto unpack2 = [](const uint4& u, float2 (&f)[4]) {
            const __half2* h = reinterpret_cast<const __half2*>(&u);
#pragma unroll
            for (int i = 0; i < 4; ++i) f[i] = __half22float2(h[i]);
        };
        // up to 1024 columns a variant serves 256 sizes, so that only a lane's last chunk may lie beyond the row
        auto holds = [&](int i) { return (NCHUNK <= 4 && i < NCHUNK - 1) || lane + 32 * i < nchunks; };
        // bias, gamma and beta of this lane's columns stay in registers as fp16 for every row the warp processes
        // (rows up to 1024 columns; longer rows read them per row to bound the register count)
        constexpr bool VECTORS_IN_REGS = NCHUNK <= 4;
        constexpr int V = VECTORS_IN_REGS ? NCHUNK : 1;
        const uint4 zeros = make_uint4(0u, 0u, 0u, 0u), ones = make_uint4(0x3C003C00u, 0x3C003C00u, 0x3C003C00u, 0x3C003C00u);
        auto vec = [&](const __half* v, int i, const uint4& none) {
            return v != nullptr ? __ldca(reinterpret_cast<const uint4*>(v + 8 * (lane + 32 * i))) : none;
        };
        uint4 ub[V], ug[V], ut[V];
        if constexpr (VECTORS_IN_REGS) {
#pragma unroll
            for (int i = 0; i < NCHUNK; ++i) {
                ub[i] = ug[i] = ut[i] = zeros;
                if (holds(i)) {
                    ub[i] = vec(bias, i, zeros);
                    ug[i] = vec(gamma, i, ones);
                    ut[i] = vec(beta, i, zeros);
                }
            }
        }
        for (int it = 0; row < groups; row += warps_total, ++it) {
            if constexpr (VECTORS_IN_REGS) {         // converted again for each group: kept as fp32 they would take twice the registers
#pragma unroll
                for (int i = 0; i < NCHUNK; ++i)
                    for (uint4* u : {&ub[i], &ug[i], &ut[i]}) asm volatile("" : "+r"(u->x), "+r"(u->y), "+r"(u->z), "+r"(u->w));
            }
            const int s = it % LN_STAGES;
            const uint32_t parity = static_cast<uint32_t>((it / LN_STAGES) & 1);
            // completes with the copy (no partner thread involved); bounded all the same by a cycle budget: a warp whose copy
            // never lands reports it and leaves its remaining rows unwritten instead of normalising stale shared memory
            if (!__all_sync(0xffffffffu, mbar_wait_budget(&bars[s], parity))) {
                if (lane == 0 && status) atomicCAS(status, 0, (s << 8) | STATUS_WAIT_TIMEOUT);
                break;
            }
            const unsigned char* src = ring + static_cast<size_t>(s) * slot_bytes;
            const int count = min(ROWS, rows - row * ROWS);          // (a missing second row works on what the slot held before)
            float2 v[ROWS][NCHUNK][4];
            float2 sum2[ROWS];
#pragma unroll
            for (int q = 0; q < ROWS; ++q) sum2[q] = make_float2(0.f, 0.f);
#pragma unroll
            for (int i = 0; i < NCHUNK; ++i) {
                const int c = lane + 32 * i;
#pragma unroll
                for (int q = 0; q < ROWS; ++q)
#pragma unroll
                    for (int j = 0; j < 4; ++j) v[q][i][j] = make_float2(0.f, 0.f);
                if (holds(i)) {
                    float2 t[4];
#pragma unroll
                    for (int q = 0; q < ROWS; ++q) {
                        unpack2(*reinterpret_cast<const uint4*>(src + q * row_bytes + 16 * c), v[q][i]);
                        if (residual) {
                            unpack2(*reinterpret_cast<const uint4*>(src + part_bytes + q * row_bytes + 16 * c), t);
#pragma unroll
                            for (int j = 0; j < 4; ++j) v[q][i][j] = add2(v[q][i][j], t[j]);
                        }
                    }
                    if (bias) {
                        unpack2(VECTORS_IN_REGS ? ub[VECTORS_IN_REGS ? i : 0] : vec(bias, i, zeros), t);
#pragma unroll
                        for (int q = 0; q < ROWS; ++q)
#pragma unroll
                            for (int j = 0; j < 4; ++j) v[q][i][j] = add2(v[q][i][j], t[j]);
                    }
#pragma unroll
                    for (int q = 0; q < ROWS; ++q)
#pragma unroll
                        for (int j = 0; j < 4; ++j) sum2[q] = add2(sum2[q], v[q][i][j]);
                }
            }
            // this slot is read out: refill the slot that was consumed one group ago with the group LN_STAGES - 1 ahead
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
                const int ahead = row + (LN_STAGES - 1) * warps_total;
                if (ahead < groups) issue(ahead, (it + LN_STAGES - 1) % LN_STAGES);
            }
            float stat[ROWS];
            float2 sq2[ROWS];
#pragma unroll
            for (int q = 0; q < ROWS; ++q) stat[q] = sum2[q].x + sum2[q].y;
            warp_sums(stat);
#pragma unroll
            for (int q = 0; q < ROWS; ++q) {
                const float mean = stat[q] * inv_n;
                const float2 nmean2 = make_float2(-mean, -mean);
                sq2[q] = make_float2(0.f, 0.f);
#pragma unroll
                for (int i = 0; i < NCHUNK; ++i) {
                    if (holds(i)) {
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            v[q][i][j] = add2(v[q][i][j], nmean2);            // centred value, kept for the output pass
                            sq2[q] = fma2(v[q][i][j], v[q][i][j], sq2[q]);
                        }
                    }
                }
            }
#pragma unroll
            for (int q = 0; q < ROWS; ++q) stat[q] = sq2[q].x + sq2[q].y;
            warp_sums(stat);
            float2 rstd2[ROWS];
#pragma unroll
            for (int q = 0; q < ROWS; ++q) {
                const float rstd = 1.0f / sqrtf(stat[q] * inv_n + eps);
                rstd2[q] = make_float2(rstd, rstd);
            }
            __half* yr = y + static_cast<size_t>(rows - 1 - row * ROWS) * ldy;
#pragma unroll
            for (int i = 0; i < NCHUNK; ++i) {
                const int c = lane + 32 * i;
                if (holds(i)) {
                    float2 gg[4], bb[4];
                    unpack2(VECTORS_IN_REGS ? ug[VECTORS_IN_REGS ? i : 0] : vec(gamma, i, ones), gg);
                    unpack2(VECTORS_IN_REGS ? ut[VECTORS_IN_REGS ? i : 0] : vec(beta, i, zeros), bb);
#pragma unroll
                    for (int q = 0; q < ROWS; ++q) {
                        uint4 u;
                        __half2* h = reinterpret_cast<__half2*>(&u);
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const float2 o = fma2(mul2(v[q][i][j], rstd2[q]), gg[j], bb[j]);
                            h[j] = __floats2half2_rn(o.x, o.y);
                        }
                        if (q < count) *reinterpret_cast<uint4*>(yr - q * ldy + 8 * c) = u;
                    }
                }
            }
        }
    } else {
        for (; row < rows; row += warps_total) {
            const __half* xr = x + static_cast<size_t>(rows - 1 - row) * ldx;
            const __half* rr = residual ? residual + static_cast<size_t>(rows - 1 - row) * ldr : nullptr;
            __half* yr = y + static_cast<size_t>(rows - 1 - row) * ldy;
            float sum = 0.f;
            for (int c = lane; c < nchunks; c += 32) {
                float t[8];
                load8(xr + 8 * c, t);
                if (bias) add8(bias + 8 * c, t);
                if (rr) add8(rr + 8 * c, t);
#pragma unroll
                for (int j = 0; j < 8; ++j) sum += t[j];
            }
            const float mean = warp_sum(sum) * inv_n;
            float sq = 0.f;
            for (int c = lane; c < nchunks; c += 32) {
                float t[8];
                load8(xr + 8 * c, t);
                if (bias) add8(bias + 8 * c, t);
                if (rr) add8(rr + 8 * c, t);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const float d = t[j] - mean;
                    sq += d * d;
                }
            }
            const float rstd = 1.0f / sqrtf(warp_sum(sq) * inv_n + eps);
            for (int c = lane; c < nchunks; c += 32) {
                float t[8], g[8], b[8];
                load8(xr + 8 * c, t);
                if (bias) add8(bias + 8 * c, t);
                if (rr) add8(rr + 8 * c, t);
                if (gamma) load8(gamma + 8 * c, g);
                if (beta) load8(beta + 8 * c, b);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    float o = (t[j] - mean) * rstd;
                    if (gamma) o *= g[j];
                    if (beta) o += b[j];
                    t[j] = o;
                }
                store8(yr + 8 * c, t);
            }
        }
    }
}

}  // namespace
}  // namespace stof

using namespace stof;

extern "C" int stof_bias_residual_layernorm(const void* x, long long ldx, const void* bias, const void* residual, long long ldr,
                                            const void* gamma, const void* beta, float eps, void* y, long long ldy, int rows, int hidden,
                                            int* status_dev, void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    STOF_REQUIRE(x && y, "layernorm: null x or y");
    STOF_REQUIRE(rows >= 0 && hidden > 0, "layernorm: bad shape (%d, %d)", rows, hidden);
    STOF_REQUIRE(hidden % 8 == 0, "layernorm: hidden %d must be a multiple of 8", hidden);
    if (hidden > 8192) {
        set_error("layernorm: hidden %d beyond the maximum of 8192", hidden);
        return STOF_E_LIMIT;
    }
    STOF_REQUIRE(ldx % 8 == 0 && ldy % 8 == 0 && (!residual || ldr % 8 == 0), "layernorm: row strides must be multiples of 8 elements");
    STOF_REQUIRE(ldx >= hidden && ldy >= hidden && (!residual || ldr >= hidden), "layernorm: row stride smaller than hidden");
    STOF_REQUIRE(aligned16(x) && aligned16(y) && aligned16(bias) && aligned16(residual) && aligned16(gamma) && aligned16(beta),
                 "layernorm: pointers must be 16-byte aligned");
    if (rows == 0) return STOF_OK;
    const __half *xp = static_cast<const __half*>(x), *bp = static_cast<const __half*>(bias), *rp = static_cast<const __half*>(residual),
                 *gp = static_cast<const __half*>(gamma), *tp = static_cast<const __half*>(beta);
    __half* yp = static_cast<__half*>(y);
    auto ring_smem = [&](int rows_each) {
        return static_cast<size_t>(LN_WARPS) * LN_STAGES * (8 + static_cast<size_t>(rows_each) * hidden * 2 * (residual ? 2 : 1));
    };
    // persistent grid: as many blocks as are resident at once (registers and the ring decide), never more than the rows need.
    // The kernel visits the rows from the last to the first: the producer of x (a GEMM walking its tiles upwards) wrote the
    // last rows most recently, so they are the ones still in L2, and the rows this kernel writes last are the first a
    // following GEMM reads (0.3 % of a BERT-large forward, measured)
    auto launch = [&](auto kernel, int rows_each, size_t smem) -> int {
        if (smem > 48 * 1024) STOF_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
        int per_sm = 0;
        STOF_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, LN_WARPS * 32, smem));
        if (per_sm < 1) per_sm = 1;
        if (per_sm > LN_BLOCKS_PER_SM) per_sm = LN_BLOCKS_PER_SM;
        int blocks = (rows + LN_WARPS * rows_each - 1) / (LN_WARPS * rows_each);
        if (blocks > sm_count() * per_sm) blocks = sm_count() * per_sm;
        LaunchConfig lc(dim3(static_cast<unsigned>(blocks)), LN_WARPS * 32, smem, stream);
        STOF_CUDA(cudaLaunchKernelEx(&lc.cfg, kernel, xp, ldx, bp, rp, ldr, gp, tp, eps, yp, ldy, rows, hidden, status_dev));
        return STOF_OK;
    };
    // Two rows at a time where each of the 16 warps that an SM holds gets at least that many, and no residual row doubles the ring
    // (8192 rows of 768: 9.5 us one at a time, 8.0 in pairs)
    if (residual == nullptr && hidden <= 1024 && rows >= sm_count() * 2 * LN_WARPS * 2) {
        if (hidden <= 256) return launch(layernorm_kernel<1, 2>, 2, ring_smem(2));
        if (hidden <= 512) return launch(layernorm_kernel<2, 2>, 2, ring_smem(2));
        if (hidden <= 768) return launch(layernorm_kernel<3, 2>, 2, ring_smem(2));
        return launch(layernorm_kernel<4, 2>, 2, ring_smem(2));
    }
    if (hidden <= 256) return launch(layernorm_kernel<1, 1>, 1, ring_smem(1));
    if (hidden <= 512) return launch(layernorm_kernel<2, 1>, 1, ring_smem(1));
    if (hidden <= 768) return launch(layernorm_kernel<3, 1>, 1, ring_smem(1));
    if (hidden <= 1024) return launch(layernorm_kernel<4, 1>, 1, ring_smem(1));
    if (hidden <= 2048) return launch(layernorm_kernel<8, 1>, 1, ring_smem(1));
    return launch(layernorm_kernel<0, 1>, 1, 0);
}
