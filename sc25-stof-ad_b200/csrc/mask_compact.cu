// Mask -> block-CSR index compaction (integer, bit-exact, HBM-bound).
//
// Semantics follow get_sparse_storage of the reference (src/util/masks.py:125-184): tiles of mask[0]
// are scanned row-major; a tile whose elements all equal 1 is "full", all equal 0 "empty", anything
// else "partial" and carries the fp16 tile -10000 * (1 - m).  `load` merges full and partial in
// column order.  The element count of non-zeros runs over the whole (batch, S, S) tensor.
//
// Phase 1 (classify_kernel): the mask is streamed once with 128-bit loads, eight in flight per thread.  A thread block owns a
// stripe of one block-row by a run of whole tiles and writes one class byte per tile; of the batch elements after the first,
// of which only the non-zeros count, it owns a flat piece.  Bound by HBM, so what is kept small is the work per 16 bytes:
// a thread stays in one column of chunks, keeps an AND and an OR of the words it saw, and settles its flags once at the end
// (position and flags per chunk, with four loads in flight: 8 x 4096 x 4096 fp32 in 130 us = 4.1 TB/s; now 88 us = 6.1 TB/s).
// The last block to finish (atomic ticket) turns the class bytes into per-row counts and into the three row-pointer arrays
// with a warp-shuffle prefix sum.
// Phase 2 (fill_kernel): thread blocks for the column indices (one warp per block-row ranks its tiles with ballots + popc)
// and one thread block per partial tile, which finds its tile from its number - block-row by bisection of the row pointers,
// column by ballots over the class bytes - and gathers it.  (Tiles handed out per block-row made the few full rows of a
// mask with global tokens a chain of eight gathers, 14 us.)
// The sizes of phase 2's outputs depend on the data, so the host has to read the counts between the phases.  In
// stof_mask_classify_notify the last block of phase 1 writes them into host memory itself: no memset before the kernel, no
// copy and no stream synchronisation after it.
#include "stof_host.h"
#include "stof_ptx.cuh"

#include <cuda_fp16.h>

#include <mutex>

namespace stof {
namespace {

constexpr int CLS_EMPTY = 0;
constexpr int CLS_FULL = 1;
constexpr int CLS_PART = 2;

constexpr int CLASSIFY_THREADS = 256;
constexpr int MAX_TILES_PER_ROW = 4096;
constexpr int FILL_THREADS = 256;

// Header of 16 bytes at the start of the caller's workspace, class bytes follow.  A workspace is 4-byte aligned, no more: the 64-bit
// count lies at the multiple of 8 behind the ticket.
struct Workspace {
    unsigned int* ticket;     // blocks that finished phase 1 (reset by the last one)
    unsigned long long* nnz;  // non-zero elements seen so far (read and reset by the last block)
    explicit Workspace(void* header)
        : ticket(static_cast<unsigned int*>(header)), nnz(reinterpret_cast<unsigned long long*>((reinterpret_cast<uintptr_t>(header) + 11) & ~uintptr_t{7})) {}
};
constexpr size_t WS_HEADER = 16;

// Where phase 1 reports to, beside the row pointers: device counts (the two-call interface), or a float with the non-zero
// share and a record in host memory
struct Report {
    unsigned long long* counts;
    float* nnz_percent;
    float inv_cells;                          // 1 / S^2
    const int* status;
    stof_mask_notice* notice;
    unsigned long long stamp;
};

__host__ __device__ inline size_t cls_bytes(int nbm, int nbn) { return (static_cast<size_t>(nbm) * nbn + 15) & ~static_cast<size_t>(15); }

// Non-zero elements of a 16-byte chunk, added to `nz` (-0.0 counts as zero, NaN as non-zero), without branches.  fp16: a half
// without its sign is at most 0x7FFF, so adding 0x7FFF sets its top bit exactly when it is not zero and carries nowhere.
template <bool F32>
__device__ __forceinline__ void count_chunk(const uint4& v, unsigned& nz) {
    if (F32) {
        nz += min(v.x & 0x7FFFFFFFu, 1u) + min(v.y & 0x7FFFFFFFu, 1u);
        nz += min(v.z & 0x7FFFFFFFu, 1u) + min(v.w & 0x7FFFFFFFu, 1u);
    } else {
        const unsigned m = 0x7FFF7FFFu, t = 0x80008000u;
        const unsigned a = ((v.x & m) + m) & t, b = ((v.y & m) + m) & t, c = ((v.z & m) + m) & t, d = ((v.w & m) + m) & t;
        nz += __popc(a | (b >> 1) | (c >> 2) | (d >> 3));
    }
}

// Runs in the last block of phase 1: class bytes -> row counts -> row pointers and totals.
__device__ void scan_rows(const unsigned char* cls, int nbm, int nbn, int* full_row_ptr, int* part_row_ptr, int* load_row_ptr,
                          const Report& report, unsigned long long nnz, int* row_counts /* smem, 2 * nbm_chunk */) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    int carry_full = 0, carry_part = 0;
    if (threadIdx.x == 0) {
        full_row_ptr[0] = 0;
        part_row_ptr[0] = 0;
        load_row_ptr[0] = 0;
    }
    // rows are processed in chunks of 32 * nwarps: every thread loads class bytes of the chunk independently
    // (no serial chain of dependent loads) and counts into shared memory, then warp 0 scans the chunk
    const int chunk = 32 * nwarps;
    for (int r0 = 0; r0 < nbm; r0 += chunk) {
        for (int i = threadIdx.x; i < 2 * chunk; i += blockDim.x) row_counts[i] = 0;
        __syncthreads();
        const int rows_here = min(chunk, nbm - r0);
        const int cells = rows_here * nbn;
        if ((nbn & 15) == 0 && (reinterpret_cast<uintptr_t>(cls) & 15) == 0) {
            // sixteen class bytes of one row at a time; bit 0 of a byte says full, bit 1 partial
            for (int i = threadIdx.x; i < cells / 16; i += blockDim.x) {
                const uint4 v = __ldcg(reinterpret_cast<const uint4*>(cls + static_cast<size_t>(r0) * nbn) + i);
                const int row = i / (nbn / 16);
                const unsigned one = 0x01010101u;
                const int nf = __popc(v.x & one) + __popc(v.y & one) + __popc(v.z & one) + __popc(v.w & one);
                const int np = __popc(v.x & (one << 1)) + __popc(v.y & (one << 1)) + __popc(v.z & (one << 1)) + __popc(v.w & (one << 1));
                if (nf) atomicAdd(&row_counts[2 * row], nf);
                if (np) atomicAdd(&row_counts[2 * row + 1], np);
            }
        } else {
            for (int i = threadIdx.x; i < cells; i += blockDim.x) {
                const int k = __ldcg(cls + static_cast<size_t>(r0) * nbn + i);
                if (k != CLS_EMPTY) atomicAdd(&row_counts[2 * (i / nbn) + (k == CLS_PART ? 1 : 0)], 1);
            }
        }
        __syncthreads();
        if (warp == 0) {
            for (int g = 0; g < nwarps; ++g) {
                const int r = r0 + g * 32 + lane;
                int nf = r < nbm ? row_counts[2 * (g * 32 + lane)] : 0;
                int np = r < nbm ? row_counts[2 * (g * 32 + lane) + 1] : 0;
                int sf = nf, sp = np;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int tf = __shfl_up_sync(0xffffffffu, sf, o);
                    const int tp = __shfl_up_sync(0xffffffffu, sp, o);
                    if (lane >= o) {
                        sf += tf;
                        sp += tp;
                    }
                }
                if (r < nbm) {
                    full_row_ptr[r + 1] = carry_full + sf;
                    part_row_ptr[r + 1] = carry_part + sp;
                    load_row_ptr[r + 1] = carry_full + sf + carry_part + sp;
                }
                carry_full += __shfl_sync(0xffffffffu, sf, 31);
                carry_part += __shfl_sync(0xffffffffu, sp, 31);
            }
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        if (report.counts != nullptr) {
            report.counts[0] = static_cast<unsigned long long>(carry_full);
            report.counts[1] = static_cast<unsigned long long>(carry_part);
            report.counts[2] = static_cast<unsigned long long>(carry_full + carry_part);
            report.counts[3] = nnz;
        }
        // the same operations, in fp32, as an int64 count divided by the number S^2 (torch multiplies by the reciprocal) times 100
        if (report.nnz_percent != nullptr)
            *report.nnz_percent = __fmul_rn(__fmul_rn(__ll2float_rn(static_cast<long long>(nnz)), report.inv_cells), 100.0f);
        if (report.notice != nullptr) {
            volatile stof_mask_notice* out = report.notice;
            out->n_full = carry_full;
            out->n_part = carry_part;
            out->nnz = static_cast<long long>(nnz);
            out->status = report.status != nullptr ? *report.status : 0;
            __threadfence_system();
            out->stamp = report.stamp;
        }
    }
}

// Where the thread blocks of phase 1 work: blocks 0 .. tile_blocks - 1 on the stripes of mask[0], the rest on equal pieces of the
// other batch elements, of which only the non-zeros count
struct Geometry {
    int seq_len, bm, bn;
    int stripe_cols, stripes, tile_blocks;
    unsigned long long rest_chunks;           // 16-byte chunks of mask[1 ..]
    unsigned rest_per_block;
};
constexpr int CLASSIFY_FLIGHT = 8;            // independent 16-byte loads of a thread

template <bool F32>
__global__ void __launch_bounds__(CLASSIFY_THREADS)
classify_kernel(const void* mask, const Geometry geo, int* full_row_ptr, int* part_row_ptr, int* load_row_ptr, const Report report,
                const Workspace ws, unsigned char* cls) {
    constexpr int EPC = F32 ? 4 : 8;                       // elements per 16-byte chunk
    constexpr unsigned ONE = F32 ? 0x3F800000u : 0x3C003C00u, MAG = F32 ? 0x7FFFFFFFu : 0x7FFF7FFFu;
    __shared__ unsigned s_flags[CLASSIFY_THREADS];         // per tile of the stripe: 1 = some element is not 1, 2 = some element is not 0
    __shared__ unsigned int s_nz[CLASSIFY_THREADS / 32];
    __shared__ int s_rows[2 * CLASSIFY_THREADS];
    __shared__ bool s_last;
    grid_dependency_wait();
    grid_launch_dependents();

    const int seq_len = geo.seq_len, bm = geo.bm, bn = geo.bn;
    const int nbn = seq_len / bn, nbm = seq_len / bm;
    unsigned nz = 0;
    if (static_cast<int>(blockIdx.x) < geo.tile_blocks) {
        const int brow = blockIdx.x / geo.stripes, stripe = blockIdx.x - brow * geo.stripes;
        const int col0 = stripe * geo.stripe_cols;
        const int cols = min(geo.stripe_cols, seq_len - col0);
        const int tiles = cols / bn;
        if (static_cast<int>(threadIdx.x) < tiles) s_flags[threadIdx.x] = 0;
        __syncthreads();
        // A thread keeps to one chunk column and walks down the rows of the block-row: what it saw is an AND and an OR of words,
        // and becomes flags once, at the end.  (A stripe has a chunk column per thread at most, unless a single tile is wider.)
        for (int c0 = 0; c0 < cols / EPC; c0 += CLASSIFY_THREADS) {
            const int width = min(CLASSIFY_THREADS, cols / EPC - c0);
            const int rows_at_once = CLASSIFY_THREADS / width, r0 = threadIdx.x / width, cc = c0 + threadIdx.x - r0 * width;
            unsigned all_and = 0xFFFFFFFFu, all_or = 0;
            if (r0 >= rows_at_once || r0 >= bm) continue;
            const size_t pitch = static_cast<size_t>(seq_len) / EPC, step = pitch * rows_at_once;
            const uint4* p = static_cast<const uint4*>(mask) + (static_cast<size_t>(brow) * bm + r0) * pitch + col0 / EPC + cc;
            for (int r = r0; r < bm; r += CLASSIFY_FLIGHT * rows_at_once, p += CLASSIFY_FLIGHT * step) {
                uint4 v[CLASSIFY_FLIGHT];
#pragma unroll
                for (int u = 0; u < CLASSIFY_FLIGHT; ++u)
                    if (r + u * rows_at_once < bm) v[u] = __ldca(p + u * step);
#pragma unroll
                for (int u = 0; u < CLASSIFY_FLIGHT; ++u)
                    if (r + u * rows_at_once < bm) {
                        all_and &= v[u].x & v[u].y & v[u].z & v[u].w;
                        all_or |= v[u].x | v[u].y | v[u].z | v[u].w;
                        count_chunk<F32>(v[u], nz);
                    }
            }
            const unsigned f = ((all_and == ONE && all_or == ONE) ? 0u : 1u) | ((all_or & MAG) != 0u ? 2u : 0u);
            atomicOr(&s_flags[cc * EPC / bn], f);
        }
        __syncthreads();
        if (static_cast<int>(threadIdx.x) < tiles) {
            const unsigned f = s_flags[threadIdx.x];
            cls[static_cast<size_t>(brow) * nbn + col0 / bn + threadIdx.x] =
                static_cast<unsigned char>((f & 1u) == 0u ? CLS_FULL : ((f & 2u) == 0u ? CLS_EMPTY : CLS_PART));
        }
    } else {
        const unsigned long long lo = static_cast<unsigned long long>(blockIdx.x - geo.tile_blocks) * geo.rest_per_block;
        const unsigned count = static_cast<unsigned>(min(static_cast<unsigned long long>(geo.rest_per_block), geo.rest_chunks - lo));
        const uint4* p = static_cast<const uint4*>(mask) + static_cast<size_t>(seq_len) * seq_len / EPC + lo;
        for (unsigned i = threadIdx.x; i < count; i += CLASSIFY_FLIGHT * CLASSIFY_THREADS) {
            uint4 v[CLASSIFY_FLIGHT];
#pragma unroll
            for (int u = 0; u < CLASSIFY_FLIGHT; ++u)
                v[u] = i + u * CLASSIFY_THREADS < count ? __ldcs(p + i + u * CLASSIFY_THREADS) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
            for (int u = 0; u < CLASSIFY_FLIGHT; ++u) count_chunk<F32>(v[u], nz);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) nz += __shfl_xor_sync(0xffffffffu, nz, o);
    if ((threadIdx.x & 31) == 0) s_nz[threadIdx.x >> 5] = nz;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long t = 0;
        for (int i = 0; i < CLASSIFY_THREADS / 32; ++i) t += s_nz[i];
        if (t) atomicAdd(ws.nnz, t);
    }
    // last block of the whole grid builds the row pointers
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned t = atomicAdd(ws.ticket, 1u);
        s_last = (t == gridDim.x - 1);
        if (s_last) *ws.ticket = 0;                        // ready for the next call
    }
    __syncthreads();
    if (s_last) {
        __threadfence();
        unsigned long long nnz = 0;
        if (threadIdx.x == 0) nnz = atomicExch(ws.nnz, 0ull);
        scan_rows(cls, nbm, nbn, full_row_ptr, part_row_ptr, load_row_ptr, report, nnz, s_rows);
    }
}

// eight mask elements -> -10000 * (1 - m) in fp16 arithmetic
template <bool F32>
__device__ __forceinline__ uint4 mask_addend8(const void* mask, size_t src) {
    const __half one = __float2half(1.0f), neg = __float2half(-10000.0f);
    __half h[8];
    if (F32) {
        const float4 a = __ldca(reinterpret_cast<const float4*>(static_cast<const float*>(mask) + src));
        const float4 b = __ldca(reinterpret_cast<const float4*>(static_cast<const float*>(mask) + src + 4));
        h[0] = __float2half_rn(a.x); h[1] = __float2half_rn(a.y); h[2] = __float2half_rn(a.z); h[3] = __float2half_rn(a.w);
        h[4] = __float2half_rn(b.x); h[5] = __float2half_rn(b.y); h[6] = __float2half_rn(b.z); h[7] = __float2half_rn(b.w);
    } else {
        *reinterpret_cast<uint4*>(h) = __ldca(reinterpret_cast<const uint4*>(static_cast<const __half*>(mask) + src));
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) h[i] = __hmul(neg, __hsub(one, h[i]));
    return *reinterpret_cast<uint4*>(h);
}

// Thread blocks 0 .. index_blocks - 1: column indices, one block-row per warp.  The blocks after them: partial tiles
// blockIdx.x - index_blocks, + tile_blocks, ...
template <bool F32>
__global__ void __launch_bounds__(FILL_THREADS)
fill_kernel(const void* mask, int seq_len, int bm, int bn, const unsigned char* cls, const int* full_row_ptr, const int* part_row_ptr,
            const int* load_row_ptr, int* full_col_idx, int* part_col_idx, int* load_col_idx, __half* part_block_mask, int index_blocks) {
    __shared__ int s_tile[2];                              // block-row and column of the tile in hand
    grid_dependency_wait();
    grid_launch_dependents();
    const int nbm = seq_len / bm, nbn = seq_len / bn;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    if (static_cast<int>(blockIdx.x) < index_blocks) {
        const int brow = blockIdx.x * (FILL_THREADS / 32) + warp;
        if (brow >= nbm) return;
        const int f0 = full_row_ptr[brow], p0 = part_row_ptr[brow], l0 = load_row_ptr[brow];
        int nf = 0, np = 0;
        for (int c0 = 0; c0 < nbn; c0 += 32) {
            const int c = c0 + lane;
            const int k = c < nbn ? cls[static_cast<size_t>(brow) * nbn + c] : CLS_EMPTY;
            const unsigned bf = __ballot_sync(0xffffffffu, k == CLS_FULL);
            const unsigned bp = __ballot_sync(0xffffffffu, k == CLS_PART);
            const int rf = nf + __popc(bf & lt), rp = np + __popc(bp & lt);
            if (k == CLS_FULL) full_col_idx[f0 + rf] = c;
            if (k == CLS_PART) part_col_idx[p0 + rp] = c;
            if (k != CLS_EMPTY) load_col_idx[l0 + rf + rp] = c;
            nf += __popc(bf);
            np += __popc(bp);
        }
        return;
    }
    const int n_part = part_row_ptr[nbm];
    const int chunks_per_tile_row = bn / 8, chunks_per_tile = bm * chunks_per_tile_row;
    for (int t = blockIdx.x - index_blocks; t < n_part; t += gridDim.x - index_blocks) {
        if (warp == 0) {
            int lo = 0, hi = nbm;                          // the block-row with part_row_ptr[row] <= t < part_row_ptr[row + 1], 32 guesses at a time
            while (hi - lo > 1) {
                const int step = (hi - lo + 31) / 32, at = min(lo + lane * step, hi);
                const unsigned le = __ballot_sync(0xffffffffu, at < hi && part_row_ptr[at] <= t);
                const int last = 31 - __clz(le);           // lane 0 always holds
                hi = min(lo + (last + 1) * step, hi);
                lo = lo + last * step;
            }
            int rank = t - part_row_ptr[lo];               // the tile's number among the row's partial ones
            for (int c0 = 0; c0 < nbn; c0 += 32) {
                const int c = c0 + lane;
                const unsigned bp = __ballot_sync(0xffffffffu, c < nbn && cls[static_cast<size_t>(lo) * nbn + c] == CLS_PART);
                if (rank < __popc(bp)) {
                    if ((bp >> lane & 1u) && __popc(bp & lt) == rank) { s_tile[0] = lo; s_tile[1] = c; }
                    break;
                }
                rank -= __popc(bp);
            }
        }
        __syncthreads();
        const int brow = s_tile[0], c = s_tile[1];
        __half* dst = part_block_mask + static_cast<size_t>(t) * bm * bn;
        for (int idx = threadIdx.x; idx < chunks_per_tile; idx += blockDim.x) {
            const int r = idx / chunks_per_tile_row, cc = idx - r * chunks_per_tile_row;
            const size_t src = (static_cast<size_t>(brow) * bm + r) * seq_len + static_cast<size_t>(c) * bn + cc * 8;
            *reinterpret_cast<uint4*>(dst + static_cast<size_t>(r) * bn + cc * 8) = mask_addend8<F32>(mask, src);
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------------------------
// Scratch for stof_mask_compact_static: lives in the module's device image instead of a caller
// allocation.  Every GPU that loads the library holds these bytes until the process exits.
// ---------------------------------------------------------------------------------------------
constexpr int STATIC_MAX_TILES = 1 << 20;           // block rows x block columns the static scratch can classify
static __device__ __align__(256) unsigned char g_static_scratch[WS_HEADER + STATIC_MAX_TILES];

// Same ranking and gather as fill_kernel, but every write is checked against the capacity of the caller's
// buffers (the caller sized them without knowing the counts): entries that do not fit are dropped.
template <bool F32>
__global__ void __launch_bounds__(FILL_THREADS)
fill_bounded_kernel(const void* __restrict__ mask, int seq_len, int bm, int bn, const unsigned char* __restrict__ cls,
                    const int* __restrict__ full_row_ptr, const int* __restrict__ part_row_ptr, const int* __restrict__ load_row_ptr,
                    int* full_col_idx, int* part_col_idx, int* load_col_idx, long long col_capacity, __half* part_block_mask,
                    long long part_capacity) {
    extern __shared__ int s_part_cols[];
    const int nbn = seq_len / bn;
    const int brow = blockIdx.x, share = blockIdx.y, shares = gridDim.y;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int f0 = full_row_ptr[brow], p0 = part_row_ptr[brow], l0 = load_row_ptr[brow];
    const int n_part = part_row_ptr[brow + 1] - p0;
    if (warp == 0) {
        int nf = 0, np = 0;
        for (int c0 = 0; c0 < nbn; c0 += 32) {
            const int c = c0 + lane;
            const int k = c < nbn ? cls[static_cast<size_t>(brow) * nbn + c] : CLS_EMPTY;
            const unsigned bf = __ballot_sync(0xffffffffu, k == CLS_FULL);
            const unsigned bp = __ballot_sync(0xffffffffu, k == CLS_PART);
            const unsigned lt = (1u << lane) - 1u;
            const int rf = nf + __popc(bf & lt), rp = np + __popc(bp & lt);
            if (k == CLS_FULL) {
                if (share == 0) {
                    if (f0 + rf < col_capacity) full_col_idx[f0 + rf] = c;
                    if (l0 + rf + rp < col_capacity) load_col_idx[l0 + rf + rp] = c;
                }
            } else if (k == CLS_PART) {
                s_part_cols[rp] = c;
                if (share == 0) {
                    if (p0 + rp < col_capacity) part_col_idx[p0 + rp] = c;
                    if (l0 + rf + rp < col_capacity) load_col_idx[l0 + rf + rp] = c;
                }
            }
            nf += __popc(bf);
            np += __popc(bp);
        }
    }
    __syncthreads();
    if (n_part == 0 || part_block_mask == nullptr) return;
    const int chunks_per_tile_row = bn / 8;
    const int chunks_per_tile = bm * chunks_per_tile_row;
    for (int p = share; p < n_part; p += shares) {
        if (p0 + p >= part_capacity) break;
        const int c = s_part_cols[p];
        __half* dst = part_block_mask + static_cast<size_t>(p0 + p) * bm * bn;
        for (int idx = threadIdx.x; idx < chunks_per_tile; idx += blockDim.x) {
            const int r = idx / chunks_per_tile_row, cc = idx - r * chunks_per_tile_row;
            const size_t src = (static_cast<size_t>(brow) * bm + r) * seq_len + static_cast<size_t>(c) * bn + cc * 8;
            *reinterpret_cast<uint4*>(dst + static_cast<size_t>(r) * bn + cc * 8) = mask_addend8<F32>(mask, src);
        }
    }
}

// Device address of g_static_scratch on the current device.  In host code the array's name is only a
// host-side handle, never a pointer a kernel may use, so the address is asked from the runtime once per
// device (with that device current) and cached.  The query may be what makes the runtime load the module (and
// with it the array) onto the device; the cached address dies with the device's primary context, so a
// cudaDeviceReset() on that device leaves it stale.
int static_scratch_address(unsigned char** out) {
    static std::mutex mu;
    static unsigned char* addr[64] = {};
    int dev = 0;
    STOF_CUDA(cudaGetDevice(&dev));
    STOF_REQUIRE(dev >= 0 && dev < 64, "mask_compact_static: device ordinal %d out of range", dev);
    std::lock_guard<std::mutex> lock(mu);
    if (addr[dev] == nullptr) {
        void* p = nullptr;
        STOF_CUDA(cudaGetSymbolAddress(&p, g_static_scratch));
        STOF_REQUIRE(p != nullptr, "mask_compact_static: the runtime returned no address for the scratch array");
        addr[dev] = static_cast<unsigned char*>(p);
    }
    *out = addr[dev];
    return STOF_OK;
}

int check_geometry(int seq_len, int bm, int bn) {
    STOF_REQUIRE(seq_len > 0 && bm > 0 && bn > 0, "mask compaction: seq_len/block sizes must be positive");
    STOF_REQUIRE(seq_len % bm == 0 && seq_len % bn == 0, "mask compaction: seq_len %d is not a multiple of block_m %d and block_n %d",
                 seq_len, bm, bn);
    STOF_REQUIRE(bn % 8 == 0, "mask compaction: block_n %d must be a multiple of 8", bn);
    STOF_REQUIRE(seq_len / bn <= MAX_TILES_PER_ROW, "mask compaction: more than %d tiles per row", MAX_TILES_PER_ROW);
    return STOF_OK;
}

int launch_classify(const void* mask, int mask_dtype, int batch, int seq_len, int bm, int bn, int* full_row_ptr, int* part_row_ptr, int* load_row_ptr,
                    const Report& report, const Workspace& ws, unsigned char* cls, cudaStream_t stream) {
    const bool f32 = mask_dtype == STOF_DTYPE_F32;
    const int epc = f32 ? 4 : 8;
    // Stripes of whole tiles, 512 bytes of a row or more (coalescing, few blocks), at most one 16-byte chunk per thread of a row
    // unless a single tile is wider
    int stripe = bn;
    while (stripe * (f32 ? 4 : 2) < 512 && stripe < seq_len && stripe + bn <= CLASSIFY_THREADS * epc) stripe += bn;
    // large masks: wider stripes, until eight blocks per multiprocessor are left (each then has its eight loads per thread several times over)
    const int nbm = seq_len / bm;
    while (2 * stripe <= CLASSIFY_THREADS * epc && static_cast<long long>(nbm) * ((seq_len + 2 * stripe - 1) / (2 * stripe)) >= 8LL * sm_count()) stripe *= 2;
    Geometry geo;
    geo.seq_len = seq_len; geo.bm = bm; geo.bn = bn;
    geo.stripe_cols = stripe;
    geo.stripes = (seq_len + stripe - 1) / stripe;
    geo.tile_blocks = geo.stripes * nbm;
    // the other batch elements in pieces of 64 KB (two rounds of eight loads per thread)
    geo.rest_chunks = static_cast<unsigned long long>(batch - 1) * seq_len * seq_len / epc;
    geo.rest_per_block = 2 * CLASSIFY_FLIGHT * CLASSIFY_THREADS;
    const unsigned long long rest_blocks = (geo.rest_chunks + geo.rest_per_block - 1) / geo.rest_per_block;
    STOF_REQUIRE(geo.tile_blocks + rest_blocks < (1ull << 31), "mask compaction: mask too large");
    LaunchConfig lc(dim3(static_cast<unsigned>(geo.tile_blocks + rest_blocks)), CLASSIFY_THREADS, 0, stream);
    STOF_CUDA(cudaLaunchKernelEx(&lc.cfg, f32 ? classify_kernel<true> : classify_kernel<false>, mask, geo, full_row_ptr, part_row_ptr, load_row_ptr, report,
                                 ws, cls));
    return STOF_OK;
}

}  // namespace
}  // namespace stof

using namespace stof;

extern "C" size_t stof_mask_workspace_bytes(int seq_len, int block_m, int block_n) {
    if (seq_len <= 0 || block_m <= 0 || block_n <= 0) return 0;
    return WS_HEADER + cls_bytes(seq_len / block_m, seq_len / block_n);
}

extern "C" int stof_mask_classify(const void* mask, int mask_dtype, int batch, int seq_len, int block_m, int block_n,
                                  int* full_row_ptr, int* part_row_ptr, int* load_row_ptr, long long* counts, void* workspace,
                                  size_t workspace_bytes, void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (int rc = check_geometry(seq_len, block_m, block_n)) return rc;
    STOF_REQUIRE(mask && full_row_ptr && part_row_ptr && load_row_ptr && counts && workspace, "mask_classify: null pointer");
    STOF_REQUIRE(mask_dtype == STOF_DTYPE_F16 || mask_dtype == STOF_DTYPE_F32, "mask_classify: mask_dtype must be f16 or f32");
    STOF_REQUIRE(batch >= 1 && batch <= 65535, "mask_classify: batch %d out of range", batch);
    STOF_REQUIRE(aligned16(mask), "mask_classify: mask must be 16-byte aligned");
    STOF_REQUIRE((reinterpret_cast<uintptr_t>(workspace) & 3u) == 0, "mask_classify: workspace must be 4-byte aligned");
    if (workspace_bytes < stof_mask_workspace_bytes(seq_len, block_m, block_n)) {
        set_error("mask_classify: workspace of %zu bytes, need %zu", workspace_bytes, stof_mask_workspace_bytes(seq_len, block_m, block_n));
        return STOF_E_WORKSPACE;
    }
    const int nbm = seq_len / block_m;
    STOF_REQUIRE(nbm <= 65535, "mask_classify: more than 65535 block rows");
    STOF_CUDA(cudaMemsetAsync(workspace, 0, WS_HEADER, stream));
    const Report report{reinterpret_cast<unsigned long long*>(counts), nullptr, 0.f, nullptr, nullptr, 0};
    return launch_classify(mask, mask_dtype, batch, seq_len, block_m, block_n, full_row_ptr, part_row_ptr, load_row_ptr, report, Workspace(workspace),
                           static_cast<unsigned char*>(workspace) + WS_HEADER, stream);
}

extern "C" int stof_mask_classify_notify(const void* mask, int mask_dtype, int batch, int seq_len, int block_m, int block_n, int* full_row_ptr,
                                         int* part_row_ptr, int* load_row_ptr, float* nnz_percent, void* workspace, size_t workspace_bytes, void* header,
                                         const int* status_dev, stof_mask_notice* notice, unsigned long long stamp, void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (int rc = check_geometry(seq_len, block_m, block_n)) return rc;
    STOF_REQUIRE(mask && full_row_ptr && part_row_ptr && load_row_ptr && nnz_percent && workspace && header && notice, "mask_classify: null pointer");
    STOF_REQUIRE(mask_dtype == STOF_DTYPE_F16 || mask_dtype == STOF_DTYPE_F32, "mask_classify: mask_dtype must be f16 or f32");
    STOF_REQUIRE(batch >= 1 && batch <= 65535, "mask_classify: batch %d out of range", batch);
    STOF_REQUIRE(aligned16(mask) && aligned16(workspace) && aligned16(header), "mask_classify: mask, workspace and header must be 16-byte aligned");
    STOF_REQUIRE(seq_len / block_m <= 65535, "mask_classify: more than 65535 block rows");
    if (workspace_bytes < stof_mask_workspace_bytes(seq_len, block_m, block_n)) {
        set_error("mask_classify: workspace of %zu bytes, need %zu", workspace_bytes, stof_mask_workspace_bytes(seq_len, block_m, block_n));
        return STOF_E_WORKSPACE;
    }
    const Report report{nullptr, nnz_percent, 1.0f / static_cast<float>(static_cast<long long>(seq_len) * seq_len), status_dev, notice, stamp};
    return launch_classify(mask, mask_dtype, batch, seq_len, block_m, block_n, full_row_ptr, part_row_ptr, load_row_ptr, report,
                           Workspace(header), static_cast<unsigned char*>(workspace) + WS_HEADER, stream);
}

extern "C" int stof_mask_fill(const void* mask, int mask_dtype, int seq_len, int block_m, int block_n, const int* full_row_ptr,
                              const int* part_row_ptr, const int* load_row_ptr, int* full_col_idx, int* part_col_idx,
                              int* load_col_idx, void* part_block_mask, const void* workspace, size_t workspace_bytes, void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (int rc = check_geometry(seq_len, block_m, block_n)) return rc;
    STOF_REQUIRE(mask && full_row_ptr && part_row_ptr && load_row_ptr && workspace, "mask_fill: null pointer");
    STOF_REQUIRE(mask_dtype == STOF_DTYPE_F16 || mask_dtype == STOF_DTYPE_F32, "mask_fill: mask_dtype must be f16 or f32");
    STOF_REQUIRE(aligned16(mask) && (part_block_mask == nullptr || aligned16(part_block_mask)), "mask_fill: 16-byte alignment required");
    if (workspace_bytes < stof_mask_workspace_bytes(seq_len, block_m, block_n)) {
        set_error("mask_fill: workspace of %zu bytes, need %zu", workspace_bytes, stof_mask_workspace_bytes(seq_len, block_m, block_n));
        return STOF_E_WORKSPACE;
    }
    const int nbm = seq_len / block_m, nbn = seq_len / block_n;
    const unsigned char* cls = static_cast<const unsigned char*>(workspace) + WS_HEADER;
    // one block per partial tile as far as the device fills (their number is in device memory; a block takes every gridDim-th)
    const int index_blocks = (nbm + FILL_THREADS / 32 - 1) / (FILL_THREADS / 32);
    const long long tiles = static_cast<long long>(nbm) * nbn;
    const int tile_blocks = part_block_mask == nullptr ? 0 : static_cast<int>(tiles < 8 * sm_count() ? tiles : 8 * sm_count());
    LaunchConfig lc(dim3(static_cast<unsigned>(index_blocks + tile_blocks)), FILL_THREADS, 0, stream);
    STOF_CUDA(cudaLaunchKernelEx(&lc.cfg, mask_dtype == STOF_DTYPE_F32 ? fill_kernel<true> : fill_kernel<false>, mask, seq_len, block_m, block_n, cls,
                                 full_row_ptr, part_row_ptr, load_row_ptr, full_col_idx, part_col_idx, load_col_idx, static_cast<__half*>(part_block_mask),
                                 index_blocks));
    return STOF_OK;
}

// One call, nothing allocated: classify + fill with the scratch in the library's own device image (see the header).
extern "C" int stof_mask_compact_static(const void* mask, int mask_dtype, int batch, int seq_len, int block_m, int block_n,
                                        int* full_row_ptr, int* part_row_ptr, int* load_row_ptr, int* full_col_idx, int* part_col_idx,
                                        int* load_col_idx, long long col_capacity, void* part_block_mask, long long part_capacity,
                                        long long* counts, void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (int rc = check_geometry(seq_len, block_m, block_n)) return rc;
    STOF_REQUIRE(mask && full_row_ptr && part_row_ptr && load_row_ptr && full_col_idx && part_col_idx && load_col_idx && counts,
                 "mask_compact_static: null pointer");
    STOF_REQUIRE(mask_dtype == STOF_DTYPE_F16 || mask_dtype == STOF_DTYPE_F32, "mask_compact_static: mask_dtype must be f16 or f32");
    STOF_REQUIRE(batch >= 1 && batch <= 65535, "mask_compact_static: batch %d out of range", batch);
    STOF_REQUIRE(col_capacity >= 0 && part_capacity >= 0, "mask_compact_static: negative capacity");
    STOF_REQUIRE(aligned16(mask) && (part_block_mask == nullptr || aligned16(part_block_mask)), "mask_compact_static: 16-byte alignment required");
    const int nbm = seq_len / block_m, nbn = seq_len / block_n;
    STOF_REQUIRE(nbm <= 65535, "mask_compact_static: more than 65535 block rows");
    if (static_cast<long long>(nbm) * nbn > STATIC_MAX_TILES) {
        set_error("mask_compact_static: %d x %d blocks exceed the %d tiles the built-in scratch holds; use stof_mask_classify / stof_mask_fill "
                  "with a workspace of your own", nbm, nbn, STATIC_MAX_TILES);
        return STOF_E_LIMIT;
    }
    unsigned char* scratch = nullptr;
    if (int rc = static_scratch_address(&scratch)) return rc;
    unsigned char* cls = scratch + WS_HEADER;

    // the array keeps what the previous call left: the ticket and the count must start at zero
    STOF_CUDA(cudaMemsetAsync(scratch, 0, WS_HEADER, stream));
    const Report report{reinterpret_cast<unsigned long long*>(counts), nullptr, 0.f, nullptr, nullptr, 0};
    if (int rc = launch_classify(mask, mask_dtype, batch, seq_len, block_m, block_n, full_row_ptr, part_row_ptr, load_row_ptr, report, Workspace(scratch), cls,
                                 stream))
        return rc;
    int shares = (4 * sm_count() + nbm - 1) / nbm;
    if (shares < 1) shares = 1;
    if (shares > 8) shares = 8;
    if (part_block_mask == nullptr) shares = 1;
    const size_t smem = static_cast<size_t>(nbn) * sizeof(int);
    dim3 fgrid(nbm, shares);
    if (mask_dtype == STOF_DTYPE_F32)
        fill_bounded_kernel<true><<<fgrid, FILL_THREADS, smem, stream>>>(mask, seq_len, block_m, block_n, cls, full_row_ptr, part_row_ptr, load_row_ptr,
                                                                         full_col_idx, part_col_idx, load_col_idx, col_capacity,
                                                                         static_cast<__half*>(part_block_mask), part_capacity);
    else
        fill_bounded_kernel<false><<<fgrid, FILL_THREADS, smem, stream>>>(mask, seq_len, block_m, block_n, cls, full_row_ptr, part_row_ptr, load_row_ptr,
                                                                          full_col_idx, part_col_idx, load_col_idx, col_capacity,
                                                                          static_cast<__half*>(part_block_mask), part_capacity);
    STOF_CUDA(cudaGetLastError());
    return STOF_OK;
}
