// The GEMM kernel for shapes with few output tiles (gemm_split.cu), as the dispatch in gemm_tc.cu calls it.
#pragma once
#include <cuda_fp16.h>
#include "stof_host.h"

namespace stof {

struct SplitCall {
    const void* a;
    long long lda;
    const CUtensorMap* map_w;          // boxes of 64 x 64
    const __half *bias, *residual;
    long long ldr;
    __half* c;
    long long ldc;
    int m, n, k;
    int split;                         // thread blocks that share a tile's K: 1, 2 or 4, at most ceil(k / 128)
    int epilogue;
    int* status;
    cudaStream_t stream;
};
// tiles of bm x bn: 64 x 64, 128 x 64 or 128 x 128
int gemm_split_dispatch(const SplitCall& x, int bm, int bn);

struct SplitLnCall {
    const void* a;
    long long lda;
    const CUtensorMap* map_w;
    const __half *bias, *residual;
    long long ldr;
    const __half *gamma, *beta;
    float eps;
    __half* c;
    long long ldc;
    int m, n, k;
    int* status;
    cudaStream_t stream;
};
// the same with the LayerNorm in its epilogue (gemm_split_ln.cu); *done = 0, and nothing launched, when the row blocks would not
// all run at once
int gemm_split_ln_dispatch(const SplitLnCall& x, int* done);

// gemm_tc.cu: rounds of tiles of the GEMM without LayerNorm, for the choice between one kernel and two
long long gemm_rounds(int m, int n, int k, int epilogue);

}  // namespace stof
