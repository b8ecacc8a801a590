// The prefill GEMM for pairs of SMs (gemm_pair.cu), as the dispatch sees it.
#pragma once

#include "common.cuh"

namespace b200gptq {

struct GemmPairPlan {
    int rows;          // of x per tile: a multiple of 32 up to 256
    int splits;        // runs of K (one tile per pair of SMs where there are several)
};
GemmPairPlan gemm_pair_plan(int M, int N, int K, int few, bool one_run = false);
size_t gemm_pair_partial_bytes(int M, int N, GemmPairPlan plan);
int gemm_pair_dispatch(const __half* x, const int32_t* qweight, const int32_t* qzeros, const __half* scales, const int32_t* g_idx,
                       const __half* bias, __half* y, int M, int K, int N, int bits, int group_size, GemmPairPlan plan,
                       unsigned int* status, float* partial, cudaStream_t stream);

}  // namespace b200gptq
