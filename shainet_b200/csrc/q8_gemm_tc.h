// Launch interface of the tensor-core Q8_0 matrix product (several activation rows) and of the row kernels around it.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "common.cuh"

namespace shainet {

// Tensor maps of one Q8_0 weight, made once per weight: int8 [N, K] and scales [N, K/32].
struct Q8Maps {
    CUtensorMap w, s;
    int N = 0, K = 0;
    bool ok = false;
};
// false (and m->ok == false) where the weight cannot take this path: K no multiple of 128, or misaligned arrays.
bool q8_gemm_maps(Q8Maps* m, const signed char* q, const float* scales, int N, int K);

// Where the columns of a product go: up to three row-major outputs beside each other (q | k | v); a launch whose
// contraction is split writes split z at ptr + z * split_stride (one segment then) for the kernel behind it to add up.
struct Q8GemmOut {
    float* ptr[3];
    int begin[3];          // first column of the segment
    int pitch[3];
    int segments;
    size_t split_stride;
    const float* residual; // nullable, one segment only: added to the product
};

struct Q8GemmArgs {
    const __nv_bfloat16* planes;   // [3][M][K]
    const Q8Maps* w[2];            // the second (nullable) weight's columns follow the first's
    int M, K;
    Q8GemmOut out;
    AttnStatus* status;
};

struct Q8GemmPlan {
    int nt;       // tokens per tile
    int splits;   // of the contraction
};
Q8GemmPlan q8_gemm_plan(int M, int K, int n0, int n1, int sm_count);
cudaError_t launch_q8_gemm_tc(const Q8GemmArgs& g, const Q8GemmPlan& plan, int sm_count, cudaStream_t s);

// One token row after another: splits == 0: row = x; otherwise row = residual + sum over splits of x, also stored to h.
// Then RMSNorm with gamma (nullable; K up to 51200) and the split into three bfloat16 planes [3][M][K].
struct Q8RowsArgs {
    const float* x;
    int splits;
    size_t split_stride;
    const float* residual;   // nullable
    float* h;                // nullable
    const float* gamma;      // nullable
    double eps;
    __nv_bfloat16* planes;
    int M, K;
};
cudaError_t launch_q8_rows(const Q8RowsArgs& a, cudaStream_t s);
// planes of silu(gate) * up; gu is [splits][M][2 * ffn], gate columns first.
cudaError_t launch_q8_swiglu(const float* gu, int splits, size_t split_stride, int M, int ffn, __nv_bfloat16* planes, int sm_count, cudaStream_t s);
// Sum of the splits [splits][M][N] into `out`.
cudaError_t launch_q8_reduce(const float* part, int splits, size_t split_stride, int M, int N, const Q8GemmOut& out, cudaStream_t s);

}  // namespace shainet
