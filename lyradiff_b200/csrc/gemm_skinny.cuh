// Interface between the dense GEMM entry points and the few-token FP8 kernel (gemm_skinny.cu).
#pragma once

#include <cuda_runtime.h>

namespace lyraq {

struct SkinnyParams {
    int           M, N, K;
    int           num_kb, splits;             // filled in by launch_gemm_skinny
    void*         C;                          // [M, N] of c_dtype, F16, BF16 or F32
    int           c_dtype;
    const float*  s_x;
    const float*  s_w;
    float         alpha, beta;
    const void*   bias;                       // [N] of c_dtype or null
    const void*   residual;                   // [M, N] of c_dtype or null
    int           gelu;
    unsigned int* status;
    unsigned long long wait_limit_ns;         // filled in by launch_gemm_skinny: longest a single wait may last,
    int           stalled_rank;               // and the rank of each cluster whose producer loads nothing (test hook; -1: none)
};

constexpr int kSkinnyRows = 16;   // most rows it takes

int launch_gemm_skinny(const void* X, const void* W, SkinnyParams p, int sms, cudaStream_t stream);

}  // namespace lyraq
