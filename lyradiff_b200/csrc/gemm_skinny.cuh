// Interface between the dense GEMM entry points and the few-token FP8 kernel (gemm_skinny.cu).
#pragma once

#include <cuda_runtime.h>

namespace lyraq {

struct SkinnyParams {
    void*         C;                  // [M, N] of c_dtype, F16, BF16 or F32
    const float*  s_x;
    const float*  s_w;
    const void*   bias;               // [N] of c_dtype or null
    const void*   residual;           // [M, N] of c_dtype or null
    unsigned int* status;
    int           M, N, K;
    int           c_dtype;
    float         alpha, beta;
    int           gelu;
    int           num_kb, splits;     // filled in by launch_gemm_skinny, as are
    int           stalled_rank;       // the rank of each cluster whose producer loads nothing (test hook; -1: none)
    unsigned int  wait_limit_ms;      // and the longest a single wait may last
};

constexpr int kSkinnyRows = 16;   // most rows it takes

int launch_gemm_skinny(const void* X, const void* W, SkinnyParams p, int sms, cudaStream_t stream);

}  // namespace lyraq
