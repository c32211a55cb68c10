// What the two W4A4 GEMM kernels share: gemm_w4a4.cu (any call) and gemm_w4a4_wide.cu (many rows, with a workspace).
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace lyraq {
namespace w4 {

struct Params {
    int           M, N, K, G;  // G = K / 64
    int           m_tiles, n_tiles;
    const float*  sa;
    const void*   sb;
    int           sb_is_f16;
    int           scale_vec_ok;  // G % 4 == 0 and 16-byte aligned scale arrays: 16-byte scale loads are legal
    void*         D;
    int           c_dtype;
    const void*   bias;
    const void*   residual;
    int           gelu;
    int           round_each;    // round to D's type after every epilogue step (the reference's separate 16-bit kernels)
    const void*   lora_act;      // [M, 32], fp32 or already of D's 16-bit type, or null
    int           lora_act_is_f32;
    const void*   lora_up;       // [N, 32] of D's 16-bit type or null
    unsigned int* status;
};

constexpr int kLoraRank = 32;

// Whether the wide path is the faster one.  In units of one wave of gemm_w4a4_kernel's 128 x 128 tiles over all SMs (26.6 us at
// K = 3072): a wave of the wide kernel's 256 x 128 tiles takes 1.47 (38.5 us measured, not 2), the rewrite of the operands
// (n + m) k * 1.5 bytes at 5 TB/s and 4 us of launch.  Measured: [4608, 12288, 3072] 24 waves 638 us against 12 waves 489 us;
// [1024, 12288, 3072] 6 / 3 waves 165 / 137 us; [2048, 3072, 3072] 3 / 2 waves 84 / 89 us.
inline bool wide_pays(size_t m, size_t n, size_t k, int sms)
{
    const size_t u      = sms > 0 ? (size_t)sms : 148;
    const size_t narrow = ((m + 127) / 128 * ((n + 127) / 128) + u - 1) / u;
    const size_t wide   = ((m + 255) / 256 * ((n + 127) / 128) + u - 1) / u;
    return 1.47 * (double)wide + 3.5e-5 * (double)(m + n) + 460.0 / (double)k < (double)narrow;
}

// Workspace of the wide path: both operands at one byte per element, and the low-rank activation at 16 bits.
size_t wide_workspace_bytes(size_t m, size_t n, size_t k);
int    launch_wide(Params p, const uint8_t* A, const uint8_t* B, void* workspace, int sms, cudaStream_t stream);

}  // namespace w4
}  // namespace lyraq
