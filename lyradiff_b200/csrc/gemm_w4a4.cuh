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
    int           scale_tma;     // wide kernel: both scale arrays can be addressed by TMA
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

// Whether the wide path is the faster one, in microseconds of each kernel.  A wave of gemm_w4a4_kernel's 128 x 128 tiles over all SMs
// takes 3.4 + 7.4 (k / 1024), one of the wide kernel's 256 x 128 tiles 7.2 + 10.3 (k / 1024); fp32 rows leave the wide kernel element
// by element, which adds 26 to a wave.  The rewrite moves 1.5 bytes per element of both operands at 5 TB/s behind a launch of 4.
// (Both kernels have become faster by about the same share since, 10 to 14 %; the line was left where it lies.)
// Fitted to 273 measured pairs, m 64 .. 8192, n 3072 .. 21504, k 64 .. 12288: on none of them is the choice more than 2 % slower than
// the other one.  16-bit outputs: [4608, 12288, 3072] 24 waves 616 us against 12 waves 477; [1024, 12288, 3072] 6 / 3 waves 159 / 137;
// [2048, 3072, 3072] 3 / 2 waves 84 / 88; [8192, 3072, 512] 11 / 6 waves 80 / 83.  fp32: [4608, 12288, 3072] 655 / 837,
// [4608, 3072, 12288] 574 / 522.
inline bool wide_pays(size_t m, size_t n, size_t k, int sms, bool fp32_out)
{
    const size_t u      = sms > 0 ? (size_t)sms : 148;
    const size_t narrow = ((m + 127) / 128 * ((n + 127) / 128) + u - 1) / u;
    const size_t wide   = ((m + 255) / 256 * ((n + 127) / 128) + u - 1) / u;
    const double ki     = (double)k / 1024.0;
    return (double)wide * (7.2 + 10.3 * ki + (fp32_out ? 26.0 : 0.0)) + 4.0 + 3.1e-4 * (double)(m + n) * ki < (double)narrow * (3.4 + 7.4 * ki);
}

// Workspace of the wide path: both operands at one byte per element, and the low-rank activation at 16 bits.
size_t wide_workspace_bytes(size_t m, size_t n, size_t k);
int    launch_wide(Params p, const uint8_t* A, const uint8_t* B, void* workspace, int sms, cudaStream_t stream);

}  // namespace w4
}  // namespace lyraq
