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

// Whether the wide path is the faster one, by what a wave of each kernel costs in microseconds.  A wave of gemm_w4a4_kernel's 128 x 128 tiles over all SMs
// takes 3.4 + 7.4 (k / 1024), one of the wide kernel's 256 x 128 tiles 7.2 + 10.3 (k / 1024); fp32 rows leave the wide kernel element
// by element, which adds 26 to a wave.  The rewrite moves 1.5 bytes per element of both operands at 5 TB/s behind a launch of 4.
// The constants were fitted to 273 pairs, m 64 .. 8192, n 3072 .. 21504, k 64 .. 12288.  Both kernels have become faster since, the wide
// one more (14 % against 5 at [4608, 12288, 3072]), so the times above are too long for both and the line lies too far on the
// narrow side.  Both timed again at 269 pairs that lie within a third of it, with either loader of the scales: where it says wide, wide
// was the faster one (within 2 %); of those where it says narrow, 28 would have been 2 to 13 % faster wide.  Now, narrow / wide, us:
// [4608, 12288, 3072] 582 / 412; [1024, 12288, 3072] 152 / 119; [2048, 3072, 3072] 79 / 75 and [8192, 3072, 512] 79 / 72, both of which go
// narrow; [8192, 12288, 128] 190 / 167 likewise.  fp32: [4608, 12288, 3072] 625 / 766, [4608, 3072, 12288] 542 / 466.
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
