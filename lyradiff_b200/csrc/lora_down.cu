// Low-rank down projection of the W4A4 linear, act[m, 32] = x[m, k] * lora_down[32, k]^T (16-bit inputs, fp32 out), and in the same
// launch the int4 quantize of x.
//
// The reference computes this inside its int4 quantize kernel with one mma.sync tile per 64 columns and a
// floating-point atomic add per tile (src/lyradiff/kernels/w4a4_gemm/w4a4_gemm.cu:769-954), so the order of the 48
// partial sums changes from run to run.  Here one CTA owns 32 rows of x for the whole of K and accumulates in tensor
// memory in a fixed order, so the result is reproducible and no output has to be zeroed first.
//
// The product is formed transposed, D[r, j] = sum_k lora_down[r, k] * x[row0 + j, k]: tcgen05.mma needs M >= 64, and
// with the 32 rows of x on the N side 4608 tokens give 144 CTAs (one per SM) instead of 36.  The M side is the 32 rows
// of lora_down; the 96 rows behind them are whatever lies next in shared memory: the tiles of other stages, which the TMA
// may be writing while the MMA reads them.  They only reach accumulator lanes that nobody reads.
//
//   warp 0   TMA producer (lora_down tile and x tile, 32 rows x 128 B each, ring of 24 stages);
//            afterwards it reads accumulator lanes 0..31 and stores act
//   warp 1   MMA issuer; owns the tensor-memory allocation
//   warps 2-17  the int4 quantize of the same x tiles.  One stage holds, for each of the CTA's 32 rows,
//            exactly one group of 64 values (a 128-byte row of the swizzled tile), so x is read from memory once for
//            both results, as in the reference's fused kernel.  A warp takes a whole stage (four share one where K is short), four
//            rows at a time with eight lanes to a group (the results of int4_g64_kernel, bit for bit): a lane's eight columns stay the
//            same over the rows, so their smoothing factors are loaded and inverted once per stage.  A stage goes back to the
//            producer when the MMAs that read it and its quantizer warps are done.
//
// The quantizer's arithmetic bounds the kernel, so it has no division in the common case: 36 instructions an element with the
// IEEE divisions x / smooth, amax / 7 and 1 / s became 20.  Measured, [4608, 12288]: 118 us -> 58; [4608, 3072]: 29 -> 15; [100, 3072]
// f16: 80 -> under 18.
// All waits are bounded; a timeout sets the status word and the block leaves.
#include "common.cuh"
#include "sm100_ptx.cuh"

namespace lyraq {

using namespace sm100;

int make_tmap_bytes_2d(CUtensorMap* map, const void* base, uint64_t rows, uint64_t k_bytes, uint64_t row_stride_bytes,
                       uint32_t box_rows, uint32_t box_bytes, bool swizzle128);  // gemm_dense.cu

namespace lora {

constexpr int kRank      = 32;
constexpr int kRows      = 32;                    // rows of x per CTA (the MMA's N)
constexpr int kBlockKB   = 128;                   // bytes of K per stage = 64 elements
constexpr int kStages    = 24;
constexpr int kTile      = kRows * kBlockKB;      // 4 KB: a stage's rows of lora_down (kRank == kRows), or of x
constexpr int kXOffset   = kStages * kTile;       // all lora_down tiles, then all x tiles: the 16 KB an MMA's A descriptor spans from
static_assert(kXOffset >= 128 * kBlockKB, "");    // the last lora_down tile stay inside the allocation
constexpr int kBarOffset = 2 * kStages * kTile;
constexpr int kSmemTotal = kBarOffset + 512 + 1024;
constexpr int kQuantWarps = 16;
constexpr int kThreads   = 64 + 32 * kQuantWarps;

struct Params {
    float*        act;   // [m, 32]
    int           m, k;
    unsigned int* status;
    uint32_t*     q;        // [m, k / 8]: eight nibbles per word
    float*        q_scale;  // [m, k / 64]
    const float*  smooth;   // [k] or null
};

__device__ __forceinline__ float max_nan(float a, float b)
{
    float d;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
    return d;
}
__device__ __forceinline__ float max3_nan(float a, float b, float c)
{
    float d;
    asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// Eight consecutive values of a group of 64 per lane, eight lanes to a group, R groups at once: nibbles and scale as
// int4_g64_quantize8 gives them for v = x / smooth, without a division.  A quotient of floats is q + (x - q b) y with y = 1 / b
// correctly rounded, q = x y and the remainder exact in an fma: correctly rounded itself (Markstein, IBM J. Res. Dev. 34, 1990) as
// long as nothing leaves the exponent range.  So x / smooth takes the columns' reciprocals (ry; ns = -smooth), amax / 7 that of 7.
// The codes come from v times an approximate reciprocal of s (|v / s| <= 7, so it is off by 1e-6 at most); where a quotient lies within 6.1e-5
// of a half-integer the division decides, as in quant8_s8_inrange.  `fits` says that every |smooth| lies within 2^-20 .. 2^20; with
// amax within 2^-40 .. 2^40 everything that can reach a code or the scale is then far from the ends of the range (an x below 2^-64
// in such a group is code 0 however it is rounded).  Returns false, for the whole warp, if some lane has a group outside that, or one with
// a NaN or an infinity: the caller then divides.
template<int R>
__device__ __forceinline__ bool int4_g64_quantize8_fast(const float2 (&x)[R][4], const float2 (&ry)[4], const float2 (&ns)[4], bool smooth, bool fits,
                                                        uint32_t (&w)[R], float (&s)[R])
{
    float2 v[R][4];
    float  amax[R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            v[i][j] = x[i][j];
            if (smooth) {
                const float2 q = mul_f32x2(x[i][j], ry[j]);
                v[i][j]        = fma_f32x2(fma_f32x2(q, ns[j], x[i][j]), ry[j], q);
            }
        }
        const float a = max3_nan(fabsf(v[i][0].x), fabsf(v[i][0].y), fabsf(v[i][1].x));
        const float b = max3_nan(fabsf(v[i][1].y), fabsf(v[i][2].x), fabsf(v[i][2].y));
        amax[i]       = max3_nan(max_nan(a, b), fabsf(v[i][3].x), fabsf(v[i][3].y));
    }
#pragma unroll
    for (int m = 1; m < 8; m <<= 1) {
#pragma unroll
        for (int i = 0; i < R; ++i) {
            amax[i] = max_nan(amax[i], __shfl_xor_sync(0xffffffffu, amax[i], m));
        }
    }
    bool ok = fits;
#pragma unroll
    for (int i = 0; i < R; ++i) {
        ok = ok && (amax[i] == 0.0f || (amax[i] >= 0x1p-40f && amax[i] <= 0x1p40f));
    }
    if (!__all_sync(0xffffffffu, ok)) {
        return false;
    }
#pragma unroll
    for (int i = 0; i < R; ++i) {
        constexpr float kSeventh = 1.0f / 7.0f;
        const float     q        = amax[i] * kSeventh;
        s[i]                     = fmaf(fmaf(-7.0f, q, amax[i]), kSeventh, q);
        float r;
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(fmaxf(s[i], 0x1p-50f)));   // an all-zero group: zeros times anything
        const float2 mg = make_float2(12582912.0f, 12582912.0f), r2 = make_float2(r, r), m1 = make_float2(-1.0f, -1.0f);
        uint32_t     b[8];
        float        d[8];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float2 t = fma_f32x2(v[i][j], r2, mg);
            const float2 e = fma_f32x2(v[i][j], r2, fma_f32x2(t, m1, mg));   // v / s - its nearest integer
            b[2 * j]       = __float_as_uint(t.x);
            b[2 * j + 1]   = __float_as_uint(t.y);
            d[2 * j]       = fabsf(e.x);
            d[2 * j + 1]   = fabsf(e.y);
        }
        const float d0 = max3_nan(d[0], d[1], d[2]), d1 = max3_nan(d[3], d[4], d[5]);
        if (max3_nan(max_nan(d0, d1), d[6], d[7]) > 0.5f - 6.1e-5f) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                b[2 * j]     = (uint32_t)f32_to_s8(v[i][j].x / s[i]);
                b[2 * j + 1] = (uint32_t)f32_to_s8(v[i][j].y / s[i]);
            }
        }
        // low nibbles of the eight words, element j at bits 4 j: pairs first (b0 | b1 << 4 in byte 0), then the bytes together
        const uint32_t p0 = (b[0] & 0xFu) | ((b[1] & 0xFu) << 4), p1 = (b[2] & 0xFu) | ((b[3] & 0xFu) << 4);
        const uint32_t p2 = (b[4] & 0xFu) | ((b[5] & 0xFu) << 4), p3 = (b[6] & 0xFu) | ((b[7] & 0xFu) << 4);
        w[i]              = __byte_perm(__byte_perm(p0, p1, 0x0040), __byte_perm(p2, p3, 0x0040), 0x5410);
    }
    return true;
}

// SHARE quantizer warps take a stage together, its rows dealt out: with fewer stages than warps most of them would have nothing to do.
template<int SHARE, typename T>
__global__ void __launch_bounds__(kThreads, 1)
lora_down_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_down, const Params p)
{
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t*       gen_base  = smem_raw + (smem_base - smem_u32(smem_raw));
    const uint32_t bars      = smem_base + kBarOffset;
    auto full_bar  = [&](int s) { return bars + 8u * s; };
    auto empty_bar = [&](int s) { return bars + 8u * (kStages + s); };
    const uint32_t done_bar   = bars + 8u * (2 * kStages);
    uint32_t*      tmem_slot  = reinterpret_cast<uint32_t*>(gen_base + kBarOffset + 8 * (2 * kStages + 1));
    volatile int*  abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = warp_index();
    const int lane = threadIdx.x & 31;

    grid_launch_dependents();
    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1 + SHARE);   // the MMAs' commit, and the stage's quantizer warps
        }
        mbar_init(done_bar, 1);
        *abort_flag = 0;
        fence_barrier_init();
        prefetch_tensormap(&tmap_x);
        prefetch_tensormap(&tmap_down);
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(tmem_slot), 32);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    grid_dependency_wait();

    const int num_kb = (p.k * 2 + kBlockKB - 1) / kBlockKB;
    const int row0   = blockIdx.x * kRows;

    auto give_up = [&](unsigned code) {
        report_timeout(p.status, code);
        *abort_flag = 1;
    };

    if (warp == 0) {
        int      stage = 0, issued = 0;
        uint32_t phase = 0;
        for (int kb = 0; kb < num_kb; ++kb) {
            // many stages lie between this warp, the issuer and the quantizers, so the two of them look rarely: their polling would
            // take a fifth of the issue slots
            if (!mbar_wait_lazy(empty_bar(stage), phase ^ 1u, abort_flag)) {
                give_up(0x2100u | (unsigned)stage);
                break;
            }
            if (elect_one()) {
                mbar_arrive_expect_tx(full_bar(stage), (uint32_t)(2 * kTile));
                tma_load_2d(smem_base + stage * kTile, &tmap_down, full_bar(stage), kb * kBlockKB, 0);
                tma_load_2d(smem_base + kXOffset + stage * kTile, &tmap_x, full_bar(stage), kb * kBlockKB, row0);
            }
            ++issued;
            if (++stage == kStages) {
                stage = 0;
                phase ^= 1u;
            }
        }
        // no load may still be in flight when the block leaves: walk back over the last slots that were filled
        for (int i = 0; i < kStages && i < issued; ++i) {
            if (stage == 0) {
                stage = kStages;
                phase ^= 1u;
            }
            --stage;
            const uint64_t t0 = global_timer_ns();
            while (!mbar_try_wait(full_bar(stage), phase)) {
                if (global_timer_ns() - t0 > kWaitLimitNs) {
                    report_timeout(p.status, 0x2400u | (unsigned)stage);
                    break;
                }
            }
        }
        __syncwarp();
        // every load has landed once the last MMA, which waited for it, has completed
        if (mbar_wait_warp(done_bar, 0u, abort_flag)) {
            tc_fence_after_sync();
            uint32_t d[32];
            tmem_ld_32x32(tmem_base, d);  // lane r of the warp = rank r; column j = row row0 + j
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < kRows; ++j) {
                if (row0 + j < p.m) {
                    p.act[(size_t)(row0 + j) * kRank + lane] = __uint_as_float(d[j]);
                }
            }
        } else if (lane == 0) {
            report_timeout(p.status, 0x2300u);
        }
    } else if (warp >= 2) {
        // ------------------------------------------------------------------ int4 quantize of the staged x tiles
        const int  part   = lane & 7;                 // which 8 values of the group of 64
        const int  sub    = lane >> 3;                // which of a pass's 4 rows
        const bool smooth = p.smooth != nullptr;
        const size_t q_pitch = (size_t)(p.k >> 3), s_pitch = (size_t)(p.k >> 6);
        const int    r0      = sub + (SHARE > 1 ? 8 * ((warp - 2) % SHARE) : 0);   // this lane's first row of a stage
        uint32_t*    q_out   = p.q + (size_t)(row0 + r0) * q_pitch + part;
        float*       s_out   = p.q_scale + (size_t)(row0 + r0) * s_pitch;
        for (int kb = (warp - 2) / SHARE; kb < num_kb; kb += kQuantWarps / SHARE) {
            const int      stage = kb % kStages;
            const uint32_t phase = (uint32_t)((kb / kStages) & 1);
            float2         ry[4], ns[4];
            bool           fits = true;
            if (smooth) {
                const float4 s0 = ld_f32x4(reinterpret_cast<const float4*>(p.smooth + kb * 64 + part * 8));
                const float4 s1 = ld_f32x4(reinterpret_cast<const float4*>(p.smooth + kb * 64 + part * 8 + 4));
                ns[0] = make_float2(-s0.x, -s0.y); ns[1] = make_float2(-s0.z, -s0.w);
                ns[2] = make_float2(-s1.x, -s1.y); ns[3] = make_float2(-s1.z, -s1.w);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float lo = fminf(fabsf(ns[j].x), fabsf(ns[j].y)), hi = fmaxf(fabsf(ns[j].x), fabsf(ns[j].y));
                    fits           = fits && lo >= 0x1p-20f && hi <= 0x1p20f && ns[j].x == ns[j].x && ns[j].y == ns[j].y;
                    ry[j]          = make_float2(-1.0f / ns[j].x, -1.0f / ns[j].y);
                }
            }
            if (!mbar_wait_warp(full_bar(stage), phase, abort_flag)) {
                give_up(0x2500u | (unsigned)stage);
                break;
            }
            const uint8_t* xt = gen_base + kXOffset + stage * kTile;   // 32 rows x 128 B, 128-byte swizzle
            uint32_t* qrow = q_out + (size_t)kb * 8;
            float*    srow = s_out + kb;
#pragma unroll 1
            for (int r = r0; r < kRows; r += 8 * SHARE) {   // this lane's rows r and r + 4: two independent chains
                float2 v[2][4];
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const Vec16 raw = *reinterpret_cast<const Vec16*>(xt + (r + 4 * i) * 128 + ((part ^ ((r + 4 * i) & 7)) << 4));
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        v[i][j] = Pair<T>::to_f32(raw.w[j]);
                    }
                }
                uint32_t w[2];
                float    sc[2];
                if (!int4_g64_quantize8_fast<2>(v, ry, ns, smooth, fits, w, sc)) {
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        float e[8];
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            e[j] = (j & 1) ? v[i][j >> 1].y : v[i][j >> 1].x;
                            if (smooth) {
                                e[j] /= (j & 1) ? -ns[j >> 1].y : -ns[j >> 1].x;
                            }
                        }
                        w[i] = int4_g64_quantize8(e, sc[i]);
                    }
                }
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    if (row0 + r + 4 * i < p.m) {
                        qrow[4 * i * q_pitch] = w[i];
                        if (part == 0) {
                            srow[4 * i * s_pitch] = sc[i];
                        }
                    }
                }
                qrow += 8 * SHARE * q_pitch;
                srow += 8 * SHARE * s_pitch;
            }
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(empty_bar(stage));
            }
        }
    } else if (warp == 1) {
        int      stage = 0;
        uint32_t phase = 0;
        const uint32_t idesc = umma_idesc(1u, TypeTag<T>::value == LYRAQ_BF16 ? 1u : 0u, 128, kRows);
        for (int kb = 0; kb < num_kb; ++kb) {
            if (!(SHARE > 1 ? mbar_wait_warp(full_bar(stage), phase, abort_flag) : mbar_wait_lazy(full_bar(stage), phase, abort_flag))) {
                give_up(0x2200u | (unsigned)stage);
                break;
            }
            tc_fence_after_sync();
            const uint64_t adesc = umma_desc_k_sw128(smem_base + stage * kTile);
            const uint64_t bdesc = umma_desc_k_sw128(smem_base + kXOffset + stage * kTile);
            if (elect_one()) {
#pragma unroll
                for (int ks = 0; ks < kBlockKB / 32; ++ks) {
                    mma_f16(tmem_base, adesc + (uint64_t)(2 * ks), bdesc + (uint64_t)(2 * ks), idesc, (kb > 0 || ks > 0) ? 1u : 0u);
                }
                tc_commit(empty_bar(stage));
                if (kb == num_kb - 1) {
                    tc_commit(done_bar);
                }
            }
            if (++stage == kStages) {
                stage = 0;
                phase ^= 1u;
            }
        }
    }

    tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, 32);
    }
}

template<int SHARE, typename T> static int launch(unsigned grid, const CUtensorMap& tx, const CUtensorMap& td, const Params& p, cudaStream_t stream)
{
    static bool smem_raised[64] = {};
    const int   st = raise_dynamic_smem_once(lora_down_kernel<SHARE, T>, (int)kSmemTotal, smem_raised,
                                           "cudaFuncSetAttribute(lora_down_kernel, dynamic shared memory)");
    if (st != LYRAQ_OK) {
        return st;
    }
    return cuda_status(launch_kernel(lora_down_kernel<SHARE, T>, grid, (unsigned)kThreads, (size_t)kSmemTotal, stream, 1u,
                                     tx, td, p),
                       "cudaLaunchKernelEx(lora_down_kernel)");
}

}  // namespace lora

// The reference's fused_quantized_and_lora_down_simple (w4a4_gemm.cu:769-954) as ONE launch over one read of x: the int4 group-64
// quantization of x / smooth (packed nibbles q [m, k / 2 bytes], fp32 scales q_scale [m, k / 64]) and act[m, 32] (fp32) =
// x[m, k] * down[32, k]^T; x and down of the same 16-bit type, k a multiple of 64.
int launch_quant_int4_lora_down(uint8_t* q, float* q_scale, float* act, const void* x, const void* down, const float* smooth, int dtype,
                                size_t m, size_t k, cudaStream_t stream)
{
    if (q == nullptr || act == nullptr || x == nullptr || down == nullptr) {
        return LYRAQ_ERR_INVALID_ARG;
    }
    if (dtype != LYRAQ_BF16 && dtype != LYRAQ_F16) {
        return LYRAQ_ERR_UNSUPPORTED;
    }
    if (!aligned16(x) || !aligned16(down) || (reinterpret_cast<uintptr_t>(act) & 3u) != 0) {
        return LYRAQ_ERR_INVALID_ARG;
    }
    if (q_scale == nullptr || (reinterpret_cast<uintptr_t>(q) & 3u) != 0 || (smooth != nullptr && !aligned16(smooth))) {
        return LYRAQ_ERR_INVALID_ARG;
    }
    if ((k & 63) != 0 || k == 0 || k > 0x3fffffffu || m > 0x7fffffffu) {
        return LYRAQ_ERR_UNSUPPORTED;
    }
    lora::Params p{};
    p.act     = act;
    p.m       = (int)m;
    p.k       = (int)k;
    p.q       = reinterpret_cast<uint32_t*>(q);
    p.q_scale = q_scale;
    p.smooth  = smooth;
    p.status  = status_word_ptr();
    if (p.status == nullptr) {
        return LYRAQ_ERR_CUDA;
    }
    CUtensorMap tx, td;
    int st = make_tmap_bytes_2d(&tx, x, (uint64_t)m, (uint64_t)k * 2, (uint64_t)k * 2, lora::kRows, lora::kBlockKB, true);
    if (st != LYRAQ_OK) {
        return st;
    }
    st = make_tmap_bytes_2d(&td, down, (uint64_t)lora::kRank, (uint64_t)k * 2, (uint64_t)k * 2, lora::kRank, lora::kBlockKB, true);
    if (st != LYRAQ_OK) {
        return st;
    }
    const unsigned grid = (unsigned)((m + lora::kRows - 1) / lora::kRows);
    const bool bf16 = dtype == LYRAQ_BF16;
    // Up to half as many stages as quantizer warps: four warps to a stage, and an issuer that polls without pauses.  With a warp to a stage
    // [4608, 64] took 4.4 us, so 2.9; [512, 128] 4.3 / 2.9; [4608, 512] 5.4 / 5.1.
    if (k <= 64 * lora::kQuantWarps / 2) {
        return bf16 ? lora::launch<4, __nv_bfloat16>(grid, tx, td, p, stream) : lora::launch<4, __half>(grid, tx, td, p, stream);
    }
    return bf16 ? lora::launch<1, __nv_bfloat16>(grid, tx, td, p, stream) : lora::launch<1, __half>(grid, tx, td, p, stream);
}

}  // namespace lyraq
