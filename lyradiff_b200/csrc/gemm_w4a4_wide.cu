// W4A4 GEMM for many rows: the operands are expanded from nibbles to bytes once, in memory, instead of once per tile.
//
//   D[m,n] = T( epi( sum_g (float(sum_{k in g} a[m,k]*b[n,k]) * sa[m,g]) * sb[n,g] + lora + bias[n] ) + R[m,n] )
//
// gemm_w4a4_kernel (gemm_w4a4.cu) expands a tile's nibbles in shared memory, which a 4608-row problem repeats 36 times for every
// weight, and its integer MMA leaves an int32 -> fp32 conversion per element and group to the CUDA cores.  Here
//   * w4_expand_kernel rewrites both packed operands as e4m3 codes (-8 .. 7 are exact) in the caller's workspace: one pass
//     over n k / 2 + m k / 2 bytes in and twice that out, a few microseconds against hundreds of the GEMM;
//   * the GEMM multiplies them with tcgen05.mma kind::f8f6f4.  A group's dot product is an integer of at most 64 * 64 = 4096 in
//     magnitude, which the fp32 accumulator holds exactly, so the partial reaches the CUDA cores as a float and the result is
//     gemm_w4a4_kernel's bit for bit;
//   * with no expansion in the way a tile is 256 x 128 and the drain warps do nothing but rescale.
// The floor is that rescale: acc = fma(p * sa, sb, acc) in group order is a multiply and an fma per output and group, 2 M N K / 64
// fp32 operations over 128 lanes per clock and SM (555 clocks per group of a tile at the measured rate of the packed forms).
//
// 384 threads, one persistent CTA per SM; registers are moved from the first warpgroup to the drain:
//   warp 0       TMA producer: A (256 x 128 B) and B (128 x 128 B) tiles of one K block = 2 groups, ring of 3 stages
//   warps 1, 3   MMA issuers of the even and the odd steps: a group's two products [128 x 128] (rows 0-127 and 128-255) into the
//                step's half of tensor memory, one commit per group; one thread that issued all of them took 900 clocks a group
//   warp 2       scale loader: every two K blocks (4 groups) it puts sa[m, g] and sb[n, g] of the tile into shared memory as
//                [g][row] (ring of 2 slots), by way of TMA where the arrays allow that; it also owns tensor memory
//   warps 4-11   drain: warp w reads TMEM lanes 32 * (w % 4) .., 64 columns, of both row halves, so a thread owns two half rows;
//                final epilogue
// Measured with the rewrite included: [4608, 12288, 3072] 416 us, [4608, 3072, 12288] 381, [1500, 9216, 3072] 115; 430, 406 and 120
// with scales loaded by the lanes (16 bytes of 32 rows per instruction, a shared-memory-pipe pass each); 484, 441 and 131 with, besides, a
// drain that asked for a group's scales and barrier when it came to it, and issuers and producer waiting as single lanes.  About 1060
// clocks a group; the drain alone -- loads from tensor memory, column scales, arithmetic -- takes 674 of them.
//
// What shaped the drain (clocks per group and SM, [4608, 12288, 3072]): a broadcast 16-byte shared load takes the SM's one
// shared-memory pipe two clocks, so with one row per thread the column scales cost 525 of them beside 384 for the operands of the
// MMAs; two rows per thread halve that.  (The 16x256b form of the tensor-memory load, where a thread needs few column scales, reads
// at a quarter of the speed of the 32x32b form.)  Loads from tensor memory run one piece ahead of the arithmetic, and the barrier of
// the next group is tested two pieces before it is needed (with test_wait: try_wait stops the warp, 449 us instead of 404).
// The low-rank branch is one more K block per tile: T(act) [m, 32] and up [n, 32] are 64-byte rows that TMA pads to 128 with
// zeros, two kind::f16 MMAs put the product into the next partial buffer and the drain adds it after the last group.
// All waits are bounded (see sm100_ptx.cuh); a timeout sets the status word and every role exits.
#include "common.cuh"
#include "sm100_ptx.cuh"
#include "gemm_w4a4.cuh"

namespace lyraq {

using namespace sm100;

// defined in gemm_dense.cu
int make_tmap_bytes_2d(CUtensorMap* map, const void* base, uint64_t rows, uint64_t k_bytes, uint64_t row_stride_bytes,
                       uint32_t box_rows, uint32_t box_bytes, bool swizzle128);
int make_tmap_store(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint64_t ld, int elem_bytes, bool wide = false);

namespace w4 {

// ---------------------------------------------------------------------------------------------- expansion
// prmt.b32: each selector nibble picks a byte of {b, a}; its bit 3 replicates the sign of that byte over the result byte
// (the __byte_perm intrinsic clears that bit, at the price of an AND)
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t selector)
{
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(selector));
    return d;
}

// Four packed nibbles (two's complement, low 16 bits of `sel` with the sign bits cleared) -> four e4m3 codes: one table for the
// values 0 .. 7, one for -8 .. -1, and a byte mask made of the sign bits picks between them.
__device__ __forceinline__ uint32_t nibbles_to_e4m3(uint32_t sel, uint32_t neg_mask)
{
    const uint32_t pos = prmt(0x44403800u, 0x4E4C4A48u, sel);
    const uint32_t neg = prmt(0xCACCCED0u, 0xB8C0C4C8u, sel);
    return (pos & ~neg_mask) | (neg & neg_mask);
}

// Eight nibbles of one word -> eight e4m3 codes in the same order.
__device__ __forceinline__ uint2 expand8(uint32_t w)
{
    const uint32_t w4  = w << 4;
    const uint32_t sel = w & 0x77777777u;
    uint2          r;
    r.x = nibbles_to_e4m3(sel, prmt(w4, w, 0xD9C8u));
    r.y = nibbles_to_e4m3(sel >> 16, prmt(w4, w, 0xFBEAu));
    return r;
}

struct ExpandParams {
    const uint4* src[2];     // packed B, packed A
    uint4*       dst[2];     // e4m3 codes
    size_t       chunks[2];  // 16-byte pieces of each source
    const float* act;        // [m, 32] fp32 low-rank activation to be rounded to T, or null
    uint32_t*    act16;
    size_t       act_pairs;
    int          act_bf16;
};

// Bound by memory: 16 bytes in and 32 out per piece, two independent pieces per thread.
__global__ void __launch_bounds__(256) w4_expand_kernel(const ExpandParams p)
{
    grid_launch_dependents();
    grid_dependency_wait();
    const size_t total  = p.chunks[0] + p.chunks[1];
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    const size_t tid    = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (size_t i0 = tid; i0 < total; i0 += 2 * stride) {
        Vec16  in[2];
        uint4* out[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const size_t i  = i0 + (size_t)u * stride;
            const bool   b  = i < p.chunks[0];
            const size_t at = b ? i : i - p.chunks[0];
            out[u]          = nullptr;
            if (i < total) {
                in[u]  = ld_nc_16((b ? p.src[0] : p.src[1]) + at);
                out[u] = (b ? p.dst[0] : p.dst[1]) + 2 * at;
            }
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            if (out[u] != nullptr) {
                const uint2 e0 = expand8(in[u].w[0]), e1 = expand8(in[u].w[1]), e2 = expand8(in[u].w[2]), e3 = expand8(in[u].w[3]);
                out[u][0] = make_uint4(e0.x, e0.y, e1.x, e1.y);
                out[u][1] = make_uint4(e2.x, e2.y, e3.x, e3.y);
            }
        }
    }
    if (p.act != nullptr) {
        for (size_t i = tid; i < p.act_pairs; i += stride) {
            const float a = ld_f32(p.act + 2 * i), b = ld_f32(p.act + 2 * i + 1);
            p.act16[i]    = p.act_bf16 ? Pair<__nv_bfloat16>::from_f32(a, b) : Pair<__half>::from_f32(a, b);
        }
    }
}

// ---------------------------------------------------------------------------------------------- GEMM
namespace wide {

constexpr int kBM          = 256;
constexpr int kBN          = 128;
constexpr int kKBlock      = 128;                       // K elements (= bytes) per block = 2 groups
constexpr int kThreads     = 384;
constexpr int kDrainWarps  = 8;
constexpr int kStages      = 3;
constexpr int kATile       = kBM * kKBlock;             // 32 KB
constexpr int kStage       = (kBM + kBN) * kKBlock;     // 48 KB
constexpr int kSSlots      = 2;
constexpr int kSlotGroups  = 4;                         // groups per scale slot = 2 K blocks
constexpr int kScaleSlot   = kSlotGroups * (kBM + kBN) * 4;   // sas[4][256] then sbs[4][128], fp32
constexpr int kBox         = 32 * 128;                  // a TMA store box: 32 rows x 128 bytes, 128-byte swizzle
constexpr int kBoxBytes    = 2 * kBox;                  // per drain warp: one per row half
constexpr int kScaleOffset = kStages * kStage;
constexpr int kRawBlock    = 128 * 16;                  // 128 rows x 4 group scales as TMA brings them, two buffers
constexpr int kRawOffset   = kScaleOffset + kSSlots * kScaleSlot;
constexpr int kOutOffset   = kRawOffset + 2 * kRawBlock;
constexpr int kBiasOffset  = kOutOffset + kDrainWarps * kBoxBytes;   // 128 bytes per drain warp: the bias of its columns
constexpr int kBarOffset   = kBiasOffset + kDrainWarps * 128;
constexpr int kSmemTotal   = kBarOffset + 256 + 1024;
static_assert(kSmemTotal <= 232448, "");
constexpr int kCols        = 64;                        // columns of a drain warp
constexpr int kHalfM       = kBM / 2;                   // rows of one MMA: an issuer covers a step with two
// Registers: 384 threads x 168 at launch = 64512; 256 x 216 + 128 x 72 is the same sum.
constexpr int kDrainRegs   = 216;
constexpr int kOtherRegs   = 72;

// gelu_tanh_f32 of both values, operation by operation, on packed pairs ([4608, 12288, 3072] with GELU: 427 -> 411 us).
__device__ __forceinline__ float2 gelu_tanh_pair(float2 v)
{
    const float2 cube = mul_f32x2(mul_f32x2(make_float2(0.044715f, 0.044715f), v), v);
    const float2 a    = mul_f32x2(make_float2(0.7978845608028654f, 0.7978845608028654f), fma_f32x2(cube, v, v));
    const float2 one  = add_f32x2(make_float2(1.0f, 1.0f), make_float2(tanh_approx(a.x), tanh_approx(a.y)));
    return mul_f32x2(v, mul_f32x2(make_float2(0.5f, 0.5f), one));
}

// The value of one output pair through the epilogue, up to the last rounding.
template<typename T>
__device__ __forceinline__ float2 finish_pair(const Params& p, float2 v, float2 bias, bool has_bias, float2 res, bool has_res)
{
    const bool each = p.round_each != 0 && sizeof(T) == 2;
    auto round_both = [&]() {
        if (each) {
            v.x = to_f32(from_f32<T>(v.x));
            v.y = to_f32(from_f32<T>(v.y));
        }
    };
    round_both();
    if (has_bias) {
        v.x += bias.x;
        v.y += bias.y;
        round_both();
    }
    if (p.gelu) {
        v = gelu_tanh_pair(v);
        round_both();
    }
    if (has_res) {
        v.x += res.x;
        v.y += res.y;
    }
    return v;
}

// Epilogue of the 64 columns of one row per thread, 16-bit output, n a multiple of 8.  `bias` is the shared-memory copy of the
// columns' bias; the residual of the row goes out as four loads before anything is computed.  The rows leave by TMA, a whole
// 128-byte line of each, from a box that nothing else uses until the next tile ends: all SMs end their tiles together, and whatever
// waits for the 64 KB that each of them then pushes at the L2 stands for 11000 to 15000 clocks (ordinary stores; two boxes in turn).
template<typename T>
__device__ __forceinline__ void store_rows16(const Params& p, const float2* acc, int row0, int col0, uint8_t* box, const uint16_t* bias, int lane,
                                             const CUtensorMap* tmap_d)
{
    const int row = row0 + lane;
#pragma unroll
    for (int b = 0; b < 2; ++b) {
        Vec16 res[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int col = col0 + 32 * b + 8 * q;
            res[q]        = Vec16{};
            if (p.residual != nullptr && col < p.N && row < p.M) {
                res[q] = ld_16(reinterpret_cast<const T*>(p.residual) + (size_t)row * p.N + col);
            }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const Vec16 bq = *reinterpret_cast<const Vec16*>(bias + 32 * b + 8 * q);
            Vec16       w;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float2 v = finish_pair<T>(p, acc[16 * b + 4 * q + j], Pair<T>::to_f32(bq.w[j]), p.bias != nullptr, Pair<T>::to_f32(res[q].w[j]),
                                                p.residual != nullptr);
                w.w[j]         = Pair<T>::from_f32(v.x, v.y);
            }
            *reinterpret_cast<Vec16*>(box + lane * 128 + (((4 * b + q) ^ (lane & 7)) << 4)) = w;
        }
    }
    fence_proxy_async_smem();
    __syncwarp();
    if (elect_one()) {
        tma_store_2d(tmap_d, smem_u32(box), col0, row0);   // clips rows and columns past the end
        tma_store_commit();
    }
}

// The same block for any output type and any n: element by element.
template<typename T>
__device__ __forceinline__ void store_block_any(const Params& p, const float2* acc, int row0, int col0, int lane)
{
    const int row = row0 + lane;
    if (row >= p.M) {
        return;
    }
    const T* b  = reinterpret_cast<const T*>(p.bias);
    const T* rs = reinterpret_cast<const T*>(p.residual);
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        const int    col = col0 + 2 * j;
        const size_t at  = (size_t)row * p.N + col;
        const bool   c0 = col < p.N, c1 = col + 1 < p.N;
        float2       bias = make_float2(0.0f, 0.0f), res = bias;
        if (b != nullptr) {
            bias = make_float2(c0 ? to_f32(b[col]) : 0.0f, c1 ? to_f32(b[col + 1]) : 0.0f);
        }
        if (rs != nullptr) {
            res = make_float2(c0 ? to_f32(rs[at]) : 0.0f, c1 ? to_f32(rs[at + 1]) : 0.0f);
        }
        const float2 v = finish_pair<T>(p, acc[j], bias, b != nullptr, res, rs != nullptr);
        T*           d = reinterpret_cast<T*>(p.D) + at;
        if (c0) {
            d[0] = from_f32<T>(v.x);
        }
        if (c1) {
            d[1] = from_f32<T>(v.y);
        }
    }
}

// Waits, bounded, for a copy that was asked for.
__device__ __forceinline__ void settle(uint32_t bar, uint32_t parity, unsigned int* status, unsigned code)
{
    const uint64_t t0 = global_timer_ns();
    while (!mbar_try_wait(bar, parity)) {
        if (global_timer_ns() - t0 > kWaitLimitNs) {
            report_timeout(status, code);
            break;
        }
    }
}

__global__ void __launch_bounds__(kThreads, 1)
gemm_w4a4_wide_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                      const __grid_constant__ CUtensorMap tmap_act, const __grid_constant__ CUtensorMap tmap_up,
                      const __grid_constant__ CUtensorMap tmap_d, const __grid_constant__ CUtensorMap tmap_sa,
                      const __grid_constant__ CUtensorMap tmap_sb, const Params p)
{
    constexpr uint32_t kTmemCols = 4 * kBN;
    constexpr uint32_t kIdesc    = umma_idesc(1u, 0u, kHalfM, kBN);

    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t*       gen_base  = smem_raw + (smem_base - smem_u32(smem_raw));
    const uint32_t bars      = smem_base + kBarOffset;
    auto full_bar   = [&](int s) { return bars + 8u * s; };
    auto empty_bar  = [&](int s) { return bars + 8u * (kStages + s); };
    auto part_full  = [&](uint32_t b) { return bars + 8u * (2 * kStages + b); };
    auto part_empty = [&](uint32_t b) { return bars + 8u * (2 * kStages + 2 + b); };
    auto sc_full    = [&](int s) { return bars + 8u * (2 * kStages + 4 + s); };
    auto sc_empty   = [&](int s) { return bars + 8u * (2 * kStages + 4 + kSSlots + s); };
    auto raw_full   = [&](int b) { return bars + 8u * (2 * kStages + 4 + 2 * kSSlots + b); };
    constexpr int kNumBars   = 2 * kStages + 6 + 2 * kSSlots;
    uint32_t*     tmem_slot  = reinterpret_cast<uint32_t*>(gen_base + kBarOffset + 8 * kNumBars);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = warp_index();
    const int lane = threadIdx.x & 31;

    grid_launch_dependents();
    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 2);           // both issuers
        }
        for (uint32_t b = 0; b < 2; ++b) {
            mbar_init(part_full(b), 1);
            mbar_init(part_empty(b), kDrainWarps);
        }
        for (int s = 0; s < kSSlots; ++s) {
            mbar_init(sc_full(s), 1);
            mbar_init(sc_empty(s), kDrainWarps);
        }
        mbar_init(raw_full(0), 1);
        mbar_init(raw_full(1), 1);
        *abort_flag = 0;
        fence_barrier_init();
        prefetch_tensormap(&tmap_a);
        prefetch_tensormap(&tmap_b);
    }
    if (warp == 2) {
        tmem_alloc(smem_u32(tmem_slot), kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    grid_dependency_wait();

    const int  num_tiles = p.m_tiles * p.n_tiles;
    const int  num_kb    = (p.K + kKBlock - 1) / kKBlock;
    const int  num_slots = (num_kb + 1) / 2;  // scale slots per tile
    const bool lora      = p.lora_act != nullptr;
    auto give_up = [&](unsigned code) {
        report_timeout(p.status, code);
        *abort_flag = 1;
    };

    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kOtherRegs));
        if (warp == 0) {
            // -------------------------------------------------------------- TMA producer
            int      stage = 0, issued = 0;
            uint32_t phase = 0;
            bool     ok = true;
            for (int tile = blockIdx.x; ok && tile < num_tiles; tile += gridDim.x) {
                const int m0 = (tile % p.m_tiles) * kBM;
                const int n0 = (tile / p.m_tiles) * kBN;
                for (int kb = 0; kb < num_kb + (lora ? 1 : 0); ++kb) {
                    if (!mbar_wait_warp(empty_bar(stage), phase ^ 1u, abort_flag)) {
                        give_up(0x5100u | (unsigned)stage);
                        ok = false;
                        break;
                    }
                    const uint32_t dst = smem_base + stage * kStage;
                    const bool     low = kb == num_kb;
                    if (elect_one()) {
                        mbar_arrive_expect_tx(full_bar(stage), (uint32_t)kStage);
                        tma_load_2d(dst, low ? &tmap_act : &tmap_a, full_bar(stage), low ? 0 : kb * kKBlock, m0);
                        tma_load_2d(dst + kATile, low ? &tmap_up : &tmap_b, full_bar(stage), low ? 0 : kb * kKBlock, n0);
                    }
                    ++issued;
                    if (++stage == kStages) {
                        stage = 0;
                        phase ^= 1u;
                    }
                }
            }
            // no copy may be in flight when the block leaves
            for (int i = 0; i < kStages && i < issued; ++i) {
                if (stage == 0) {
                    stage = kStages;
                    phase ^= 1u;
                }
                --stage;
                settle(full_bar(stage), phase, p.status, 0x5500u | (unsigned)stage);
            }
        } else if (warp != 2) {
            // -------------------------------------------------------------- MMA issuer of the steps n with n & 1 == q
            const uint32_t q     = (uint32_t)(warp >> 1);
            const uint32_t d     = tmem_base + q * kBN;
            int            stage = 0;
            uint32_t       phase = 0;
            uint32_t       n     = 0;  // steps (groups and low-rank products) of both issuers
            bool           ok    = true;
            const uint32_t idesc_low = umma_idesc(1u, p.c_dtype == LYRAQ_BF16 ? 1u : 0u, kHalfM, kBN);
            for (int tile = blockIdx.x; ok && tile < num_tiles; tile += gridDim.x) {
                for (int kb = 0; kb < num_kb + (lora ? 1 : 0); ++kb) {
                    const bool     low    = kb == num_kb;
                    const int      groups = low ? 1 : min(2, p.G - 2 * kb);
                    const int      g      = (int)((n ^ q) & 1u);   // this issuer's group of the block, if the block has it
                    // a K step of 32 bytes is 2 in 16-byte units
                    const uint64_t a0 = umma_desc_k_sw128(smem_base + stage * kStage) + (uint64_t)(g * 4);
                    const uint64_t a1 = a0 + (uint64_t)((kHalfM * kKBlock) >> 4);
                    const uint64_t b0 = a0 + (uint64_t)(kATile >> 4);
                    ok = mbar_wait_warp(full_bar(stage), phase, abort_flag);
                    if (ok && g < groups) {
                        // the half of tensor memory, once the drain has given it back
                        ok = mbar_wait_warp(part_empty(q), (((n + (uint32_t)g) >> 1) & 1u) ^ 1u, abort_flag);
                    }
                    if (!ok) {
                        give_up(0x5200u | (unsigned)stage);
                        break;
                    }
                    tc_fence_after_sync();
                    if (elect_one()) {
                        if (g < groups) {
                            if (low) {
                                mma_f16(d, a0, b0, idesc_low, 0u);
                                mma_f16(d, a0 + 2, b0 + 2, idesc_low, 1u);
                                mma_f16(d + 2 * kBN, a1, b0, idesc_low, 0u);
                                mma_f16(d + 2 * kBN, a1 + 2, b0 + 2, idesc_low, 1u);
                            } else {
                                mma_f8f6f4(d, a0, b0, kIdesc, 0u);
                                mma_f8f6f4(d, a0 + 2, b0 + 2, kIdesc, 1u);
                                mma_f8f6f4(d + 2 * kBN, a1, b0, kIdesc, 0u);
                                mma_f8f6f4(d + 2 * kBN, a1 + 2, b0 + 2, kIdesc, 1u);
                            }
                            tc_commit(part_full(q));
                        }
                        tc_commit(empty_bar(stage));   // each issuer once per block, after its own MMAs on it (if any)
                    }
                    n += (uint32_t)groups;
                    if (++stage == kStages) {
                        stage = 0;
                        phase ^= 1u;
                    }
                }
            }
        } else if (p.scale_tma) {
            // -------------------------------------------------------------- scale loader (warp 2), scales that TMA can address
            // A slot is three blocks of 128 rows x 4 groups (rows 0-127 and 128-255 of A, the columns of B), which TMA fetches two blocks
            // ahead as they lie in memory, 16 bytes a row; a lane turns its four rows' pieces into [g][row].
            const int tiles_here = (num_tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
            const int blocks     = tiles_here * num_slots * 3;
            int       i_tile = blockIdx.x, i_slot = 0, i_part = 0;   // the block to ask for next
            auto ask = [&](int j) {
                if (j < blocks && elect_one()) {
                    const int      m0  = (i_tile % p.m_tiles) * kBM, n0 = (i_tile / p.m_tiles) * kBN;
                    const uint32_t dst = smem_base + kRawOffset + (j & 1) * kRawBlock;
                    mbar_arrive_expect_tx(raw_full(j & 1), (uint32_t)kRawBlock);
                    if (i_part < 2) {
                        tma_load_2d(dst, &tmap_sa, raw_full(j & 1), i_slot * kSlotGroups * 4, m0 + i_part * 128);
                    } else {
                        // 16-bit scales: the 16 bytes hold this slot's four groups and a neighbour's
                        tma_load_2d(dst, &tmap_sb, raw_full(j & 1), p.sb_is_f16 ? (i_slot & ~1) * kSlotGroups * 2 : i_slot * kSlotGroups * 4, n0);
                    }
                }
                if (++i_part == 3) {
                    i_part = 0;
                    if (++i_slot == num_slots) {
                        i_slot = 0;
                        i_tile += (int)gridDim.x;
                    }
                }
            };
            ask(0);
            ask(1);
            int      slot = 0, part = 0, s_tile = 0, asked = min(blocks, 2);
            uint32_t sphase = 0;
            for (int j = 0; j < blocks; ++j) {
                if ((part == 0 && !mbar_wait_warp(sc_empty(slot), sphase ^ 1u, abort_flag)) ||
                    !mbar_wait_warp(raw_full(j & 1), (uint32_t)((j >> 1) & 1), abort_flag)) {
                    give_up(0x5800u | (unsigned)slot);
                    break;
                }
                const uint8_t* raw  = gen_base + kRawOffset + (j & 1) * kRawBlock;
                float*         dst  = reinterpret_cast<float*>(gen_base + kScaleOffset + slot * kScaleSlot) + (part < 2 ? part * 128 : kSlotGroups * kBM) + lane;
                const int      step = part < 2 ? kBM : kBN;
                const bool     half = part == 2 && p.sb_is_f16;
                Vec16          v[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    v[i] = *reinterpret_cast<const Vec16*>(raw + (i * 32 + lane) * 16);
                }
                __syncwarp();
                asked += j + 2 < blocks ? 1 : 0;
                ask(j + 2);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    float x[4];
                    if (half) {
                        const float2 lo = Pair<__half>::to_f32((s_tile & 1) ? v[i].w[2] : v[i].w[0]);
                        const float2 hi = Pair<__half>::to_f32((s_tile & 1) ? v[i].w[3] : v[i].w[1]);
                        x[0] = lo.x; x[1] = lo.y; x[2] = hi.x; x[3] = hi.y;
                    } else {
#pragma unroll
                        for (int g = 0; g < 4; ++g) {
                            x[g] = __uint_as_float(v[i].w[g]);
                        }
                    }
#pragma unroll
                    for (int g = 0; g < 4; ++g) {
                        dst[g * step + i * 32] = x[g];
                    }
                }
                if (++part == 3) {
                    part = 0;
                    __syncwarp();
                    if (lane == 0) {
                        mbar_arrive(sc_full(slot));
                    }
                    if (++slot == kSSlots) {
                        slot = 0;
                        sphase ^= 1u;
                    }
                    s_tile = s_tile + 1 == num_slots ? 0 : s_tile + 1;   // slot number inside its tile
                }
            }
            // no copy may be in flight when the block leaves: block j is the (j >> 1)-th of its buffer
            for (int j = max(0, asked - 2); j < asked; ++j) {
                settle(raw_full(j & 1), (uint32_t)((j >> 1) & 1), p.status, 0x5900u | (unsigned)(j & 1));
            }
        } else {
            // -------------------------------------------------------------- scale loader (warp 2), any scales
            constexpr int kRowSets = (kBM + kBN) / 32;   // sets of 32 rows
            constexpr int kBatch   = 6;                  // sets whose loads are in flight together
            int      slot = 0;
            uint32_t sphase = 0;
            bool     ok = true;
            for (int tile = blockIdx.x; ok && tile < num_tiles; tile += gridDim.x) {
                const int m0 = (tile % p.m_tiles) * kBM;
                const int n0 = (tile / p.m_tiles) * kBN;
                for (int sl = 0; sl < num_slots; ++sl) {
                    if (!mbar_wait_warp(sc_empty(slot), sphase ^ 1u, abort_flag)) {
                        give_up(0x5800u | (unsigned)slot);
                        ok = false;
                        break;
                    }
                    float*     sas  = reinterpret_cast<float*>(gen_base + kScaleOffset + slot * kScaleSlot);
                    float*     sbs  = sas + kSlotGroups * kBM;
                    const int  g0   = sl * kSlotGroups;
                    const bool full = p.scale_vec_ok && (g0 + kSlotGroups <= p.G);
#pragma unroll 1
                    for (int s0 = 0; s0 < kRowSets; s0 += kBatch) {
                        float v[kBatch][kSlotGroups];   // 16-bit scales: their bits at first
#pragma unroll
                        for (int i = 0; i < kBatch; ++i) {
                            const int    r    = (s0 + i) * 32 + lane;   // 0 .. 255: A rows, then B rows
                            const bool   is_a = r < kBM;
                            const int    grow = is_a ? m0 + r : n0 + r - kBM;
                            const bool   in   = grow < (is_a ? p.M : p.N);
                            const size_t at   = (size_t)grow * p.G + g0;
                            if (!is_a && p.sb_is_f16) {
                                const __half* q = reinterpret_cast<const __half*>(p.sb) + at;
                                if (full && in) {
                                    const uint2 w = *reinterpret_cast<const uint2*>(q);
                                    v[i][0] = __uint_as_float(w.x & 0xffffu); v[i][1] = __uint_as_float(w.x >> 16);
                                    v[i][2] = __uint_as_float(w.y & 0xffffu); v[i][3] = __uint_as_float(w.y >> 16);
                                } else {
#pragma unroll
                                    for (int g = 0; g < kSlotGroups; ++g) {
                                        v[i][g] = (in && g0 + g < p.G) ? __uint_as_float(ld_u16(q + g)) : 0.0f;
                                    }
                                }
                            } else {
                                const float* q = (is_a ? p.sa : reinterpret_cast<const float*>(p.sb)) + at;
                                if (full && in) {
                                    const float4 x = ld_f32x4(reinterpret_cast<const float4*>(q));
                                    v[i][0] = x.x; v[i][1] = x.y; v[i][2] = x.z; v[i][3] = x.w;
                                } else {
#pragma unroll
                                    for (int g = 0; g < kSlotGroups; ++g) {
                                        v[i][g] = (in && g0 + g < p.G) ? ld_f32(q + g) : 0.0f;
                                    }
                                }
                            }
                        }
                        if (p.sb_is_f16) {
                            // 16-bit scales are converted only now: beside its load each conversion waited for it before the next load went
                            // out ([4608, 3072, 3136]: 208 us, 133 so)
#pragma unroll
                            for (int i = 0; i < kBatch; ++i) {
                                if (s0 + i >= kBM / 32) {
#pragma unroll
                                    for (int g = 0; g < kSlotGroups; ++g) {
                                        v[i][g] = __half2float(__ushort_as_half((unsigned short)__float_as_uint(v[i][g])));
                                    }
                                }
                            }
                        }
#pragma unroll
                        for (int i = 0; i < kBatch; ++i) {
                            const int r      = (s0 + i) * 32 + lane;
                            float*    dst    = r < kBM ? sas + r : sbs + r - kBM;
                            const int stride = r < kBM ? kBM : kBN;
#pragma unroll
                            for (int g = 0; g < kSlotGroups; ++g) {
                                dst[g * stride] = v[i][g];
                            }
                        }
                    }
                    __syncwarp();
                    if (lane == 0) {
                        mbar_arrive(sc_full(slot));
                    }
                    if (++slot == kSSlots) {
                        slot = 0;
                        sphase ^= 1u;
                    }
                }
            }
        }
    } else {
        // ------------------------------------------------------------------ drain + epilogue (warps 4 .. 11)
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kDrainRegs));
        const int      quad      = warp & 3;
        const int      part      = (warp - 4) >> 2;     // 64-column half of the tile
        const uint32_t lane_addr = ((uint32_t)(quad * 32) << 16) + (uint32_t)(part * kCols);
        uint8_t*       box       = gen_base + kOutOffset + (warp - 4) * kBoxBytes;
        int            slot = 0;
        uint32_t       sphase = 0;
        uint32_t       n = 0;          // steps (groups and low-rank products) drained
        bool           ok = true;
        auto wait_step = [&](bool ready) {   // ready: the barrier was seen complete ahead of time
            if (!__all_sync(0xffffffffu, ready) && !mbar_wait_warp(part_full(n & 1u), (n >> 1) & 1u, abort_flag)) {
                give_up(0x5700u);
                ok = false;
            }
            tc_fence_after_sync();
            return tmem_base + lane_addr + (n & 1u) * kBN;
        };
        auto release_step = [&]() {
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(part_empty(n & 1u));
            }
            ++n;
        };
        for (int tile = blockIdx.x; ok && tile < num_tiles; tile += gridDim.x) {
            const int m_blk = tile % p.m_tiles;
            const int n_blk = tile / p.m_tiles;
            // the bias of the warp's columns, 16-bit outputs: fetched now, used at the end of the tile
            uint32_t bias2 = 0;
            if (p.bias != nullptr && p.c_dtype != LYRAQ_F32) {
                const int       col = n_blk * kBN + part * kCols + 2 * lane;
                const uint16_t* b   = static_cast<const uint16_t*>(p.bias);
                bias2 = (col < p.N ? b[col] : 0u) | (col + 1 < p.N ? (uint32_t)b[col + 1] << 16 : 0u);
            }
            float2    acc[2][kCols / 2];   // this thread's two half rows, as packed pairs
#pragma unroll
            for (int i = 0; i < kCols / 2; ++i) {
                acc[0][i] = make_float2(0.0f, 0.0f);
                acc[1][i] = make_float2(0.0f, 0.0f);
            }
            // What a group needs first is fetched while the last piece of the group before is rescaled, and its barriers are looked at
            // in that group, so that a group begins without a pause: the drain warps of a scheduler run in step, and whatever one waits
            // for, both wait for.
            uint32_t pcs[2][16];
            float4   sb[2][4];
            float2   sa[2];
            auto slot_scales = [&](int sl, int in_slot) {
                return reinterpret_cast<const float*>(gen_base + kScaleOffset + sl * kScaleSlot) + in_slot * kBM + quad * 32 + lane;
            };
            auto slot_columns = [&](int sl, int in_slot) {
                return reinterpret_cast<const float4*>(gen_base + kScaleOffset + sl * kScaleSlot + (kSlotGroups * kBM + in_slot * kBN + part * kCols) * 4);
            };
            auto wait_scales = [&](int sl, uint32_t ph) {
                if (!mbar_wait_warp(sc_full(sl), ph, abort_flag)) {
                    give_up(0x5600u | (unsigned)sl);
                    ok = false;
                }
            };
            wait_scales(slot, sphase);
            uint32_t t_addr = ok ? wait_step(false) : 0u;
            if (!ok) {
                break;
            }
            tmem_ld_32x16(t_addr, pcs[0]);
            const float*  sas = slot_scales(slot, 0);
            const float4* sb4 = slot_columns(slot, 0);
            sa[0] = make_float2(sas[0], sas[0]);
            sa[1] = make_float2(sas[kHalfM], sas[kHalfM]);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                sb[0][j] = sb4[j];
            }
            int in_slot = 0;
#pragma unroll 1
            for (int g = 0; g < p.G; ++g) {
                const bool    more  = g + 1 < p.G;
                const bool    leave = in_slot == kSlotGroups - 1 || !more;   // the slot's last group
                const int     slot2 = !leave ? slot : (slot + 1 == kSSlots ? 0 : slot + 1);
                float2        sa2[2];
                bool          ready     = false;
                const float4* nb4       = sb4;
                uint32_t      next_addr = t_addr;
                // piece i: 16 columns 16 (i / 2) .. of row half i & 1; the load of piece i + 1 (of the next group's first one, at
                // the end) is in flight while piece i is rescaled, and the column scales of the next 16 columns are fetched a piece
                // ahead as well
#pragma unroll
                for (int i = 0; i < kCols / 8; ++i) {
                    const int h = i & 1, c = i >> 1;
                    tmem_ld_wait();
                    if (i + 1 < kCols / 8) {
                        tmem_ld_32x16(t_addr + (uint32_t)(((i + 1) & 1) * 2 * kBN + ((i + 1) >> 1) * 16), pcs[(i + 1) & 1]);
                    } else {
                        release_step();   // all of the group is in registers
                        if (more) {
                            next_addr = wait_step(ready);
                            if (ok) {
                                tmem_ld_32x16(next_addr, pcs[0]);
                            }
                        }
                    }
                    if (i == kCols / 8 - 2) {
                        ready = mbar_test_wait(part_full((n + 1) & 1u), ((n + 1) >> 1) & 1u);   // test_wait: try_wait would stop here
                    }
                    if (i == kCols / 16 && leave && more) {
                        wait_scales(slot2, slot2 == 0 ? sphase ^ 1u : sphase);
                    }
                    if (h == 1) {
                        if (c + 1 < kCols / 16) {
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                sb[(c + 1) & 1][j] = sb4[(c + 1) * 4 + j];
                            }
                        } else {
                            const int    in2 = leave ? 0 : in_slot + 1;
                            const float* na  = slot_scales(slot2, in2);
                            nb4              = slot_columns(slot2, in2);
                            sa2[0]           = make_float2(na[0], na[0]);
                            sa2[1]           = make_float2(na[kHalfM], na[kHalfM]);
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                sb[0][j] = nb4[j];
                            }
                        }
                    }
                    const uint32_t* pc = pcs[i & 1];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        // acc = fma(p * sa, sb, acc): the contraction the reference's compiler makes of
                        // `acc += float(p) * sa * sb` (w4a4_gemm.cu:504-507); two columns per instruction
                        const float4 s4 = sb[c & 1][j];
                        const float2 p0 = make_float2(__uint_as_float(pc[4 * j]), __uint_as_float(pc[4 * j + 1]));
                        const float2 p1 = make_float2(__uint_as_float(pc[4 * j + 2]), __uint_as_float(pc[4 * j + 3]));
                        float2*      a  = &acc[h][c * 8 + 2 * j];
                        a[0] = fma_f32x2(mul_f32x2(p0, sa[h]), make_float2(s4.x, s4.y), a[0]);
                        a[1] = fma_f32x2(mul_f32x2(p1, sa[h]), make_float2(s4.z, s4.w), a[1]);
                    }
                }
                if (!ok) {
                    break;
                }
                if (leave) {
                    __syncwarp();
                    if (lane == 0) {
                        mbar_arrive(sc_empty(slot));
                    }
                    slot = slot2;
                    sphase ^= slot2 == 0 ? 1u : 0u;
                }
                in_slot = leave ? 0 : in_slot + 1;
                sb4     = nb4;
                t_addr  = next_addr;
                sa[0]   = sa2[0];
                sa[1]   = sa2[1];
            }
            if (ok && lora) {
                const uint32_t t_addr = wait_step(false);
                if (ok) {
#pragma unroll
                    for (int i = 0; i < kCols / 8; ++i) {
                        uint32_t pc[16];
                        tmem_ld_32x16(t_addr + (uint32_t)((i & 1) * 2 * kBN + (i >> 1) * 16), pc);
                        tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            float2& a = acc[i & 1][(i >> 1) * 8 + j];
                            a         = add_f32x2(a, make_float2(__uint_as_float(pc[2 * j]), __uint_as_float(pc[2 * j + 1])));
                        }
                    }
                    release_step();
                }
            }
            if (!ok) {
                break;
            }
            uint16_t* bias_s = reinterpret_cast<uint16_t*>(gen_base + kBiasOffset + (warp - 4) * 128);
            reinterpret_cast<uint32_t*>(bias_s)[lane] = bias2;
            if (elect_one()) {
                tma_store_wait_read();   // the last tile's stores have drained the boxes
            }
            __syncwarp();
            const int col0 = n_blk * kBN + part * kCols;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int row0 = m_blk * kBM + h * kHalfM + quad * 32;
                if (row0 < p.M && col0 < p.N) {
                    if (p.c_dtype == LYRAQ_F32) {
                        store_block_any<float>(p, acc[h], row0, col0, lane);
                        store_block_any<float>(p, acc[h] + 16, row0, col0 + 32, lane);
                    } else if (p.c_dtype == LYRAQ_BF16) {
                        if ((p.N & 7) == 0) {
                            store_rows16<__nv_bfloat16>(p, acc[h], row0, col0, box + h * kBox, bias_s, lane, &tmap_d);
                        } else {
                            store_block_any<__nv_bfloat16>(p, acc[h], row0, col0, lane);
                            store_block_any<__nv_bfloat16>(p, acc[h] + 16, row0, col0 + 32, lane);
                        }
                    } else {
                        if ((p.N & 7) == 0) {
                            store_rows16<__half>(p, acc[h], row0, col0, box + h * kBox, bias_s, lane, &tmap_d);
                        } else {
                            store_block_any<__half>(p, acc[h], row0, col0, lane);
                            store_block_any<__half>(p, acc[h] + 16, row0, col0 + 32, lane);
                        }
                    }
                }
            }
        }
        if (elect_one()) {
            tma_store_wait_read();  // shared memory must outlive the last stores' reads of it
        }
    }

    tc_fence_before_sync();
    __syncthreads();
    if (warp == 2) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, kTmemCols);
    }
}

}  // namespace wide

static size_t up256(size_t v) { return (v + 255) / 256 * 256; }

size_t wide_workspace_bytes(size_t m, size_t n, size_t k) { return up256(n * k) + up256(m * k) + up256(m * 64); }

int launch_wide(Params p, const uint8_t* A, const uint8_t* B, void* workspace, int sms, cudaStream_t stream)
{
    const size_t m = (size_t)p.M, n = (size_t)p.N, k = (size_t)p.K;
    uint8_t*     be  = static_cast<uint8_t*>(workspace);
    uint8_t*     ae  = be + up256(n * k);
    uint8_t*     a16 = ae + up256(m * k);
    ExpandParams e{};
    e.src[0]    = reinterpret_cast<const uint4*>(B);
    e.dst[0]    = reinterpret_cast<uint4*>(be);
    e.chunks[0] = n * k / 32;
    e.src[1]    = reinterpret_cast<const uint4*>(A);
    e.dst[1]    = reinterpret_cast<uint4*>(ae);
    e.chunks[1] = m * k / 32;
    if (p.lora_act != nullptr && p.lora_act_is_f32) {
        e.act       = static_cast<const float*>(p.lora_act);
        e.act16     = reinterpret_cast<uint32_t*>(a16);
        e.act_pairs = m * (kLoraRank / 2);
        e.act_bf16  = p.c_dtype == LYRAQ_BF16 ? 1 : 0;
        p.lora_act  = a16;
        p.lora_act_is_f32 = 0;
    }
    const size_t blocks = (e.chunks[0] + e.chunks[1] + 511) / 512;
    const size_t cap    = (size_t)sms * 32;
    int          st = cuda_status(launch_kernel(w4_expand_kernel, (unsigned)(blocks < cap ? blocks : cap), 256u, (size_t)0, stream, 1u, e),
                                  "cudaLaunchKernelEx(w4_expand_kernel)");
    if (st != LYRAQ_OK) {
        return st;
    }
    p.m_tiles = (p.M + wide::kBM - 1) / wide::kBM;
    p.n_tiles = (p.N + wide::kBN - 1) / wide::kBN;
    CUtensorMap ta, tb, tact, tup;
    st = make_tmap_bytes_2d(&ta, ae, m, k, k, wide::kBM, wide::kKBlock, true);
    if (st != LYRAQ_OK) {
        return st;
    }
    st = make_tmap_bytes_2d(&tb, be, n, k, k, wide::kBN, wide::kKBlock, true);
    if (st != LYRAQ_OK) {
        return st;
    }
    tact = ta;   // never read without a low-rank branch
    tup  = tb;
    if (p.lora_act != nullptr) {
        // rows of 32 sixteen-bit values: TMA fills the second half of each 128-byte line with zeros
        st = make_tmap_bytes_2d(&tact, p.lora_act, m, 64, 64, wide::kBM, wide::kKBlock, true);
        if (st != LYRAQ_OK) {
            return st;
        }
        st = make_tmap_bytes_2d(&tup, p.lora_up, n, 64, 64, wide::kBN, wide::kKBlock, true);
        if (st != LYRAQ_OK) {
            return st;
        }
    }
    CUtensorMap td = ta;   // never used where the output leaves by ordinary stores
    if (p.c_dtype != LYRAQ_F32 && (p.N & 7) == 0) {
        st = make_tmap_store(&td, p.D, m, n, n, 2, true);
        if (st != LYRAQ_OK) {
            return st;
        }
    }
    CUtensorMap tsa = ta, tsb = ta;   // never read where the lanes load the scales
    // TMA wants 16-byte rows: pitches that are multiples of 16 bytes, from aligned arrays
    p.scale_tma = (p.G & (p.sb_is_f16 ? 7 : 3)) == 0 && aligned16(p.sa) && aligned16(p.sb) ? 1 : 0;
    if (p.scale_tma) {
        const uint64_t sa_row = (uint64_t)p.G * 4, sb_row = (uint64_t)p.G * (p.sb_is_f16 ? 2 : 4);
        st = make_tmap_bytes_2d(&tsa, p.sa, m, sa_row, sa_row, 128, 16, false);
        if (st != LYRAQ_OK) {
            return st;
        }
        st = make_tmap_bytes_2d(&tsb, p.sb, n, sb_row, sb_row, 128, 16, false);
        if (st != LYRAQ_OK) {
            return st;
        }
    }
    const long  tiles = (long)p.m_tiles * p.n_tiles;
    const int   grid  = (int)(tiles < sms ? tiles : sms);
    static bool smem_raised[64] = {};
    st = raise_dynamic_smem_once(wide::gemm_w4a4_wide_kernel, (int)wide::kSmemTotal, smem_raised,
                                 "cudaFuncSetAttribute(gemm_w4a4_wide_kernel, dynamic shared memory)");
    if (st != LYRAQ_OK) {
        return st;
    }
    return cuda_status(launch_kernel(wide::gemm_w4a4_wide_kernel, (unsigned)grid, (unsigned)wide::kThreads, (size_t)wide::kSmemTotal,
                                     stream, 1u, ta, tb, tact, tup, td, tsa, tsb, p),
                       "cudaLaunchKernelEx(gemm_w4a4_wide_kernel)");
}

}  // namespace w4
}  // namespace lyraq
