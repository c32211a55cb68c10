// Attention forward for the FLUX blocks: out[b, s, h, :] = softmax(q k^T * scale) v over the packed projection
// qkv [batch, seq, 3, heads, 128] (16-bit), no mask, no dropout.  Replaces the reference's FlashAttention-2 layer
// (src/lyradiff/layers/flash_attn2/flash_attn2.cu:59-118, kernels flash_fwd_kernel.h) on the path between the QKV
// linear and the output linear, and writes its result either in the 16-bit type or already quantized to e4m3 for the
// FP8 linear that follows (the reference runs cudaD2DScaleCpyConvert over the attention output as a separate pass,
// FluxSingleTransformerFP8Block.cc:254, FluxAttnPostFP8Processor.cc:135,168).
//
// A persistent CTA takes blocks of 256 query rows of one head (two tiles of 128) in turn and walks their keys in steps of 128:
//   warp 12     TMA producer: per block Q (2 x 32 KB), then K_0, V_0, K_1, V_1, ... through a ring of five 32 KB slots.  Every tile is
//               two SWIZZLE_128B boxes of 128 rows x 64 columns, so q and k tiles are K-major operands and the v tile is an MN-major
//               operand as it lies in memory.
//   warp 13     MMA issuer of both query tiles; owns tensor memory (512 columns: S_0 | S_1 | O_0 | O_1, 128 fp32 columns each).
//               Per step and tile: O += P V (8 x tcgen05.mma kind::f16, M 128, N 128, K 16; P is read from tensor memory, where the
//               softmax warps wrote it over the first half of S), then the next step's S = Q K^T over it (8 more), while the other
//               tile is in its softmax.  The scores of the next block's first step follow the last step of a block in the same way.
//   warps 0-3   softmax of query tile 0, warps 4-7 of tile 1: a thread owns one query row (its tensor-memory lane), so row maxima
//               and sums need no shuffles.  exp2 with the scale folded in; the running maximum is only raised when it grew by more
//               than 2^8 (the accumulator and the row sum then share the stale reference, which cancels in O / l), so O is rescaled
//               in tensor memory rarely, by these same warps, between two of their tile's P V products.  P goes to the issuer in
//               two halves of 64 keys.
//   warps 8-11  epilogue: O / l of a finished block is read, converted and stored while the next block is under way.
// Every wait is bounded; on a timeout the role records it in the status word, raises the block's abort flag and all roles leave; tensor
// memory is freed at the common exit.
//
// What bounds it (4608 x 24 x 128, per 128-key step of both tiles): 2048 clocks of tensor pipe, 2048 of the exponent unit (16 ex2 per
// clock and SM; an eighth of them goes to the FMA pipe, which leaves 1792), against about 2950 measured.  The softmax of a tile and
// the MMAs it waits for form a chain of about 2900 (softmax 1800 with the other tile's warps on the same unit for half of it, hand-over 100,
// half of P V and Q K^T 770, completion to the first score 280).  At that rate the chip runs into its power limit: 1.65 GHz in a short
// burst, 1.45 under sustained load (1.83 with all-zero inputs).
// Measured, bf16 in, e4m3 out: 250 us -> 221 (issuer entered through elect.sync) -> 197, back to back for a second 326 -> 221; 1667
// tokens 71 -> 54.  What made the difference over 64-key steps with double-buffered scores: N = 128 score products (N = 64 ones are
// bound by shared memory), the next block's start and the last one's epilogue out of the way of the softmax, and above all an issuer
// whose code between two MMAs is short: whole-warp waits of a few instructions (see mbar_wait_warp) and no slow path in between.
// Not kept: exponentials started from the old maximum with the new one found beside them (the same time), two softmax warps per
// 32 rows (3 % fewer clocks, the same time at the power limit), P handed over in parts of 96 + 32 keys (3 to 4 % slower), a quarter of the exponentials on the FMA
// pipe (2 % slower than an eighth).
#include "common.cuh"
#include "sm100_ptx.cuh"

namespace lyraq {

using namespace sm100;

typedef CUresult (*EncodeTiledFnAttn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                      const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                      CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

int device_sm_count();  // gemm_dense.cu

namespace attn {

constexpr int kHeadDim   = 128;
constexpr int kTile      = 128;                       // rows of a query tile, keys of a step
constexpr int kQTiles    = 2;
constexpr int kTileBytes = kTile * kHeadDim * 2;      // 32 KB: two boxes of 128 rows x 128 bytes
constexpr int kBoxBytes  = kTileBytes / 2;
constexpr int kSlots     = 5;
constexpr int kQOffset   = 0;
constexpr int kRingOffset = kQTiles * kTileBytes;
constexpr int kSumOffset = kRingOffset + kSlots * kTileBytes;   // row sums on their way to the epilogue warps: [tile][128] fp32
constexpr int kBarOffset = kSumOffset + kQTiles * kTile * 4;
constexpr int kNumBars   = 2 * kSlots + 9 * kQTiles;
constexpr int kSmemUsed  = kBarOffset + 8 * kNumBars + 16;
constexpr int kSmemTotal = 232448;                    // all a block may have; the tiles need 1024-byte alignment, which leaves
static_assert(kSmemTotal - kSmemUsed >= 768, "");     // room for a base that is only 256-byte aligned
constexpr int kThreads   = 512;
constexpr int kEpiWarp   = 8;                         // warps 0-7 softmax, 8-11 epilogue
constexpr int kProducerWarp = 12;
constexpr int kMmaWarp   = 13;
// registers: 512 threads x 128 at launch = 65536; 256 x 184 + 128 x 104 + 128 x 40 is the same sum
constexpr int kSoftmaxRegs = 184;
constexpr int kEpiRegs   = 104;
constexpr int kOtherRegs = 40;
constexpr int kTmemCols  = 512;                       // S_0 | S_1 | O_0 | O_1, 128 columns each; P_t lies over the first half of S_t
constexpr float kRescaleThreshold = 8.0f;             // in log2 units
constexpr int kPolyPairs = 2;                         // of 16 pairs of scores, how many take their exponentials from the FMA pipe

struct Params {
    void*         out[2];        // rows [0, split) of every batch go to out[0], the rest to out[1] (row index - split)
    long long     out_ld[2];     // row pitch in elements of the output type
    long long     out_batch[2];  // batch pitch in elements
    const float*  out_scale[2];  // e4m3 output: per-tensor scale of each part (1 / scale applied); unused otherwise
    int           out_e4m3;
    int           split;
    int           seq, heads;
    int           q_blocks;      // ceil(seq / 256)
    int           blocks;        // batch * heads * q_blocks
    float         scale_log2;    // softmax scale * log2(e)
    unsigned int* status;
    unsigned long long wait_limit_ns;  // longest a single wait may last (2 s; a test hook shortens it)
    int           skip_loads;          // test hook: the producer issues no copy, so every consumer's wait runs out
};

__device__ __forceinline__ float ex2_approx(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// 2^x of two values on the FMA and ALU pipes: x = n + f with n an integer and f in [-1/2, 1/2]; 2^f from its minimax polynomial of
// degree 5 (Remez exchange on the relative error: 7.5e-8 in exact arithmetic, 2.1e-7 evaluated in fp32, which is what ex2.approx
// has), and n added to the exponent.  x of -127 and below gives the smallest subnormal, which both 16-bit types round to a weight of zero,
// as ex2.approx.ftz does: such a key adds nothing to O, whatever its value row holds.  (Between -126 and -127 the result is some subnormal.)
// NaN and infinity do not come through: the caller looks for them in the row's maximum.
__device__ __forceinline__ float2 ex2_poly(float2 x)
{
    const float  magic = 12582912.0f;   // 1.5 * 2^23: the sum's low mantissa bits are n
    x                  = make_float2(fmaxf(x.x, -127.0f), fmaxf(x.y, -127.0f));
    const float2 t     = add_f32x2(x, make_float2(magic, magic));
    const float2 n     = add_f32x2(t, make_float2(-magic, -magic));
    const float2 f     = fma_f32x2(n, make_float2(-1.0f, -1.0f), x);
    auto two = [](float v) { return make_float2(v, v); };
    float2 q = fma_f32x2(two(0.0013276472454890609f), f, two(0.009675540961325169f));
    q        = fma_f32x2(q, f, two(0.05550713092088699f));
    q        = fma_f32x2(q, f, two(0.24022120237350464f));
    q        = fma_f32x2(q, f, two(0.6931469440460205f));
    q        = fma_f32x2(q, f, two(1.0000001192092896f));
    return make_float2(__uint_as_float((__float_as_uint(t.x) << 23) + __float_as_uint(q.x)), __uint_as_float((__float_as_uint(t.y) << 23) + __float_as_uint(q.y)));
}

__device__ __forceinline__ float max3(float a, float b, float c)
{
    float d;
    asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

__device__ __forceinline__ void tma_load_3d(uint32_t smem_dst, const CUtensorMap* m, uint32_t bar, int x, int y, int z)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(smem_dst), "l"(m), "r"(bar), "r"(x), "r"(y), "r"(z)
        : "memory");
}

// FOLD: the softmax scale is positive.  Other scales have an instance of their own: as a branch in the one kernel, 128 multiplications that
// ordinary calls jump over, they cost 64 tokens 0.2 us of 6.6.
template<typename T, bool FOLD>
__global__ void __launch_bounds__(kThreads, 1)
attention_fwd_kernel(const __grid_constant__ CUtensorMap tmap_qkv, const __grid_constant__ Params p)
{
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t*       gen_base  = smem_raw + (smem_base - smem_u32(smem_raw));
    if (smem_base - smem_u32(smem_raw) + (uint32_t)kSmemUsed > (uint32_t)kSmemTotal) {
        if (threadIdx.x == 0) {
            report_timeout(p.status, 0x3001u);  // the aligned layout does not fit: nothing is touched
        }
        return;
    }
    const uint32_t bars = smem_base + kBarOffset;
    auto slot_full  = [&](int s) { return bars + 8u * s; };                              // k / v tile s has landed
    auto slot_empty = [&](int s) { return bars + 8u * (kSlots + s); };                   // ... and has been read
    auto tile_bar   = [&](int kind, int t) { return bars + 8u * (2 * kSlots + 2 * kind + t); };
    auto q_full     = [&](int t) { return tile_bar(0, t); };
    auto q_empty    = [&](int t) { return tile_bar(1, t); };
    auto s_full     = [&](int t) { return tile_bar(2, t); };   // scores of a step
    auto p_first    = [&](int t) { return tile_bar(3, t); };   // P of the step's keys 0 .. 63 is in tensor memory
    auto p_second   = [&](int t) { return tile_bar(4, t); };   // ... and of keys 64 .. 127
    auto o_full     = [&](int t) { return tile_bar(5, t); };   // accumulator of a block is final
    auto o_empty    = [&](int t) { return tile_bar(6, t); };   // ... and has been read
    auto l_full     = [&](int t) { return tile_bar(7, t); };   // row sums of a block are in shared memory
    auto l_empty    = [&](int t) { return tile_bar(8, t); };
    uint32_t*     tmem_slot  = reinterpret_cast<uint32_t*>(gen_base + kBarOffset + 8 * kNumBars);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = warp_index();
    const int lane = threadIdx.x & 31;

    grid_launch_dependents();
    if (threadIdx.x == 0) {
        for (int s = 0; s < kSlots; ++s) {
            mbar_init(slot_full(s), 1);
            mbar_init(slot_empty(s), 1);
        }
        for (int t = 0; t < kQTiles; ++t) {
            mbar_init(q_full(t), 1);
            mbar_init(q_empty(t), 1);
            mbar_init(s_full(t), 1);
            mbar_init(p_first(t), 4);
            mbar_init(p_second(t), 4);
            mbar_init(o_full(t), 1);
            mbar_init(o_empty(t), 4);
            mbar_init(l_full(t), 4);
            mbar_init(l_empty(t), 4);
        }
        *abort_flag = 0;
        fence_barrier_init();
        prefetch_tensormap(&tmap_qkv);
    }
    if (warp == kMmaWarp) {
        tmem_alloc(smem_u32(tmem_slot), kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    grid_dependency_wait();

    // Blocks of 256 query rows of one head, dealt out in turn: the CTAs in flight together share heads, so they read the same
    // k / v through L2.
    const int n_steps = (p.seq + kTile - 1) / kTile;    // steps of 128 keys
    auto give_up = [&](unsigned code) {
        report_timeout(p.status, code);
        *abort_flag = 1;
    };

    if (warp >= kProducerWarp) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kOtherRegs));
        if (warp == kProducerWarp && p.skip_loads == 0) {
            // -------------------------------------------------------------- TMA producer
            int      slot = 0, issued = 0, done = 0, q_loads[kQTiles] = {0, 0};
            uint32_t phase = 0;
            bool     ok = true;
            auto load_kv = [&](int col, int row, int b) {
                if (!mbar_wait_warp(slot_empty(slot), phase ^ 1u, abort_flag, p.wait_limit_ns)) {
                    give_up(0x3100u | (unsigned)slot);
                    ok = false;
                    return;
                }
                const uint32_t dst = smem_base + kRingOffset + slot * kTileBytes;
                if (elect_one()) {
                    mbar_arrive_expect_tx(slot_full(slot), (uint32_t)kTileBytes);
                    tma_load_3d(dst, &tmap_qkv, slot_full(slot), col, row, b);
                    tma_load_3d(dst + kBoxBytes, &tmap_qkv, slot_full(slot), col + 64, row, b);
                }
                ++issued;
                if (++slot == kSlots) {
                    slot = 0;
                    phase ^= 1u;
                }
            };
            for (int blk = blockIdx.x; ok && blk < p.blocks; blk += gridDim.x, ++done) {
                const int q0 = (blk % p.q_blocks) * (kQTiles * kTile);
                const int h  = (blk / p.q_blocks) % p.heads;
                const int b  = blk / (p.q_blocks * p.heads);
                const int col_q = h * kHeadDim, col_k = (p.heads + h) * kHeadDim, col_v = (2 * p.heads + h) * kHeadDim;
                load_kv(col_k, 0, b);
#pragma unroll
                for (int t = 0; t < kQTiles; ++t) {
                    if (!ok) {
                        break;
                    }
                    if (!mbar_wait_warp(q_empty(t), (uint32_t)((done & 1) ^ 1), abort_flag, p.wait_limit_ns)) {
                        give_up(0x3110u | (unsigned)t);
                        ok = false;
                        break;
                    }
                    const uint32_t dst = smem_base + kQOffset + t * kTileBytes;
                    if (elect_one()) {
                        mbar_arrive_expect_tx(q_full(t), (uint32_t)kTileBytes);
                        tma_load_3d(dst, &tmap_qkv, q_full(t), col_q, q0 + t * kTile, b);
                        tma_load_3d(dst + kBoxBytes, &tmap_qkv, q_full(t), col_q + 64, q0 + t * kTile, b);
                    }
                    ++q_loads[t];
                }
                for (int i = 0; ok && i < n_steps; ++i) {
                    load_kv(col_v, i * kTile, b);
                    if (ok && i + 1 < n_steps) {
                        load_kv(col_k, (i + 1) * kTile, b);
                    }
                }
            }
            // no copy may be in flight when the block leaves: wait (bounded) for the slots filled last, and for q
            auto settle = [&](uint32_t bar, uint32_t parity, unsigned code) {
                const uint64_t t0 = global_timer_ns();
                while (!mbar_try_wait(bar, parity)) {
                    if (global_timer_ns() - t0 > p.wait_limit_ns) {
                        report_timeout(p.status, code);
                        break;
                    }
                }
            };
            for (int i = 0; i < kSlots && i < issued; ++i) {
                if (slot == 0) {
                    slot = kSlots;
                    phase ^= 1u;
                }
                --slot;
                settle(slot_full(slot), phase, 0x3400u | (unsigned)slot);
            }
#pragma unroll
            for (int t = 0; t < kQTiles; ++t) {
                if (q_loads[t] > 0) {
                    settle(q_full(t), (uint32_t)((q_loads[t] - 1) & 1), 0x3410u | (unsigned)t);
                }
            }
        } else if (warp == kMmaWarp) {
            // -------------------------------------------------------------- MMA issuer of both query tiles
            constexpr uint32_t kAb = TypeTag<T>::value == LYRAQ_BF16 ? 1u : 0u;
            constexpr uint32_t idesc_qk = umma_idesc(1u, kAb, 128, kTile);
            constexpr uint32_t idesc_pv = umma_idesc(1u, kAb, 128, 128) | kIdescBMajorMN;
            unsigned bad = 0;
            auto     wait_for = [&](uint32_t bar, uint32_t parity, unsigned code) {
                if (!mbar_wait_warp(bar, parity, abort_flag, p.wait_limit_ns)) {
                    bad = code;
                    return false;
                }
                return true;
            };
            int      kslot = 0, vslot = 1;      // items of the ring alternate k, v, k, v, ...
            uint32_t kphase = 0, vphase = 0;
            auto advance = [&](int& slot, uint32_t& phase) {
                slot += 2;
                if (slot >= kSlots) {
                    slot -= kSlots;
                    phase ^= 1u;
                }
            };
            // S_t = Q_t K^T with the k tile in kslot; the second query tile gives it back.  One thread.
            auto issue_qk = [&](int t, bool last) {
                const uint64_t qdesc = umma_desc_k_sw128(smem_base + kQOffset + t * kTileBytes);
                const uint64_t kdesc = umma_desc_k_sw128(smem_base + kRingOffset + kslot * kTileBytes);
                const uint32_t d     = tmem_base + (uint32_t)(t * 128);
#pragma unroll
                for (int ks = 0; ks < 8; ++ks) {
                    const uint64_t off = (uint64_t)(((ks >> 2) * kBoxBytes + (ks & 3) * 32) >> 4);
                    mma_f16(d, qdesc + off, kdesc + off, idesc_qk, ks > 0 ? 1u : 0u);
                }
                tc_commit(s_full(t));
                if (t == 1) {
                    tc_commit(slot_empty(kslot));
                }
                if (last) {
                    tc_commit(q_empty(t));
                }
            };
            const int blocks = (p.blocks - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;   // of this CTA
            const int steps  = blocks * n_steps;
            bool ok = wait_for(slot_full(kslot), kphase, 0x3210u);
#pragma unroll 1
            for (int t = 0; t < kQTiles && ok; ++t) {
                ok = wait_for(q_full(t), 0u, 0x3200u);
                if (ok) {
                    tc_fence_after_sync();
                    if (elect_one()) {
                        issue_qk(t, n_steps == 1);
                    }
                }
            }
            advance(kslot, kphase);
            // Step g of the CTA, step i of its block: per query tile O (+)= P V, then the scores of step g + 1 over P, which those MMAs read
            // before, in order.
            int      i      = 0;
            uint32_t bphase = 0;    // parity of the block's number
#pragma unroll 1
            for (int g = 0; g < steps && ok; ++g) {
                const bool last = i == n_steps - 1;              // of the block
                const bool more = g + 1 < steps;
                const int  i2   = last ? 0 : i + 1;
                ok = wait_for(slot_full(vslot), vphase, 0x3230u) && (!more || wait_for(slot_full(kslot), kphase, 0x3211u));
#pragma unroll 1
                for (int t = 0; t < kQTiles && ok; ++t) {
                    const uint32_t o_acc = tmem_base + (uint32_t)(256 + t * 128);
                    const uint32_t p_in  = tmem_base + (uint32_t)(t * 128);
                    const uint64_t vdesc = umma_desc_mn_sw128(smem_base + kRingOffset + vslot * kTileBytes, (uint32_t)kBoxBytes);
                    const uint32_t acc   = i > 0 ? 1u : 0u;
                    if (i == 0 && !wait_for(o_empty(t), bphase ^ 1u, 0x3220u)) {
                        ok = false;
                        break;
                    }
                    if (last && more && !wait_for(q_full(t), bphase ^ 1u, 0x3201u)) {
                        ok = false;
                        break;
                    }
                    if (!wait_for(p_first(t), (uint32_t)(g & 1), 0x3240u)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after_sync();
                    if (elect_one()) {
#pragma unroll
                        for (int k4 = 0; k4 < 4; ++k4) {   // 16 keys each: 8 columns of P, 2048 bytes of v
                            mma_f16_ts(o_acc, p_in + (uint32_t)(k4 * 8), vdesc + (uint64_t)(k4 * 128), idesc_pv, k4 > 0 ? 1u : acc);
                        }
                    }
                    if (!wait_for(p_second(t), (uint32_t)(g & 1), 0x3241u)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after_sync();
                    if (elect_one()) {
#pragma unroll
                        for (int k4 = 4; k4 < 8; ++k4) {
                            mma_f16_ts(o_acc, p_in + (uint32_t)(k4 * 8), vdesc + (uint64_t)(k4 * 128), idesc_pv, 1u);
                        }
                        if (last) {
                            tc_commit(o_full(t));
                        }
                        if (t == 1) {
                            tc_commit(slot_empty(vslot));
                        }
                        if (more) {
                            issue_qk(t, i2 == n_steps - 1);
                        }
                    }
                }
                advance(vslot, vphase);
                advance(kslot, kphase);
                i = i2;
                if (last) {
                    bphase ^= 1u;
                }
            }
            if (!ok) {
                give_up(bad);
            }
        }
    } else if (warp >= kEpiWarp) {
        // ------------------------------------------------------------------ epilogue: O / l, rounded to T, stored as T or as e4m3 of that value
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kEpiRegs));
        const int    quadrant = warp & 3;
        const float* sums     = reinterpret_cast<const float*>(gen_base + kSumOffset);
        // Read once, ahead of the work: behind each block's waits the load and the division took 0.6 of 256 tokens' 9.65 us.  A scale that
        // belongs to no row is not read (out_scale[1] may be null).
        const float  qs0      = p.out_e4m3 && p.split > 0 ? 1.0f / ld_f32(p.out_scale[0]) : 1.0f;
        const float  qs1      = p.out_e4m3 && p.split < p.seq ? 1.0f / ld_f32(p.out_scale[1]) : 1.0f;
        bool         ok       = true;
        int          done     = 0;
        for (int blk = blockIdx.x; ok && blk < p.blocks; blk += gridDim.x, ++done) {
            const int q0 = (blk % p.q_blocks) * (kQTiles * kTile);
            const int h  = (blk / p.q_blocks) % p.heads;
            const int b  = blk / (p.q_blocks * p.heads);
#pragma unroll 1
            for (int t = 0; t < kQTiles; ++t) {
                const int       row   = q0 + t * kTile + quadrant * 32 + lane;   // row inside the sequence
                const int       part  = row >= p.split ? 1 : 0;
                const long long r_out = part ? row - p.split : row;
                if (!mbar_wait_lazy(l_full(t), (uint32_t)(done & 1), abort_flag, p.wait_limit_ns) ||
                    !mbar_wait_warp(o_full(t), (uint32_t)(done & 1), abort_flag, p.wait_limit_ns)) {
                    give_up(0x3320u | (unsigned)t);
                    ok = false;
                    break;
                }
                tc_fence_after_sync();
                const float     inv_l  = 1.0f / sums[t * kTile + quadrant * 32 + lane];
                const float     qs     = part ? qs1 : qs0;
                const uint32_t  o_addr = tmem_base + ((uint32_t)(quadrant * 32) << 16) + (uint32_t)(256 + t * 128);
                uint8_t*        dst    = static_cast<uint8_t*>(p.out[part]) +
                               ((long long)b * p.out_batch[part] + r_out * p.out_ld[part] + (long long)h * kHeadDim) * (p.out_e4m3 ? 1 : 2);
                auto value = [&](uint32_t lo, uint32_t hi) {
                    const float2 v = mul_f32x2(make_float2(__uint_as_float(lo), __uint_as_float(hi)), make_float2(inv_l, inv_l));
                    return Pair<T>::from_f32(v.x, v.y);
                };
                // the whole row is read before the first store: the accumulator and the sums may be overwritten while the rows go out
                auto release = [&]() {
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) {
                        mbar_arrive(o_empty(t));
                        mbar_arrive(l_empty(t));
                    }
                };
                if (q0 + t * kTile >= p.seq) {
                    release();   // a tile without rows: converting it all the same took 64 tokens 0.4 of 6.5 us
                } else if (p.out_e4m3) {
                    uint32_t w[32];
#pragma unroll
                    for (int cc = 0; cc < 4; ++cc) {
                        uint32_t o[32];
                        tmem_ld_32x32(o_addr + cc * 32, o);
                        tmem_ld_wait();
#pragma unroll
                        for (int k = 0; k < 8; ++k) {
                            const float2 q2 = make_float2(qs, qs);
                            const float2 x  = mul_f32x2(Pair<T>::to_f32(value(o[4 * k], o[4 * k + 1])), q2);
                            const float2 y  = mul_f32x2(Pair<T>::to_f32(value(o[4 * k + 2], o[4 * k + 3])), q2);
                            w[cc * 8 + k]   = f32x2_to_e4m3x2(x.x, x.y) | (f32x2_to_e4m3x2(y.x, y.y) << 16);
                        }
                    }
                    release();
                    if (row < p.seq) {
#pragma unroll
                        for (int k = 0; k < 8; ++k) {
                            reinterpret_cast<uint4*>(dst)[k] = make_uint4(w[4 * k], w[4 * k + 1], w[4 * k + 2], w[4 * k + 3]);
                        }
                    }
                } else {
                    uint32_t w[64];
#pragma unroll
                    for (int cc = 0; cc < 8; ++cc) {
                        uint32_t o[16];
                        tmem_ld_32x16(o_addr + cc * 16, o);
                        tmem_ld_wait();
#pragma unroll
                        for (int k = 0; k < 8; ++k) {
                            w[cc * 8 + k] = value(o[2 * k], o[2 * k + 1]);
                        }
                    }
                    release();
                    if (row < p.seq) {
#pragma unroll
                        for (int k = 0; k < 16; ++k) {
                            reinterpret_cast<uint4*>(dst)[k] = make_uint4(w[4 * k], w[4 * k + 1], w[4 * k + 2], w[4 * k + 3]);
                        }
                    }
                }
            }
        }
    } else {
        // ------------------------------------------------------------------ softmax, one thread per query row
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kSoftmaxRegs));
        const int      t        = warp >> 2;                                   // query tile
        const int      quadrant = warp & 3;                                    // tensor-memory lane quadrant of this warp
        const uint32_t lanes    = tmem_base + ((uint32_t)(quadrant * 32) << 16);
        const uint32_t s_addr   = lanes + (uint32_t)(t * 128);
        const uint32_t o_addr   = lanes + (uint32_t)(256 + t * 128);
        // A positive scale is folded into the exponent, where the order of the scores and the -inf of keys past the end survive it.  Any other
        // one (zero: a plain mean of the values) is multiplied in first.
        const float    c        = FOLD ? p.scale_log2 : 1.0f;
        float*         sums     = reinterpret_cast<float*>(gen_base + kSumOffset) + t * kTile + quadrant * 32 + lane;
        bool           ok       = true;
        uint32_t       g        = 0;                                           // steps, all blocks
        int            done     = 0;
        for (int blk = blockIdx.x; ok && blk < p.blocks; blk += gridDim.x, ++done) {
            float m = -INFINITY;                                               // reference maximum of this row (raw scores, if folded)
            float l = 0.0f;                                                    // sum of exp2((s - m) c)
#pragma unroll 1
            for (int i = 0; i < n_steps; ++i, ++g) {
                if (!mbar_wait_warp(s_full(t), g & 1u, abort_flag, p.wait_limit_ns)) {
                    give_up(0x3300u | (unsigned)t);
                    ok = false;
                    break;
                }
                tc_fence_after_sync();
                uint32_t s[128];
#pragma unroll
                for (int cc = 0; cc < 4; ++cc) {
                    tmem_ld_32x32(s_addr + cc * 32, s + cc * 32);
                }
                tmem_ld_wait();
                if (!FOLD) {
#pragma unroll
                    for (int k = 0; k < 128; ++k) {
                        s[k] = __float_as_uint(__uint_as_float(s[k]) * p.scale_log2);
                    }
                }
                const int valid = p.seq - i * kTile;                           // keys of this step inside the sequence
                if (valid < kTile) {
#pragma unroll
                    for (int k = 0; k < 128; ++k) {
                        if (k >= valid) {
                            s[k] = 0xff800000u;                                // -inf: zero-filled keys take no weight
                        }
                    }
                }
                float mx[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    mx[j] = max3(__uint_as_float(s[3 * j]), __uint_as_float(s[3 * j + 1]), __uint_as_float(s[3 * j + 2]));
                }
#pragma unroll
                for (int k = 12; k < 124; k += 8) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        mx[j] = max3(mx[j], __uint_as_float(s[k + 2 * j]), __uint_as_float(s[k + 2 * j + 1]));
                    }
                }
                mx[0] = max3(mx[0], __uint_as_float(s[124]), __uint_as_float(s[125]));
                mx[1] = max3(mx[1], __uint_as_float(s[126]), __uint_as_float(s[127]));
                const float mxx = max3(max3(mx[0], mx[1], mx[2]), mx[3], mx[3]);
                const bool finite = fabsf(mxx) < INFINITY;                     // else the row holds a NaN or an infinity, and comes out as NaN
                if (i == 0) {
                    m = finite ? mxx : 0.0f;
                    l = finite ? 0.0f : __uint_as_float(0x7fc00000u);
                } else {
                    const bool raise = !((mxx - m) * c <= kRescaleThreshold);
                    if (__any_sync(0xffffffffu, raise)) {
                        // S of this step was issued behind the previous step's P V, so the accumulator is at rest; the next P V
                        // waits for this step's P
                        const float f = raise ? ex2_approx((m - mxx) * c) : 1.0f;
                        if (raise) {
                            l = finite ? l * f : __uint_as_float(0x7fc00000u);
                            m = finite ? mxx : m;
                        }
#pragma unroll
                        for (int cc = 0; cc < 8; ++cc) {                       // rare path: small pieces keep the registers free
                            uint32_t o[16];
                            tmem_ld_32x16(o_addr + cc * 16, o);
                            tmem_ld_wait();
#pragma unroll
                            for (int k = 0; k < 16; ++k) {
                                o[k] = __float_as_uint(__uint_as_float(o[k]) * f);
                            }
                            tmem_st_32x16(o_addr + cc * 16, o);
                        }
                        tmem_st_wait();
                    }
                }
                const float2 c2   = make_float2(c, c);
                const float  nmc  = -m * c;
                const float2 nmc2 = make_float2(nmc, nmc);
                float2 sum_a = make_float2(0.0f, 0.0f), sum_b = make_float2(0.0f, 0.0f);
#pragma unroll
                for (int cc = 0; cc < 4; ++cc) {
                    uint32_t w[16];
#pragma unroll
                    for (int k = 0; k < 16; ++k) {
                        const float2 x = fma_f32x2(make_float2(__uint_as_float(s[cc * 32 + 2 * k]), __uint_as_float(s[cc * 32 + 2 * k + 1])), c2, nmc2);
                        const bool   poly = (k + 1) * kPolyPairs / 16 != k * kPolyPairs / 16;
                        const float2 e = poly ? ex2_poly(x) : make_float2(ex2_approx(x.x), ex2_approx(x.y));
                        if (k & 1) {
                            sum_b = add_f32x2(sum_b, e);
                        } else {
                            sum_a = add_f32x2(sum_a, e);
                        }
                        w[k] = Pair<T>::from_f32(e.x, e.y);
                    }
                    // P over the start of S: columns [16 cc, 16 cc + 16) hold keys [32 cc, 32 cc + 32)
                    tmem_st_32x16(s_addr + (uint32_t)(cc * 16), w);
                    if (cc & 1) {
                        tmem_st_wait();
                        tc_fence_before_sync();
                        __syncwarp();
                        if (lane == 0) {
                            mbar_arrive(cc == 1 ? p_first(t) : p_second(t));
                        }
                    }
                }
                const float2 sum = add_f32x2(sum_a, sum_b);
                l += sum.x + sum.y;
            }
            if (!ok) {
                break;
            }
            if (!mbar_wait_warp(l_empty(t), (uint32_t)((done & 1) ^ 1), abort_flag, p.wait_limit_ns)) {
                give_up(0x3310u | (unsigned)t);
                ok = false;
                break;
            }
            *sums = l;
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(l_full(t));
            }
        }
    }

    tc_fence_before_sync();
    __syncthreads();
    if (warp == kMmaWarp) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, kTmemCols);
    }
}

template<typename T, bool FOLD> static int launch(unsigned grid, const CUtensorMap& tm, const Params& p, cudaStream_t stream)
{
    static bool smem_raised[64] = {};
    const int   st = raise_dynamic_smem_once(attention_fwd_kernel<T, FOLD>, (int)kSmemTotal, smem_raised, "cudaFuncSetAttribute(attention_fwd_kernel)");
    if (st != LYRAQ_OK) {
        return st;
    }
    return cuda_status(launch_kernel(attention_fwd_kernel<T, FOLD>, grid, (unsigned)kThreads, (size_t)kSmemTotal, stream, 1u, tm, p),
                       "cudaLaunchKernelEx(attention_fwd_kernel)");
}

}  // namespace attn

// Test hook (lyraq_debug_attention_wait_test): a producer that never signals and a short wait limit, so that the path a
// timed-out wait takes -- status word, abort flag, every role leaving, tensor memory freed -- can be run without a fault.
static int                g_attn_skip_loads    = 0;
static unsigned long long g_attn_wait_limit_ns = kWaitLimitNs;

int launch_attention(void* out, int out_dtype, size_t out_ld, const float* out_scale, void* out2, size_t out2_ld,
                     const float* out2_scale, size_t split, const void* qkv, int dtype, size_t batch, size_t seq, int heads,
                     int head_dim, float softmax_scale, cudaStream_t stream)
{
    if (out == nullptr || qkv == nullptr) {
        return LYRAQ_ERR_INVALID_ARG;
    }
    if ((dtype != LYRAQ_BF16 && dtype != LYRAQ_F16) || head_dim != attn::kHeadDim || heads <= 0 ||
        (out_dtype != dtype && out_dtype != LYRAQ_E4M3)) {
        return LYRAQ_ERR_UNSUPPORTED;
    }
    if (batch == 0 || seq == 0) {
        return LYRAQ_OK;
    }
    if (out2 == nullptr) {
        split = seq;
    }
    const bool   e4m3 = out_dtype == LYRAQ_E4M3;
    const size_t esz  = e4m3 ? 1 : 2;
    if (split > seq || seq > 0x3fffffffu || batch > 0xffffu || (e4m3 && (out_scale == nullptr || (out2 != nullptr && out2_scale == nullptr)))) {
        return LYRAQ_ERR_INVALID_ARG;
    }
    const size_t width = (size_t)heads * attn::kHeadDim;
    if (out_ld < width || (out2 != nullptr && out2_ld < width) || !aligned16(out) || !aligned16(out2) || !aligned16(qkv) ||
        (out_ld * esz) % 16 != 0 || (out2_ld * esz) % 16 != 0) {
        return LYRAQ_ERR_INVALID_ARG;
    }
    static EncodeTiledFnAttn encode = nullptr;
    if (encode == nullptr) {
        void*                           fp = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fp, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) {
            return LYRAQ_ERR_CUDA;
        }
        encode = reinterpret_cast<EncodeTiledFnAttn>(fp);
    }
    CUtensorMap      tm;
    const cuuint64_t dims[3]    = {(cuuint64_t)(3 * width), (cuuint64_t)seq, (cuuint64_t)batch};
    const cuuint64_t strides[2] = {(cuuint64_t)(3 * width * 2), (cuuint64_t)(3 * width * 2) * seq};
    const cuuint32_t box[3]     = {64, (cuuint32_t)attn::kTile, 1};
    const cuuint32_t estr[3]    = {1, 1, 1};
    if (encode(&tm, CU_TENSOR_MAP_DATA_TYPE_UINT16, 3, const_cast<void*>(qkv), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) {
        record_cuda_error(cudaErrorInvalidValue, "cuTensorMapEncodeTiled refused the qkv tensor map");
        return LYRAQ_ERR_CUDA;
    }
    attn::Params p{};
    p.out[0]       = out;
    p.out[1]       = out2;
    p.out_ld[0]    = (long long)out_ld;
    p.out_ld[1]    = (long long)out2_ld;
    p.out_batch[0] = (long long)(split * out_ld);
    p.out_batch[1] = (long long)((seq - split) * out2_ld);
    p.out_scale[0] = out_scale;
    p.out_scale[1] = out2_scale;
    p.out_e4m3     = e4m3 ? 1 : 0;
    p.split        = (int)split;
    p.seq          = (int)seq;
    p.heads        = heads;
    p.q_blocks     = (int)((seq + attn::kQTiles * attn::kTile - 1) / (attn::kQTiles * attn::kTile));
    p.scale_log2   = softmax_scale * 1.4426950408889634f;
    p.status       = status_word_ptr();
    p.wait_limit_ns = g_attn_wait_limit_ns;
    p.skip_loads    = g_attn_skip_loads;
    if (p.status == nullptr) {
        return LYRAQ_ERR_CUDA;
    }
    const int sms       = device_sm_count();
    p.blocks            = (int)(batch * (size_t)heads * (size_t)p.q_blocks);
    const unsigned grid = (unsigned)(p.blocks < sms ? p.blocks : sms);
    if (dtype == LYRAQ_BF16) {
        return p.scale_log2 > 0.0f ? attn::launch<__nv_bfloat16, true>(grid, tm, p, stream) : attn::launch<__nv_bfloat16, false>(grid, tm, p, stream);
    }
    return p.scale_log2 > 0.0f ? attn::launch<__half, true>(grid, tm, p, stream) : attn::launch<__half, false>(grid, tm, p, stream);
}

}  // namespace lyraq

extern "C" int lyraq_debug_attention_wait_test(int skip_loads, unsigned int wait_limit_ms)
{
    lyraq::g_attn_skip_loads    = skip_loads ? 1 : 0;
    lyraq::g_attn_wait_limit_ns = wait_limit_ms == 0 ? lyraq::sm100::kWaitLimitNs : (unsigned long long)wait_limit_ms * 1000000ull;
    return LYRAQ_OK;
}

extern "C" int lyraq_attention(void* out, int out_dtype, size_t out_ld, const float* out_scale, void* out2, size_t out2_ld,
                               const float* out2_scale, size_t split, const void* qkv, int dtype, size_t batch, size_t seq_len,
                               int heads, int head_dim, float softmax_scale, void* stream)
{
    return lyraq::launch_attention(out, out_dtype, out_ld, out_scale, out2, out2_ld, out2_scale, split, qkv, dtype, batch, seq_len,
                                   heads, head_dim, softmax_scale, (cudaStream_t)stream);
}
