// FP8 linear for few tokens: Y[m,n] = T(epi(alpha s_x s_w (X W^T) + beta R + bias)) with so few rows of X that the tiles of
// gemm_tcgen05_kernel (128 or 256 rows of X, all of K) leave most of the chip idle.
//
// What bounds it is the weight: every byte of W is read once (28 MB for a modulation linear of FLUX, 4.4 us of HBM), the
// arithmetic is negligible.  So the operands change places -- 128 rows of W are the M side of the MMA, the rows of X its
// N side (16, the rest zero-filled by TMA), which wastes no tensor memory and no loads on absent rows -- and
// K is split over the CTAs of a cluster until all SMs stream: a CTA owns one 128-row block of W and 1/S of K.  The S partial
// products meet through distributed shared memory: each CTA of the cluster owns 1/S of the block's token columns, receives
// the others' partials for them and adds them in rank order, so the result does not depend on timing.
// Measured with the quantize of X in front, dense kernel -> this one: one row of [9216, 3072] 14.7 -> 9.1 us, of [18432, 3072] 19.3 ->
// 13.3, 8 rows of [3072, 12288] 29.5 -> 12.0, 16 rows of [12288, 3072] 18.1 -> 14.2.  The store per partial value, 0.1 to 0.25 us a row,
// is what keeps it to 16 rows, and to fewer for small K (few_tokens in gemm_dense.cu; 64 rows of [9216, 3072]: 34 us against 13).
//
//   warp 0  lane 0: TMA producer (W 128 x 128 B, X 16 x 128 B per stage).  Before it waits for the kernels in front of it, it
//           asks its share of W into L2: the weight stream starts while the previous kernel (usually the quantize of X)
//           still runs.  A prefetch is not a read: whatever that kernel writes is what the loads behind the wait see.  It asks for the
//           whole share at once, so of a weight beyond L2's 126 MB some lines may be fetched twice (236 MB of [15360, 15360]: 50 us,
//           4.7 TB/s; the dense kernel takes 69 for one row).
//   warp 1  lane 0: MMA issuer; the warp owns tensor memory
//   warps 2-5: accumulator -> shared memory of the owning CTA -> sum, epilogue, store
// All waits are bounded.  A timeout sets the status word and the abort flag of every CTA of the cluster: the sums a CTA stores
// need the partial products of all of them, so when one gives up none of the cluster stores anything.
#include "common.cuh"
#include "sm100_ptx.cuh"
#include "gemm_skinny.cuh"

namespace lyraq {

using namespace sm100;

int make_tmap_bytes_2d(CUtensorMap* map, const void* base, uint64_t rows, uint64_t k_bytes, uint64_t row_stride_bytes,
                       uint32_t box_rows, uint32_t box_bytes, bool swizzle128);  // gemm_dense.cu

namespace skinny {

constexpr int kWRows   = 128;
constexpr int kBlockK  = 128;
constexpr int kWTile   = kWRows * kBlockK;   // 16 KB
constexpr int kThreads = 192;

constexpr int kRows      = kSkinnyRows;      // N side of the MMA: rows of X, the missing ones zero
constexpr int kStages    = 5;                // two CTAs share an SM
constexpr int kStage     = kWTile + kRows * kBlockK;
constexpr int kRedOffset = kStages * kStage;
constexpr int kRedBytes  = kRows * kWRows * 4;
constexpr int kBarOffset = kRedOffset + kRedBytes;
constexpr int kSmemTotal = kBarOffset + 256 + 1024;
static_assert(kSmemTotal <= 115000, "");

__device__ __forceinline__ void tma_prefetch_2d(const CUtensorMap* m, int x, int y)
{
    asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global [%0, {%1, %2}];" ::"l"(reinterpret_cast<uint64_t>(m)), "r"(x), "r"(y) : "memory");
}

__device__ __forceinline__ void st_cluster_f32(uint32_t cluster_addr, float v)
{
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(cluster_addr), "f"(v) : "memory");
}

__device__ __forceinline__ void st_cluster_u32(uint32_t cluster_addr, uint32_t v)
{
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cluster_addr), "r"(v) : "memory");
}

template<typename T>
__device__ __forceinline__ void finish(const SkinnyParams& p, float acc, float scale, int m, int n)
{
    const size_t at = (size_t)m * (size_t)p.N + (size_t)n;
    float        t  = acc * scale;
    if (p.residual != nullptr) {
        t = fmaf(p.beta, to_f32(reinterpret_cast<const T*>(p.residual)[at]), t);
    }
    if (p.bias != nullptr) {
        t += to_f32(reinterpret_cast<const T*>(p.bias)[n]);
    }
    if (p.gelu) {
        t = gelu_tanh_f32(t);
    }
    reinterpret_cast<T*>(p.C)[at] = from_f32<T>(t);
}

__global__ void __launch_bounds__(kThreads, 2)
gemm_skinny_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, const SkinnyParams p)
{
    constexpr uint32_t kTmemCols = 32;   // the smallest allocation
    constexpr uint32_t kIdesc    = umma_idesc(1u, 0u, kWRows, kRows);

    extern __shared__ uint8_t smem_raw[];
    // the dynamic shared window starts at the same offset in every CTA of the kernel, so the layout is that of the peers too
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t*       gen_base  = smem_raw + (smem_base - smem_u32(smem_raw));
    const uint32_t bars      = smem_base + kBarOffset;
    auto full_bar  = [&](int s) { return bars + 8u * s; };
    auto empty_bar = [&](int s) { return bars + 8u * (kStages + s); };
    const uint32_t acc_bar    = bars + 8u * (2 * kStages);
    uint32_t*      tmem_slot  = reinterpret_cast<uint32_t*>(gen_base + kBarOffset + 8 * (2 * kStages + 1));
    volatile int*  abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = warp_index();
    const int lane = threadIdx.x & 31;
    const int rank = (int)cluster_ctarank();
    const int n0   = (int)blockIdx.x / p.splits * kWRows;
    const int kb0  = (int)((long long)p.num_kb * rank / p.splits);
    const int kb1  = (int)((long long)p.num_kb * (rank + 1) / p.splits);
    const uint64_t wait_limit_ns = (uint64_t)p.wait_limit_ms * 1000000u;
    // records a wait that ran out and stops the whole cluster; its writes are visible to the peers behind the barrier in front of the sums
    auto give_up = [&](unsigned code) {
        report_timeout(p.status, code);
        for (int r = 0; r < p.splits; ++r) {
            st_cluster_u32(map_to_cta(smem_u32(const_cast<int*>(abort_flag)), (uint32_t)r), 1u);
        }
    };

    grid_launch_dependents();
    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        mbar_init(acc_bar, 1);
        *abort_flag = 0;
        fence_barrier_init();
        for (int kb = kb0; kb < kb1; ++kb) {
            tma_prefetch_2d(&tmap_w, kb * kBlockK, n0);
        }
        prefetch_tensormap(&tmap_x);
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(tmem_slot), kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    cluster_sync_all();   // every CTA of the cluster runs before a peer writes to its shared memory
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    grid_dependency_wait();

    if (warp == 0) {
        if (elect_one()) {
            int      stage = 0, issued = 0;
            uint32_t phase = 0;
            for (int kb = kb0; kb < kb1 && rank != p.stalled_rank; ++kb) {
                if (!mbar_wait(empty_bar(stage), phase ^ 1u, abort_flag, wait_limit_ns)) {
                    give_up(0x4100u | (unsigned)stage);
                    break;
                }
                const uint32_t dst = smem_base + stage * kStage;
                mbar_arrive_expect_tx(full_bar(stage), (uint32_t)kStage);
                tma_load_2d(dst, &tmap_w, full_bar(stage), kb * kBlockK, n0);
                tma_load_2d(dst + kWTile, &tmap_x, full_bar(stage), kb * kBlockK, 0);
                ++issued;
                if (++stage == kStages) {
                    stage = 0;
                    phase ^= 1u;
                }
            }
            // no copy may be in flight when the block leaves
            int      s  = stage;
            uint32_t ph = phase;
            for (int i = 0; i < kStages && i < issued; ++i) {
                if (s == 0) {
                    s = kStages;
                    ph ^= 1u;
                }
                --s;
                const uint64_t t0 = global_timer_ns();
                while (!mbar_try_wait(full_bar(s), ph)) {
                    if (global_timer_ns() - t0 > wait_limit_ns) {
                        report_timeout(p.status, 0x4500u | (unsigned)s);
                        break;
                    }
                }
            }
        }
    } else if (warp == 1) {
        if (elect_one()) {
            int      stage = 0;
            uint32_t phase = 0;
            bool     ok    = true;
            for (int kb = kb0; kb < kb1; ++kb) {
                if (!mbar_wait(full_bar(stage), phase, abort_flag, wait_limit_ns)) {
                    give_up(0x4200u | (unsigned)stage);
                    ok = false;
                    break;
                }
                tc_fence_after_sync();
                const uint64_t adesc = umma_desc_k_sw128(smem_base + stage * kStage);
                const uint64_t bdesc = umma_desc_k_sw128(smem_base + stage * kStage + kWTile);
#pragma unroll
                for (int k = 0; k < kBlockK / 32; ++k) {
                    mma_f8f6f4(tmem_base, adesc + (uint64_t)(2 * k), bdesc + (uint64_t)(2 * k), kIdesc, (kb > kb0 || k > 0) ? 1u : 0u);
                }
                tc_commit(empty_bar(stage));
                if (++stage == kStages) {
                    stage = 0;
                    phase ^= 1u;
                }
            }
            if (ok) {
                tc_commit(acc_bar);
            }
        }
    }
    // ---- accumulator lane = row of W; the CTA of rank r owns the token columns [r NB / S, (r + 1) NB / S)
    const int slice = kRows / p.splits;
    const int wrow  = (warp & 3) * 32 + lane;
    if (warp >= 2) {
        if (!__all_sync(0xffffffffu, mbar_wait(acc_bar, 0u, abort_flag, wait_limit_ns))) {
            if (lane == 0) {
                give_up(0x4300u);
            }
        } else {
            tc_fence_after_sync();
            uint32_t v[kRows];
            tmem_ld_32x16(tmem_base + ((uint32_t)((warp & 3) * 32) << 16), v);
            tmem_ld_wait();
#pragma unroll
            for (int c = 0; c < kRows; ++c) {
                if (c < p.M) {
                    const int      owner = c / slice;
                    const uint32_t at    = smem_base + kRedOffset + (uint32_t)(((rank * slice + c - owner * slice) * kWRows + wrow) * 4);
                    st_cluster_f32(map_to_cta(at, (uint32_t)owner), __uint_as_float(v[c]));
                }
            }
        }
    }
    tc_fence_before_sync();
    cluster_sync_all();   // all partials of this CTA's columns have arrived
    tc_fence_after_sync();
    if (warp == 1) {
        tmem_dealloc(tmem_base, kTmemCols);
    }
    if (warp >= 2 && *abort_flag == 0 && n0 + wrow < p.N) {
        const float* red   = reinterpret_cast<const float*>(gen_base + kRedOffset);
        const float  scale = p.alpha * ld_f32(p.s_x) * ld_f32(p.s_w);
        for (int c = 0; c < slice; ++c) {
            const int m = rank * slice + c;
            if (m >= p.M) {
                break;
            }
            float acc = red[c * kWRows + wrow];
            for (int s = 1; s < p.splits; ++s) {
                acc += red[(s * slice + c) * kWRows + wrow];
            }
            if (p.c_dtype == LYRAQ_BF16) {
                finish<__nv_bfloat16>(p, acc, scale, m, n0 + wrow);
            } else if (p.c_dtype == LYRAQ_F16) {
                finish<__half>(p, acc, scale, m, n0 + wrow);
            } else {
                finish<float>(p, acc, scale, m, n0 + wrow);
            }
        }
    }
}

// Clusters of `size` CTAs that run at once, two CTAs to an SM: a cluster lies within one GPC, and clusters of 4 or 8 leave some of a
// GPC's SMs over.  Measured on a B200 (148 SMs), K = 4096, 4 rows: four CTAs along K 10.8 us with 71 tiles and 14.1 with 72, eight 7.5
// with 33 tiles and 10.0 with 34, two 18.4 with 148 and 23.1 with 149.  (cudaOccupancyMaxActiveClusters allows this kernel one CTA
// per SM, and two run.)
static long clusters_at_once(int size, int sms)
{
    return size == 2 ? sms : size == 4 ? sms * 71l / 148 : sms * 33l / 148;
}

// CTAs along K: as many (1, 2, 4 or 8) as keep the clusters within one wave, with at least four K blocks each.
static int pick_splits(long tiles, int num_kb, int sms)
{
    int s = 1;
    while (s < 8 && num_kb >= 4 * (2 * s) && tiles <= clusters_at_once(2 * s, sms)) {
        s *= 2;
    }
    return s;
}

}  // namespace skinny

// Test hook (lyraq_debug_skinny_wait_test)
static int          g_stalled_rank  = -1;
static unsigned int g_wait_limit_ms = kWaitLimitNs / 1000000;

int launch_gemm_skinny(const void* X, const void* W, SkinnyParams p, int sms, cudaStream_t stream)
{
    using namespace skinny;
    const int n_tiles = (p.N + kWRows - 1) / kWRows;
    p.num_kb          = (p.K + kBlockK - 1) / kBlockK;
    p.splits          = pick_splits(n_tiles, p.num_kb, sms);
    p.stalled_rank    = g_stalled_rank;
    p.wait_limit_ms   = g_wait_limit_ms;
    CUtensorMap tw, tx;
    int         st = make_tmap_bytes_2d(&tw, W, (uint64_t)p.N, (uint64_t)p.K, (uint64_t)p.K, kWRows, kBlockK, true);
    if (st != LYRAQ_OK) {
        return st;
    }
    st = make_tmap_bytes_2d(&tx, X, (uint64_t)p.M, (uint64_t)p.K, (uint64_t)p.K, kRows, kBlockK, true);
    if (st != LYRAQ_OK) {
        return st;
    }
    static bool smem_raised[64] = {};
    st = raise_dynamic_smem_once(gemm_skinny_kernel, kSmemTotal, smem_raised, "cudaFuncSetAttribute(gemm_skinny_kernel)");
    if (st != LYRAQ_OK) {
        return st;
    }
    return cuda_status(launch_kernel(gemm_skinny_kernel, (unsigned)(n_tiles * p.splits), (unsigned)kThreads, (size_t)kSmemTotal, stream,
                                     (unsigned)p.splits, tw, tx, p),
                       "cudaLaunchKernelEx(gemm_skinny_kernel)");
}

}  // namespace lyraq

extern "C" int lyraq_debug_skinny_wait_test(int stalled_rank, unsigned int wait_limit_ms)
{
    lyraq::g_stalled_rank  = stalled_rank;
    lyraq::g_wait_limit_ms = wait_limit_ms == 0 ? (unsigned int)(lyraq::sm100::kWaitLimitNs / 1000000) : wait_limit_ms;
    return LYRAQ_OK;
}
