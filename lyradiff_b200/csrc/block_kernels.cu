// The element-wise kernels that sit between the quantized linears of a FLUX single-stream block:
//   - QK RMSNorm + rotary embedding on the packed QKV projection (the attention's input),
//   - e4m3 quantize of a [rows, cols] tensor into a column window of a wider e4m3 matrix (the concat in front of
//     proj_out, so that attention output and MLP activation are never concatenated in 16-bit form),
//   - gate * y + residual (the block's output).
// All are HBM-bound streaming kernels with 16-byte accesses; arithmetic follows the reference's rounding steps.
#include <type_traits>

#include "common.cuh"

namespace lyraq {

int device_sm_count();  // gemm_dense.cu

// One thread owns 8 consecutive elements of one head; the head_dim / 8 threads of a head (8 or 16 consecutive lanes)
// reduce the sum of squares with shuffles.  Reference: fuseRmsNormAndRope
// (src/lyradiff/kernels/rope/flux_apply_rope.cu:8-76): inv = rsqrt(mean(x^2) + eps) in fp32; t = T(x * inv);
// t = T(t * scale); out.x = T(T(t.x * r0.x) + T(t.y * r0.y)); out.y = T(T(t.x * r1.x) + T(t.y * r1.y)); V heads are copied.
//
// A token's heads are taken by threads that each keep the same four pairs, so the rotation and the norm weights stay in registers over the
// heads and no index is divided; three vectors per thread are in flight.  Bound by memory: 113 MB at 4608 tokens x 24 heads in
// place, where it takes 16.9 us (30.8 with a flat index over all vectors, two 64-bit divisions each).  rope_split chooses the threads of a token.
//
// THREADS > 0: a block of THREADS takes a token at a time.  THREADS = 0: a block of 256 has 2^tpt_log2 threads to a token, several tokens at
// a time where that leaves room, and `chunks` blocks share a token.
template<typename T, int LANES, int THREADS, int FLIGHT>
__global__ void __launch_bounds__(THREADS > 0 ? THREADS : 256) rmsnorm_rope_kernel(T* out, const T* qkv, const T* scale, const T* rope,
                                                                                   float eps, size_t tokens, int heads, int tpt_log2, int chunks)
{
    using P2 = Pair<T>;
    grid_launch_dependents();
    grid_dependency_wait();
    constexpr int kHeadDim = LANES * 8;
    const int     part     = threadIdx.x % LANES;                    // which 8 elements of a head
    const int     n_q      = heads * LANES, n_qk = 2 * n_q;          // vectors of the q heads, of the q and k heads
    const int     n_vec    = out == qkv ? n_qk : 3 * n_q;            // the v heads are copied unless they are in place
    const size_t  pitch    = (size_t)3 * heads * kHeadDim;
    const Vec16   sc_q     = ld_nc_16_keep(scale + part * 8);
    const Vec16   sc_k     = ld_nc_16_keep(scale + kHeadDim + part * 8);
    constexpr bool kSplit  = THREADS == 0;
    const int     tpt      = kSplit ? 1 << tpt_log2 : THREADS;
    const int     mine     = kSplit ? (int)threadIdx.x & (tpt - 1) : (int)threadIdx.x;
    const bool    shared   = kSplit && chunks > 1;                  // (spares other calls the division)
    const unsigned blk     = shared ? blockIdx.x / (unsigned)chunks : blockIdx.x, blks = shared ? gridDim.x / (unsigned)chunks : gridDim.x;
    const int     first    = (shared ? (int)(blockIdx.x - blk * (unsigned)chunks) * tpt : 0) + mine;    // of the token's vectors
    const int     step     = kSplit ? tpt * chunks : THREADS;
    const size_t  sub      = kSplit ? threadIdx.x >> tpt_log2 : 0;
    const size_t  at_once  = kSplit ? 256u >> tpt_log2 : 1;
    for (size_t t0 = blk * at_once; t0 < tokens; t0 += blks * at_once) {
        const bool   live = !kSplit || t0 + sub < tokens;
        const size_t tok  = live ? t0 + sub : t0;
        const int    n    = live ? n_vec : 0;
        // rope: [tokens, head_dim / 2, 2, 2]; this thread's 4 pairs are 16 consecutive values
        const T*    rp  = rope + tok * (size_t)(kHeadDim * 2) + part * 16;
        const Vec16 r0  = ld_nc_16_keep(rp);
        const Vec16 r1  = ld_nc_16_keep(rp + 8);
        const T*    src = qkv + tok * pitch;
        T*          dst = out + tok * pitch;
        // every lane of a warp takes part in the shuffles: those past the end reduce zeros and store nothing
        for (int v0 = first; v0 - mine < n_vec; v0 += FLIGHT * step) {
            uint4 raw[FLIGHT];
#pragma unroll
            for (int u = 0; u < FLIGHT; ++u) {
                const int vi = v0 + u * step;
                raw[u] = make_uint4(0u, 0u, 0u, 0u);
                if (vi < n) {
                    // an ordered plain load, not the read-only (.nc) path: with out == qkv this kernel writes what it reads
                    raw[u] = ld_u32x4(reinterpret_cast<const uint4*>(src + (size_t)vi * 8));
                }
            }
#pragma unroll
            for (int u = 0; u < FLIGHT; ++u) {
                if (kSplit && u > 0 && v0 - mine + u * step >= n_vec) {
                    break;
                }
                const int vi = v0 + u * step;
                Vec16     x;
                x.w[0] = raw[u].x; x.w[1] = raw[u].y; x.w[2] = raw[u].z; x.w[3] = raw[u].w;
                float f[8];
                unpack8<T>(x, f);
                float ss = 0.0f;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    ss = fmaf(f[j], f[j], ss);
                }
#pragma unroll
                for (int m = LANES / 2; m > 0; m >>= 1) {
                    ss += __shfl_xor_sync(0xffffffffu, ss, m);
                }
                if (vi < n_qk) {
                    const float inv = rsqrtf(ss / (float)kHeadDim + eps);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        uint32_t t = P2::from_f32(f[2 * j] * inv, f[2 * j + 1] * inv);
                        t          = P2::mul(t, vi < n_q ? sc_q.w[j] : sc_k.w[j]);
                        // pair j uses rope values 4j .. 4j+3 = (r0.x, r0.y, r1.x, r1.y): two words of r0 (j < 2) or r1
                        const uint32_t ra = (j < 2) ? r0.w[2 * j] : r1.w[2 * (j - 2)];        // (rope0.x, rope0.y)
                        const uint32_t rb = (j < 2) ? r0.w[2 * j + 1] : r1.w[2 * (j - 2) + 1];  // (rope1.x, rope1.y)
                        const float2 pa = P2::to_f32(P2::mul(t, ra));  // (T(t.x r0.x), T(t.y r0.y))
                        const float2 pb = P2::to_f32(P2::mul(t, rb));
                        x.w[j]          = P2::from_f32(pa.x + pa.y, pb.x + pb.y);  // fp32 sum of two T values, rounded once = T add
                    }
                }
                if (vi < n) {
                    st_16(dst + (size_t)vi * 8, x);
                }
            }
        }
    }
}

// Threads of a token.  The q and k heads of 24 x 128 are three vectors for each of 256 threads, with the v heads (out of place) 384: a block
// a token, three vectors a thread.  Elsewhere such a block idles or takes turns:
// - up to 1024 threads an SM a call is latency, so every vector gets a thread of a kernel whose code holds one vector only (with room for
//   three it took 0.1 to 0.25 us of 1.7 more: slower than the flat index).  Not at 257 to 767 vectors, which would double the blocks to save
//   a second vector: 64 tokens x 12 x 128 out of place 1.94 us so, 1.75 with a block a token;
// - up to 256 vectors, and up to 384 with many tokens (1024 x 12 x 64 out of place 3.4 us without, 2.75), several tokens share a block;
// - more than 1152 vectors of few tokens are shared by several blocks.
// Measured, us, a flat index over all vectors / 256 threads to every token / here: 65536 tokens x 1 head x 64 in place 12.0 / 114 / 7.3; 4608 x
// 2 x 128 4.4 / 10.0 / 3.0; out of place 1 x 24 x 128 1.6 / 2.3 / 1.45, 128 x 38 x 128 3.25 / 4.2 / 3.0, 256 x 24 x 128 3.2 / 3.9 / 2.8.
struct RopeSplit {
    int      threads, flight;    // of the kernel's template: 0 with 1 or 3, 256 or 384 with 3
    int      tpt_log2, chunks;
    unsigned grid;
};
static RopeSplit rope_split(size_t tokens, int heads, int lanes, bool in_place, int sms)
{
    const size_t n_vec = (size_t)heads * (size_t)lanes * (in_place ? 2 : 3);
    RopeSplit    r{0, 1, 3, 1, 0u};
    auto deal = [&](size_t vectors) {   // among 8 .. 256 threads, whole heads, and as many blocks as that takes
        r.tpt_log2 = 3;
        while (r.tpt_log2 < 8 && ((size_t)1 << r.tpt_log2 < vectors || (1 << r.tpt_log2) < lanes)) {
            ++r.tpt_log2;
        }
        r.chunks = (int)((vectors + 255) / 256);
    };
    deal(n_vec);
    if ((n_vec > 256 && n_vec < 768) || (tokens << r.tpt_log2) * (size_t)r.chunks > (size_t)sms * 1024) {
        r.flight = 3;
        if (n_vec <= 256 || (n_vec <= 384 && tokens > (size_t)sms * 4) || (n_vec > 1152 && tokens <= (size_t)sms * 2)) {
            deal((n_vec + 2) / 3);
        } else {
            r.threads = n_vec > 768 && n_vec <= 1152 ? 384 : 256;
            r.chunks  = 1;
        }
    }
    const size_t at_once = r.threads > 0 ? 1 : 256u >> r.tpt_log2;
    const size_t blocks  = (tokens + at_once - 1) / at_once;
    const size_t most    = (size_t)sms * 8;
    r.grid               = (unsigned)((blocks < most ? blocks : most) * (size_t)r.chunks);
    return r;
}

// dst[r, col0 + c] = e4m3(src[r, c] / scale) for a [rows, cols] source into a matrix with row pitch dst_ld bytes.
template<typename T>
__global__ void __launch_bounds__(256) fp8_cast_2d_kernel(uint8_t* dst, size_t dst_ld, const T* src, const float* scale,
                                                          size_t rows, int cols)
{
    grid_launch_dependents();
    grid_dependency_wait();
    const float  r       = 1.0f / ld_f32(scale);
    const int    vec_row = cols >> 3;
    const size_t total   = rows * (size_t)vec_row;
    const size_t stride  = (size_t)gridDim.x * blockDim.x;
    for (size_t vi = (size_t)blockIdx.x * blockDim.x + threadIdx.x; vi < total; vi += stride) {
        const size_t row = vi / vec_row;
        const int    c   = (int)(vi - row * vec_row) << 3;
        float        v[8];
        unpack8<T>(ld_nc_16(src + (vi << 3)), v);
        const uint32_t w0 = f32x2_to_e4m3x2(v[0] * r, v[1] * r) | (f32x2_to_e4m3x2(v[2] * r, v[3] * r) << 16);
        const uint32_t w1 = f32x2_to_e4m3x2(v[4] * r, v[5] * r) | (f32x2_to_e4m3x2(v[6] * r, v[7] * r) << 16);
        st_8(dst + row * dst_ld + c, w0, w1);
    }
}

// out = T(T(y * gate[b]) + x): fuseGateAndResidual (src/lyradiff/kernels/flux_single_transformer_block/
// flux_single_transformer_kernels.cu:43-65).
template<typename T>
__global__ void __launch_bounds__(256) gate_residual_kernel(T* out, const T* y, const T* gate, const T* x, size_t rows,
                                                            int rows_per_batch, int dim)
{
    using P2 = Pair<T>;
    grid_launch_dependents();
    grid_dependency_wait();
    const int    vec_row = dim >> 3;
    const size_t total   = rows * (size_t)vec_row;
    const size_t stride  = (size_t)gridDim.x * blockDim.x;
    for (size_t vi = (size_t)blockIdx.x * blockDim.x + threadIdx.x; vi < total; vi += stride) {
        const size_t row = vi / vec_row;
        const int    c   = (int)(vi - row * vec_row) << 3;
        const Vec16  a   = ld_nc_16(y + (vi << 3));
        const Vec16  r   = ld_nc_16(x + (vi << 3));
        const Vec16  g   = ld_nc_16_keep(gate + (row / (size_t)rows_per_batch) * (size_t)dim + c);
        Vec16        o;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            o.w[j] = P2::add(P2::mul(a.w[j], g.w[j]), r.w[j]);
        }
        st_16(out + (vi << 3), o);
    }
}

// w[i] = T(w[i] + T(lora[i] * T(alpha))), each step in T's own arithmetic: loadLora<T>
// (src/lyradiff/kernels/lora/load_lora.cu:6-14).  n8 vectors of 8 elements, then a scalar tail.  A thread has VECS vectors of
// each operand in flight: the kernel is a pass over memory and bound by the bytes outstanding, and two do better once every thread
// has many passes to make (38.4 -> 37.4 us at [12288, 3072] bf16 = 6.0 TB/s, 29.3 -> 28.4 at [9216, 3072]).  With few, one is better:
// 3.1 against 3.9 us at [1280, 1280], 4.5 against 5.6 at [3072, 1024], 13.9 against 14.3 at [4096, 3072] (five passes).
template<typename T, int VECS>
__global__ void __launch_bounds__(256) load_lora_kernel(T* w, const T* lora, size_t n, float alpha)
{
    using P2 = Pair<T>;
    grid_launch_dependents();
    grid_dependency_wait();
    const uint32_t a2     = P2::from_f32(alpha, alpha);
    const size_t   n8     = n >> 3;
    const size_t   stride = (size_t)gridDim.x * blockDim.x;
    const size_t   tid    = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (size_t v0 = tid; v0 < n8; v0 += VECS * stride) {
        Vec16 o[VECS], l[VECS];
#pragma unroll
        for (int q = 0; q < VECS; ++q) {
            if (q == 0 || v0 + q * stride < n8) {
                o[q] = ld_16(w + ((v0 + q * stride) << 3));
                l[q] = ld_nc_16(lora + ((v0 + q * stride) << 3));
            }
        }
#pragma unroll
        for (int q = 0; q < VECS; ++q) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                o[q].w[j] = P2::add(o[q].w[j], P2::mul(l[q].w[j], a2));
            }
        }
#pragma unroll
        for (int q = 0; q < VECS; ++q) {
            if (q == 0 || v0 + q * stride < n8) {
                st_16(w + ((v0 + q * stride) << 3), o[q]);
            }
        }
    }
    for (size_t i = (n8 << 3) + tid; i < n; i += stride) {
        const T t = from_f32<T>(to_f32(lora[i]) * to_f32(from_f32<T>(alpha)));  // exact product of two T values, one rounding
        w[i]      = from_f32<T>(to_f32(w[i]) + to_f32(t));
    }
}

static unsigned stream_grid(size_t nvec)
{
    size_t       g   = (nvec + 255) / 256;
    const size_t cap = 148 * 8;
    if (g > cap) {
        g = cap;
    }
    return g == 0 ? 1u : (unsigned)g;
}

}  // namespace lyraq

using namespace lyraq;

extern "C" {

int lyraq_rmsnorm_rope(void* out, const void* qkv, const void* scale, const void* rope, int dtype, double eps, size_t batch,
                       size_t seq_len, int heads, int head_dim, void* stream)
{
    if (batch * seq_len == 0) {
        return LYRAQ_OK;
    }
    if (out == nullptr || qkv == nullptr || scale == nullptr || rope == nullptr || heads <= 0) {
        return LYRAQ_ERR_INVALID_ARG;
    }
    if (!aligned16(out) || !aligned16(qkv) || !aligned16(scale) || !aligned16(rope)) {
        return LYRAQ_ERR_INVALID_ARG;
    }
    if ((head_dim != 64 && head_dim != 128) || seq_len > 0x7fffffffu || (dtype != LYRAQ_BF16 && dtype != LYRAQ_F16)) {
        return LYRAQ_ERR_UNSUPPORTED;
    }
    const size_t tokens = batch * seq_len;
    const int    sms    = device_sm_count();
    if (sms <= 0) {
        return LYRAQ_ERR_CUDA;
    }
    const RopeSplit split = rope_split(tokens, heads, head_dim / 8, out == qkv, sms);
    cudaStream_t    s     = (cudaStream_t)stream;
    auto launch = [&](auto* kernel, auto type) {
        using T = decltype(type);
        return launch_kernel(kernel, split.grid, split.threads > 0 ? (unsigned)split.threads : 256u, (size_t)0, s, 1u, (T*)out, (const T*)qkv,
                             (const T*)scale, (const T*)rope, (float)eps, tokens, heads, split.tpt_log2, split.chunks);
    };
    auto pick = [&](auto type, auto lanes) {
        using T             = decltype(type);
        constexpr int kLanes = decltype(lanes)::value;
        return split.flight == 1      ? launch(rmsnorm_rope_kernel<T, kLanes, 0, 1>, type)
               : split.threads == 0   ? launch(rmsnorm_rope_kernel<T, kLanes, 0, 3>, type)
               : split.threads == 256 ? launch(rmsnorm_rope_kernel<T, kLanes, 256, 3>, type)
                                      : launch(rmsnorm_rope_kernel<T, kLanes, 384, 3>, type);
    };
    auto pick_lanes = [&](auto type) {
        return head_dim == 128 ? pick(type, std::integral_constant<int, 16>{}) : pick(type, std::integral_constant<int, 8>{});
    };
    const cudaError_t e = dtype == LYRAQ_BF16 ? pick_lanes(__nv_bfloat16{}) : pick_lanes(__half{});
    return cuda_status(e, "cudaLaunchKernelEx(rmsnorm_rope_kernel)");
}

int lyraq_quant_fp8_2d(uint8_t* dst, size_t dst_ld, const void* src, int src_dtype, const float* scale, size_t rows,
                       size_t cols, void* stream)
{
    if (rows * cols == 0) {
        return LYRAQ_OK;
    }
    if (dst == nullptr || src == nullptr || scale == nullptr) {
        return LYRAQ_ERR_INVALID_ARG;
    }
    if (!aligned16(src) || (reinterpret_cast<uintptr_t>(dst) & 7u) != 0 || (dst_ld & 7u) != 0 || dst_ld < cols) {
        return LYRAQ_ERR_INVALID_ARG;
    }
    if ((cols & 7u) != 0 || cols > 0x7fffffffu) {
        return LYRAQ_ERR_UNSUPPORTED;
    }
    const unsigned grid = stream_grid(rows * (cols >> 3));
    cudaError_t    e;
    if (src_dtype == LYRAQ_BF16) {
        e = launch_kernel(fp8_cast_2d_kernel<__nv_bfloat16>, grid, 256u, (size_t)0, (cudaStream_t)stream, 1u, dst, dst_ld,
                          (const __nv_bfloat16*)src, scale, rows, (int)cols);
    } else if (src_dtype == LYRAQ_F16) {
        e = launch_kernel(fp8_cast_2d_kernel<__half>, grid, 256u, (size_t)0, (cudaStream_t)stream, 1u, dst, dst_ld,
                          (const __half*)src, scale, rows, (int)cols);
    } else {
        return LYRAQ_ERR_UNSUPPORTED;
    }
    return cuda_status(e, "cudaLaunchKernelEx(fp8_cast_2d_kernel)");
}

int lyraq_gate_residual(void* out, const void* y, const void* gate, const void* x, int dtype, size_t batch, size_t seq_len,
                        size_t dim, void* stream)
{
    if (batch * seq_len * dim == 0) {
        return LYRAQ_OK;
    }
    if (out == nullptr || y == nullptr || gate == nullptr || x == nullptr) {
        return LYRAQ_ERR_INVALID_ARG;
    }
    if (!aligned16(out) || !aligned16(y) || !aligned16(gate) || !aligned16(x)) {
        return LYRAQ_ERR_INVALID_ARG;
    }
    if ((dim & 7u) != 0 || dim > 0x7fffffffu || seq_len > 0x7fffffffu) {
        return LYRAQ_ERR_UNSUPPORTED;
    }
    const size_t   rows = batch * seq_len;
    const unsigned grid = stream_grid(rows * (dim >> 3));
    cudaError_t    e;
    if (dtype == LYRAQ_BF16) {
        using T = __nv_bfloat16;
        e = launch_kernel(gate_residual_kernel<T>, grid, 256u, (size_t)0, (cudaStream_t)stream, 1u, (T*)out, (const T*)y,
                          (const T*)gate, (const T*)x, rows, (int)seq_len, (int)dim);
    } else if (dtype == LYRAQ_F16) {
        using T = __half;
        e = launch_kernel(gate_residual_kernel<T>, grid, 256u, (size_t)0, (cudaStream_t)stream, 1u, (T*)out, (const T*)y,
                          (const T*)gate, (const T*)x, rows, (int)seq_len, (int)dim);
    } else {
        return LYRAQ_ERR_UNSUPPORTED;
    }
    return cuda_status(e, "cudaLaunchKernelEx(gate_residual_kernel)");
}

int lyraq_load_lora(void* weight, const void* lora, int dtype, float alpha, size_t n, void* stream)
{
    if (n == 0) {
        return LYRAQ_OK;
    }
    if (weight == nullptr || lora == nullptr || !aligned16(weight) || !aligned16(lora)) {
        return LYRAQ_ERR_INVALID_ARG;
    }
    const unsigned grid = stream_grid((n + 7) / 8);
    const bool     two  = (n >> 3) >= 8ull * 256 * grid;   // eight passes over the grid
    cudaError_t    e;
    if (dtype == LYRAQ_BF16) {
        using T = __nv_bfloat16;
        e = launch_kernel(two ? load_lora_kernel<T, 2> : load_lora_kernel<T, 1>, grid, 256u, (size_t)0, (cudaStream_t)stream, 1u, (T*)weight,
                          (const T*)lora, n, alpha);
    } else if (dtype == LYRAQ_F16) {
        using T = __half;
        e = launch_kernel(two ? load_lora_kernel<T, 2> : load_lora_kernel<T, 1>, grid, 256u, (size_t)0, (cudaStream_t)stream, 1u, (T*)weight,
                          (const T*)lora, n, alpha);
    } else {
        return LYRAQ_ERR_UNSUPPORTED;
    }
    return cuda_status(e, "cudaLaunchKernelEx(load_lora_kernel)");
}

}  // extern "C"
