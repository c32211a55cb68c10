// The element-wise kernels that sit between the quantized linears of a FLUX single-stream block:
//   - QK RMSNorm + rotary embedding on the packed QKV projection (the attention's input),
//   - e4m3 quantize of a [rows, cols] tensor into a column window of a wider e4m3 matrix (the concat in front of
//     proj_out, so that attention output and MLP activation are never concatenated in 16-bit form),
//   - gate * y + residual (the block's output).
// All are HBM-bound streaming kernels with 16-byte accesses; arithmetic follows the reference's rounding steps.
#include "common.cuh"

namespace lyraq {

int device_sm_count();  // gemm_dense.cu

// One thread owns 8 consecutive elements of one head; the head_dim / 8 threads of a head (8 or 16 consecutive lanes)
// reduce the sum of squares with shuffles.  Reference: fuseRmsNormAndRope
// (src/lyradiff/kernels/rope/flux_apply_rope.cu:8-76): inv = rsqrt(mean(x^2) + eps) in fp32; t = T(x * inv);
// t = T(t * scale); out.x = T(T(t.x * r0.x) + T(t.y * r0.y)); out.y = T(T(t.x * r1.x) + T(t.y * r1.y)); V heads are copied.
//
// A block takes a token at a time, so the rotation of a lane's four pairs and the norm weights stay in registers over the heads and no
// index is divided; three vectors per thread are in flight (the q and k heads of 24 x 128 are exactly that).  Bound by memory: 113 MB
// at 4608 tokens x 24 heads in place, where it takes 16.9 us (30.8 with a flat index over all vectors, two 64-bit divisions each).
template<typename T, int LANES>
__global__ void __launch_bounds__(256) rmsnorm_rope_kernel(T* out, const T* qkv, const T* scale, const T* rope, float eps,
                                                           size_t tokens, int seq_len, int heads)
{
    using P2 = Pair<T>;
    grid_launch_dependents();
    grid_dependency_wait();
    constexpr int kHeadDim = LANES * 8;
    constexpr int kFlight  = 3;
    const int     part     = threadIdx.x % LANES;                    // which 8 elements of a head
    const int     n_q      = heads * LANES, n_qk = 2 * n_q;          // vectors of the q heads, of the q and k heads
    const int     n_vec    = out == qkv ? n_qk : 3 * n_q;            // the v heads are copied unless they are in place
    const size_t  pitch    = (size_t)3 * heads * kHeadDim;
    const Vec16   sc_q     = ld_nc_16_keep(scale + part * 8);
    const Vec16   sc_k     = ld_nc_16_keep(scale + kHeadDim + part * 8);
    for (size_t tok = blockIdx.x; tok < tokens; tok += gridDim.x) {
        // rope: [tokens, head_dim / 2, 2, 2]; this thread's 4 pairs are 16 consecutive values
        const T*    rp  = rope + tok * (size_t)(kHeadDim * 2) + part * 16;
        const Vec16 r0  = ld_nc_16_keep(rp);
        const Vec16 r1  = ld_nc_16_keep(rp + 8);
        const T*    src = qkv + tok * pitch;
        T*          dst = out + tok * pitch;
        // every lane of a warp takes part in the shuffles: those past the end reduce zeros and store nothing
        for (int v0 = (int)threadIdx.x; v0 - (int)threadIdx.x < n_vec; v0 += kFlight * 256) {
            uint4 raw[kFlight];
#pragma unroll
            for (int u = 0; u < kFlight; ++u) {
                raw[u] = make_uint4(0u, 0u, 0u, 0u);
                if (v0 + u * 256 < n_vec) {
                    // an ordered plain load, not the read-only (.nc) path: with out == qkv this kernel writes what it reads
                    raw[u] = ld_u32x4(reinterpret_cast<const uint4*>(src + (size_t)(v0 + u * 256) * 8));
                }
            }
#pragma unroll
            for (int u = 0; u < kFlight; ++u) {
                const int vi = v0 + u * 256;
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
                if (vi < n_vec) {
                    st_16(dst + (size_t)vi * 8, x);
                }
            }
        }
    }
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
    const size_t   tokens = batch * seq_len;
    const int      sms    = device_sm_count();
    if (sms <= 0) {
        return LYRAQ_ERR_CUDA;
    }
    const unsigned grid   = (unsigned)(tokens < (size_t)sms * 8 ? tokens : (size_t)sms * 8);
    cudaStream_t   s      = (cudaStream_t)stream;
    cudaError_t    e;
    if (dtype == LYRAQ_BF16) {
        using T = __nv_bfloat16;
        e = (head_dim == 128) ? launch_kernel(rmsnorm_rope_kernel<T, 16>, grid, 256u, (size_t)0, s, 1u, (T*)out, (const T*)qkv,
                                              (const T*)scale, (const T*)rope, (float)eps, tokens, (int)seq_len, heads)
                              : launch_kernel(rmsnorm_rope_kernel<T, 8>, grid, 256u, (size_t)0, s, 1u, (T*)out, (const T*)qkv,
                                              (const T*)scale, (const T*)rope, (float)eps, tokens, (int)seq_len, heads);
    } else {
        using T = __half;
        e = (head_dim == 128) ? launch_kernel(rmsnorm_rope_kernel<T, 16>, grid, 256u, (size_t)0, s, 1u, (T*)out, (const T*)qkv,
                                              (const T*)scale, (const T*)rope, (float)eps, tokens, (int)seq_len, heads)
                              : launch_kernel(rmsnorm_rope_kernel<T, 8>, grid, 256u, (size_t)0, s, 1u, (T*)out, (const T*)qkv,
                                              (const T*)scale, (const T*)rope, (float)eps, tokens, (int)seq_len, heads);
    }
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
