// Row kernels of a model whose layers run in passes, of mixers that stand side by side, and of a squared-relu
// feed-forward:
//
//   add_rows     out = x + e + s      (32-bit rows; e: rows of the same shape or none; s: one vector for all rows or none)
//   add_bias     y += b               (in place, the sum 32-bit, rounded once)
//   scaled_sum   out = sa * a + sb * b
//   relu2        max(z, 0)^2
#include "common.cuh"

__global__ void add_rows_kernel(const float* __restrict__ x, const float* __restrict__ e, const float* __restrict__ s,
                                float* __restrict__ out, long long n, int width) {
    pdl_wait();
    pdl_launch_dependents();
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        float v = x[i];
        if (e != nullptr) v += e[i];
        if (s != nullptr) v += s[i % width];
        out[i] = v;
    }
}

template <class T>
__global__ void add_bias_kernel(T* __restrict__ y, const float* __restrict__ b, long long n, int width) {
    pdl_wait();
    pdl_launch_dependents();
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        y[i] = from_f<T>(to_f<T>(y[i]) + b[i % width]);
}

// bfloat16 rows whose width is a multiple of 8, 16 bytes a thread: 3,333 rows of 2,048, a number a thread 19 us, this 10.
__global__ void __launch_bounds__(256) add_bias_vec_kernel(__nv_bfloat16* __restrict__ y, const float* __restrict__ b, long long n8, int width8) {
    pdl_wait();
    pdl_launch_dependents();
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n8; i += (long long)gridDim.x * blockDim.x) {
        float f[8];
        load_bf16<8>(y + i * 8, f);
        const float* bb = b + (i % width8) * 8;
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] += bb[e];
        store_bf16<8>(y + i * 8, f);
    }
}

template <class T>
__global__ void scaled_sum_kernel(const T* __restrict__ a, float sa, const T* __restrict__ b, float sb, T* __restrict__ out, long long n) {
    pdl_wait();
    pdl_launch_dependents();
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        out[i] = from_f<T>(fmaf(sa, to_f<T>(a[i]), sb * to_f<T>(b[i])));
}

template <class T>
__global__ void relu2_kernel(const T* __restrict__ z, T* __restrict__ out, long long n) {
    pdl_wait();
    pdl_launch_dependents();
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float v = fmaxf(to_f<T>(z[i]), 0.f);
        out[i] = from_f<T>(v * v);
    }
}

// The same 16 bytes a thread: 3,333 rows of 8,192, a number a thread 27 us, this 15 (109 MB: 17 us at the copy bandwidth).
__global__ void __launch_bounds__(256) relu2_vec_kernel(const __nv_bfloat16* __restrict__ z, __nv_bfloat16* __restrict__ out, long long n8) {
    pdl_wait();
    pdl_launch_dependents();
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n8; i += (long long)gridDim.x * blockDim.x) {
        float f[8];
        load_bf16<8>(z + i * 8, f);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const float v = fmaxf(f[e], 0.f);
            f[e] = v * v;
        }
        store_bf16<8>(out + i * 8, f);
    }
}

static inline int flat_blocks(long long n) { return (int)((n + 255) / 256 < 8192 ? (n + 255) / 256 : 8192); }

extern "C" {

int sb_add_rows(const float* x, const float* e, const float* s, float* out, long long rows, int width, cudaStream_t stream) {
    if (rows <= 0) return 0;
    sb_launch(add_rows_kernel, flat_blocks(rows * width), 256, 0, stream, x, e, s, out, rows * width, width);
    SB_LAUNCH_CHECK();
}

int sb_add_bias(int dtype, void* y, const float* b, long long rows, int width, cudaStream_t stream) {
    if (rows <= 0) return 0;
    if (dtype == SB_F32) sb_launch(add_bias_kernel<float>, flat_blocks(rows * width), 256, 0, stream, (float*)y, b, rows * width, width);
    else if (width % 8 == 0 && sb_aligned(16, y))
        sb_launch(add_bias_vec_kernel, flat_blocks(rows * width / 8), 256, 0, stream, (__nv_bfloat16*)y, b, rows * width / 8, width / 8);
    else sb_launch(add_bias_kernel<__nv_bfloat16>, flat_blocks(rows * width), 256, 0, stream, (__nv_bfloat16*)y, b, rows * width, width);
    SB_LAUNCH_CHECK();
}

int sb_scaled_sum(int dtype, const void* a, float sa, const void* b, float sb, void* out, long long n, cudaStream_t stream) {
    if (n <= 0) return 0;
    if (dtype == SB_F32)
        sb_launch(scaled_sum_kernel<float>, flat_blocks(n), 256, 0, stream, (const float*)a, sa, (const float*)b, sb, (float*)out, n);
    else
        sb_launch(scaled_sum_kernel<__nv_bfloat16>, flat_blocks(n), 256, 0, stream, (const __nv_bfloat16*)a, sa, (const __nv_bfloat16*)b,
                  sb, (__nv_bfloat16*)out, n);
    SB_LAUNCH_CHECK();
}

int sb_relu2(int dtype, const void* z, void* out, long long n, cudaStream_t stream) {
    if (n <= 0) return 0;
    if (dtype == SB_F32) sb_launch(relu2_kernel<float>, flat_blocks(n), 256, 0, stream, (const float*)z, (float*)out, n);
    else if (n % 8 == 0 && sb_aligned(16, z, out))
        sb_launch(relu2_vec_kernel, flat_blocks(n / 8), 256, 0, stream, (const __nv_bfloat16*)z, (__nv_bfloat16*)out, n / 8);
    else sb_launch(relu2_kernel<__nv_bfloat16>, flat_blocks(n), 256, 0, stream, (const __nv_bfloat16*)z, (__nv_bfloat16*)out, n);
    SB_LAUNCH_CHECK();
}

}  // extern "C"
