// What the attention with two score maps per head needs beside the attention kernels themselves: the rotation of
// queries and keys with the cache write, and the join of a head's two maps.
//
// Rotation: of a head's first `rot` columns, pair i turns by the angle position * freqs[i]: columns i and i + rot / 2
// ("rotate half", `halves`), or the neighbours 2i and 2i + 1.  Angle, sine and cosine are 32-bit, and both are multiplied by
// `mag`.  Later columns pass.
//
// Join: with a1, a2 the two maps' results of one head, o = a1 - lam * a2, then o / sqrt(mean(o^2) + eps) * post, and with
// a gate (pre-activations [rows, H * V], a view of wider rows) times sigmoid(gate), element by element.
#include "attention_flex.cuh"

template <class T>
__device__ __forceinline__ float turned(const T* src, int c, int rot, int halves, const float* cs, const float* sn) {
    const int half = rot >> 1;
    if (!halves) {
        if (c >= rot) return to_f<T>(src[c]);
        const float own = to_f<T>(src[c]), other = to_f<T>(src[c ^ 1]);
        return c & 1 ? own * cs[c >> 1] + other * sn[c >> 1] : own * cs[c >> 1] - other * sn[c >> 1];
    }
    if (c < half) return to_f<T>(src[c]) * cs[c] - to_f<T>(src[c + half]) * sn[c];
    if (c < rot) return to_f<T>(src[c]) * cs[c - half] + to_f<T>(src[c - half]) * sn[c - half];
    return to_f<T>(src[c]);
}

// gridDim.y blocks per row share the row's heads out.  q [rows, nq heads, D] and k [rows, n_kv_heads, D] are views of
// wider rows (row strides in elements, heads side by side); v [rows, v_heads * v_dim] likewise.  The turned queries go
// to q_out (contiguous), the turned keys and the values to the row's place in the cache.
template <class T>
__global__ void rotate_store_kernel(const T* __restrict__ q, long long q_row, const T* __restrict__ k, long long k_row,
                                         const T* __restrict__ v, long long v_row, T* __restrict__ q_out, SbBatch batch, SbFlex p,
                                         const float* __restrict__ freqs, int rot, float mag, int halves, int nq, int* status) {
    extern __shared__ float trig[];
    pdl_wait();
    const int row = blockIdx.x, D = p.k_dim, half = rot >> 1;
    int slot, pos;
    row_place(batch, row, slot, pos);
    float* cs = trig;
    float* sn = trig + half;
    for (int i = threadIdx.x; i < half; i += blockDim.x) {
        float s, c;
        sincosf((float)pos * freqs[i], &s, &c);
        cs[i] = c * mag;
        sn[i] = s * mag;
    }
    __syncthreads();
    // units of work: a query head, a key head, a value head; the blocks of a row share them out
    const int vh = p.v_heads > 0 ? p.v_heads : p.n_kv_heads, per = p.n_kv_heads / vh;
    const int units = nq + p.n_kv_heads + vh;
    for (int u = blockIdx.y; u < units; u += gridDim.y) {
        if (u < nq) {
            const T* src = q + row * q_row + (long long)u * D;
            T* dst = q_out + ((long long)row * nq + u) * D;
            for (int c = threadIdx.x; c < D; c += blockDim.x) dst[c] = from_f<T>(turned<T>(src, c, rot, halves, cs, sn));
        } else if (u < nq + p.n_kv_heads) {
            const int h = u - nq;
            const long long tok = flex_token(p, slot, pos, h);
            if (tok < 0) {
                if (threadIdx.x == 0) atomicOr(status, SB_STATUS_NO_PAGE);
                continue;
            }
            const T* src = k + row * k_row + (long long)h * D;
            T* dst = (T*)p.k + tok * D;
            for (int c = threadIdx.x; c < D; c += blockDim.x) dst[c] = from_f<T>(turned<T>(src, c, rot, halves, cs, sn));
        } else {
            const int h = u - nq - p.n_kv_heads;
            const long long tok = flex_value_token(p, flex_token(p, slot, pos, h * per), h * per);
            if (tok < 0) continue;
            const T* src = v + row * v_row + (long long)h * p.v_dim;
            T* dst = (T*)p.v + tok * p.v_row;
            for (int c = threadIdx.x; c < p.v_dim; c += blockDim.x) dst[c] = src[c];
        }
    }
}

#define RS_ROWS 4

// Many bfloat16 rows: RS_ROWS rows per block, their sines and cosines taken once, 16 bytes of a head per thread and turn (of a
// turned head with `halves` the two pieces whose columns turn together).  A number a thread, with the sines taken again by each of
// a row's four blocks: 4,599 rows of 20 heads of 64 and 128 values 29 us, this 12; 3,333 of 24 heads of 128 and 512 values 47, this 17.
__global__ void __launch_bounds__(256)
rotate_store_rows_kernel(const __nv_bfloat16* __restrict__ q, long long q_row, const __nv_bfloat16* __restrict__ k, long long k_row,
                         const __nv_bfloat16* __restrict__ v, long long v_row, __nv_bfloat16* __restrict__ q_out, SbBatch batch, SbFlex p,
                         const float* __restrict__ freqs, int rot, float mag, int halves, int nq, int* status) {
    typedef __nv_bfloat16 bf;
    extern __shared__ float trig[];       // [RS_ROWS][rot]: cosines, then sines
    __shared__ int slot_s[RS_ROWS], pos_s[RS_ROWS];
    pdl_wait();
    const int row0 = blockIdx.x * RS_ROWS, nr = min(RS_ROWS, batch.n_rows - row0), D = p.k_dim, half = rot >> 1;
    if (threadIdx.x < nr) row_place(batch, row0 + threadIdx.x, slot_s[threadIdx.x], pos_s[threadIdx.x]);
    __syncthreads();
    for (int e = threadIdx.x; e < nr * half; e += blockDim.x) {
        const int r = e / half, i = e - r * half;
        float s, c;
        sincosf((float)pos_s[r] * freqs[i], &s, &c);
        trig[r * rot + i] = c * mag;
        trig[r * rot + half + i] = s * mag;
    }
    __syncthreads();
    const int vh = p.v_heads > 0 ? p.v_heads : p.n_kv_heads, per = p.n_kv_heads / vh;
    const int turned = halves ? half / 8 : rot / 8, pieces = turned + (D - rot) / 8, v_pieces = p.v_dim / 8;
    const int head_items = (nq + p.n_kv_heads) * pieces, items = head_items + vh * v_pieces;
    for (int it = threadIdx.x; it < nr * items; it += blockDim.x) {
        const int r = it / items, i = it - r * items, row = row0 + r, slot = slot_s[r], pos = pos_s[r];
        if (i >= head_items) {
            const int h = (i - head_items) / v_pieces, c = (i - head_items - h * v_pieces) * 8;
            const long long tok = flex_value_token(p, flex_token(p, slot, pos, h * per), h * per);
            if (tok >= 0)
                *reinterpret_cast<uint4*>((bf*)p.v + tok * p.v_row + c) = *reinterpret_cast<const uint4*>(v + row * v_row + (long long)h * p.v_dim + c);
            continue;
        }
        const int u = i / pieces, c = i - u * pieces;
        const bf* src;
        bf* dst;
        if (u < nq) {
            src = q + row * q_row + (long long)u * D;
            dst = q_out + ((long long)row * nq + u) * D;
        } else {
            const long long tok = flex_token(p, slot, pos, u - nq);
            if (tok < 0) {
                atomicOr(status, SB_STATUS_NO_PAGE);
                continue;
            }
            src = k + row * k_row + (long long)(u - nq) * D;
            dst = (bf*)p.k + tok * D;
        }
        if (c >= turned) {
            const int at = rot + (c - turned) * 8;
            *reinterpret_cast<uint4*>(dst + at) = *reinterpret_cast<const uint4*>(src + at);
            continue;
        }
        const float* cs = trig + r * rot;
        const float* sn = cs + half;
        float x[8], y[8];
        load_bf16<8>(src + c * 8, x);
        if (halves) {
            float a[8], b[8];
            load_bf16<8>(src + half + c * 8, y);
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                a[e] = x[e] * cs[c * 8 + e] - y[e] * sn[c * 8 + e];
                b[e] = y[e] * cs[c * 8 + e] + x[e] * sn[c * 8 + e];
            }
            store_bf16<8>(dst + c * 8, a);
            store_bf16<8>(dst + half + c * 8, b);
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                y[2 * e] = x[2 * e] * cs[c * 4 + e] - x[2 * e + 1] * sn[c * 4 + e];
                y[2 * e + 1] = x[2 * e + 1] * cs[c * 4 + e] + x[2 * e] * sn[c * 4 + e];
            }
            store_bf16<8>(dst + c * 8, y);
        }
    }
}

// diff_combine in bfloat16 with heads of 32 N values, N of them a lane and access: 4,599 rows of 8 heads of 64, a number a lane 14
// us, this 9; 3,333 rows of 8 heads of 128 with a gate 16, this 11.
template <int N>
__global__ void diff_combine_vec_kernel(const __nv_bfloat16* __restrict__ a, __nv_bfloat16* __restrict__ out, int rows, int H, int G, float lam,
                                        float eps, float post, const __nv_bfloat16* __restrict__ gate, long long gate_ld) {
    constexpr int V = 32 * N;
    pdl_wait();
    const long long wid = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (wid >= (long long)rows * H) return;
    const long long row = wid / H;
    const int h = (int)(wid % H), per = H / G, g = h / per, r = h % per;
    float x[N], y[N], ss = 0.f;
    load_bf16<N>(a + ((row * 2 * H) + (long long)(2 * g) * per + r) * V + lane * N, x);
    load_bf16<N>(a + ((row * 2 * H) + (long long)(2 * g + 1) * per + r) * V + lane * N, y);
#pragma unroll
    for (int e = 0; e < N; ++e) {
        x[e] = fmaf(-lam, y[e], x[e]);
        ss = fmaf(x[e], x[e], ss);
    }
    ss = warp_sum(ss);
    const float mul = post / sqrtf(ss / (float)V + eps);
    if (gate != nullptr) {
        load_bf16<N>(gate + row * gate_ld + (long long)h * V + lane * N, y);
#pragma unroll
        for (int e = 0; e < N; ++e) x[e] = x[e] * mul / (1.0f + expf(-y[e]));
    } else {
#pragma unroll
        for (int e = 0; e < N; ++e) x[e] *= mul;
    }
    store_bf16<N>(out + (row * H + h) * V + lane * N, x);
}

// One warp per (row, head).  a [rows, 2 H, V] holds the maps in the order (key/value head, map, head of the group).
template <class T>
__global__ void diff_combine_kernel(const T* __restrict__ a, T* __restrict__ out, int rows, int H, int G, int V, float lam, float eps,
                                    float post, const T* __restrict__ gate, long long gate_ld) {
    pdl_wait();
    const long long wid = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (wid >= (long long)rows * H) return;
    const long long row = wid / H;
    const int h = (int)(wid % H), per = H / G, g = h / per, r = h % per;
    const T* a1 = a + ((row * 2 * H) + (long long)(2 * g) * per + r) * V;
    const T* a2 = a + ((row * 2 * H) + (long long)(2 * g + 1) * per + r) * V;
    float ss = 0.f;
    for (int c = lane; c < V; c += 32) {
        const float o = fmaf(-lam, to_f<T>(a2[c]), to_f<T>(a1[c]));
        ss = fmaf(o, o, ss);
    }
    ss = warp_sum(ss);
    const float mul = post / sqrtf(ss / (float)V + eps);
    T* o_row = out + (row * H + h) * V;
    if (gate == nullptr) {
        for (int c = lane; c < V; c += 32) o_row[c] = from_f<T>(fmaf(-lam, to_f<T>(a2[c]), to_f<T>(a1[c])) * mul);
        return;
    }
    const T* g_row = gate + row * gate_ld + (long long)h * V;
    for (int c = lane; c < V; c += 32)
        o_row[c] = from_f<T>(fmaf(-lam, to_f<T>(a2[c]), to_f<T>(a1[c])) * mul / (1.0f + expf(-to_f<T>(g_row[c]))));
}

extern "C" {

int sb_rotate_store(int dtype, const void* q, long long q_row, const void* k, long long k_row, const void* v, long long v_row,
                         void* q_out, SbBatch batch, SbFlex p, const float* freqs, int rot, float mag, int halves, int nq, int* status,
                    cudaStream_t stream) {
    if (batch.n_rows <= 0) return 0;
    if (rot < 0 || rot % 2 || rot > p.k_dim || (rot > 0 && freqs == nullptr)) return (int)cudaErrorInvalidValue;
    const int threads = p.k_dim >= 128 || p.v_dim >= 128 ? 128 : 64;
    const int vh = p.v_heads > 0 ? p.v_heads : p.n_kv_heads, units = nq + p.n_kv_heads + vh;
    // few rows: a block per head, so that a decode step's rows are spread over the SMs; many rows: a few blocks per row
    const int per_row = batch.n_rows >= 1024 ? min(units, 4) : (batch.n_rows >= 128 ? min(units, 8) : min(units, 64));
    dim3 grid(batch.n_rows, per_row);
    const size_t smem = (size_t)rot * sizeof(float);
    // Below 256 rows the blocks per head of the kernel above reach more SMs than blocks of four rows would (us, above / four rows; 24 heads
    // of 64 and of 128): 128 rows 4.5 / 4.7 and 4.9 / 6.5, 200 4.9 / 4.7 and 5.5 / 6.4, 256 6.4 / 4.7 and 6.8 / 6.4.
    if (dtype == SB_BF16 && batch.n_rows >= 256 && p.k_dim % 8 == 0 && p.v_dim % 8 == 0 && p.v_row % 8 == 0 && rot % (halves ? 16 : 8) == 0
        && q_row % 8 == 0 && k_row % 8 == 0 && v_row % 8 == 0 && rot <= 1024 && sb_aligned(16, q, k, v, q_out, p.k, p.v)) {
        typedef __nv_bfloat16 bf;
        sb_launch(rotate_store_rows_kernel, (batch.n_rows + RS_ROWS - 1) / RS_ROWS, 256, RS_ROWS * smem, stream, (const bf*)q, q_row, (const bf*)k,
                  k_row, (const bf*)v, v_row, (bf*)q_out, batch, p, freqs, rot, mag, halves, nq, status);
        SB_LAUNCH_CHECK();
    }
    if (dtype == SB_F32)
        sb_launch(rotate_store_kernel<float>, grid, threads, smem, stream, (const float*)q, q_row, (const float*)k, k_row,
                  (const float*)v, v_row, (float*)q_out, batch, p, freqs, rot, mag, halves, nq, status);
    else
        sb_launch(rotate_store_kernel<__nv_bfloat16>, grid, threads, smem, stream, (const __nv_bfloat16*)q, q_row,
                  (const __nv_bfloat16*)k, k_row, (const __nv_bfloat16*)v, v_row, (__nv_bfloat16*)q_out, batch, p, freqs, rot, mag, halves, nq,
                  status);
    SB_LAUNCH_CHECK();
}

int sb_diff_combine(int dtype, const void* a, void* out, int rows, int H, int G, int V, float lam, float eps, float post,
                    const void* gate, long long gate_ld, cudaStream_t stream) {
    if (rows <= 0) return 0;
    if (H < 1 || G < 1 || H % G) return (int)cudaErrorInvalidValue;
    const long long warps = (long long)rows * H;
    const int threads = 128;
    const unsigned int blocks = (unsigned int)((warps * 32 + threads - 1) / threads);
    typedef __nv_bfloat16 bf;
    if (dtype == SB_BF16 && V == 64 && gate_ld % 2 == 0 && sb_aligned(4, a, out, gate))
        sb_launch(diff_combine_vec_kernel<2>, blocks, threads, 0, stream, (const bf*)a, (bf*)out, rows, H, G, lam, eps, post, (const bf*)gate,
                  gate_ld);
    else if (dtype == SB_BF16 && V == 128 && gate_ld % 4 == 0 && sb_aligned(8, a, out, gate))
        sb_launch(diff_combine_vec_kernel<4>, blocks, threads, 0, stream, (const bf*)a, (bf*)out, rows, H, G, lam, eps, post, (const bf*)gate,
                  gate_ld);
    else if (dtype == SB_F32)
        sb_launch(diff_combine_kernel<float>, blocks, threads, 0, stream, (const float*)a, (float*)out, rows, H, G, V, lam, eps, post,
                  (const float*)gate, gate_ld);
    else
        sb_launch(diff_combine_kernel<__nv_bfloat16>, blocks, threads, 0, stream, (const __nv_bfloat16*)a, (__nv_bfloat16*)out, rows, H,
                  G, V, lam, eps, post, (const __nv_bfloat16*)gate, gate_ld);
    SB_LAUNCH_CHECK();
}

}  // extern "C"
