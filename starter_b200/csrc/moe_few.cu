// The experts of a step of few rows (decoding), bfloat16: a block takes an expert and 16 of its columns and serves all pairs
// (row, k) that chose the expert with one read of the weights (moe.cu says what is computed).
//
// What bounds it: the weights of the experts that were chosen.  The weights are the left operand of mma.sync (16 columns x 16
// inputs), the pairs' rows the right one (8 pairs); both go straight from global memory into registers: a lane reads 16 bytes of a
// weight row and of a pair's row, and the inputs stand in the product in the order in which the lanes hold them.  The block's
// four warps share the inputs out 32 at a time and add their sums up in shared memory, in the order of the warps.  Put in the
// order of their experts, gathered and handed to the library's grouped product, the pairs of a step cost nine launches and, for 96
// pairs of 16 experts of 3 x 1,024 x 512, 38 us a layer; this takes 19 (50 MB: 8 at the copy bandwidth).  Eight warps a block with the reads
// of a turn behind one another took 27.
#include "common.cuh"
#include "mma_utils.cuh"

#define MF_WARPS 4
#define MF_DEEP 4           // reads of 32 inputs that a warp has in flight
#define MF_NT 2            // groups of 8 pairs that one read of the weights serves
#define MF_MAX_PAIRS 1024

__device__ __forceinline__ uint4 mf_load(const __nv_bfloat16* p) { return *reinterpret_cast<const uint4*>(p); }

__device__ __forceinline__ void mf_mma(float (&c)[4], const uint4& a, const uint4& b, const uint4& x) {
    const unsigned int lo[4] = {a.x, b.x, a.y, b.y}, hi[4] = {a.z, b.z, a.w, b.w};
    mma_bf16(c, lo, x.x, x.y);
    mma_bf16(c, hi, x.z, x.w);
}

// An expert that every row of the step takes beside the chosen ones (a shared expert): its columns are blocks of the same launches,
// the first ones, since it is the widest.
struct MfShared {
    const __nv_bfloat16* x;
    const __nv_bfloat16* w;
    __nv_bfloat16* out;
    int rows, K, n_cols, silu;
    float alpha, limit;
};

// GATE_UP: out[pair][c] = act(gate_c, up_c) of x = h's row pair / top, w = [2 n_cols][K] per expert, gate over up.  Otherwise
// out[pair][c] = w_c x with x = the pair's own row, w = [n_cols][K] per expert.
template <bool GATE_UP, bool SHARED>
__global__ void __launch_bounds__(32 * MF_WARPS, 3)
moe_few_kernel(const __nv_bfloat16* __restrict__ x_in, const int* __restrict__ chosen, const __nv_bfloat16* __restrict__ w_in,
               __nv_bfloat16* __restrict__ out_in, int n_pairs, int top_in, int K_in, int n_cols_in, float alpha_in, float limit_in, int silu_in,
               MfShared shared) {
    constexpr int M = GATE_UP ? 2 : 1;
    __shared__ int list[MF_MAX_PAIRS];
    __shared__ int count_s;
    __shared__ float red[MF_WARPS][M][MF_NT][16][9];
    pdl_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    // Without a shared expert a block's expert and column are its place in the grid, and what it reads are the launch's arguments.
    const int first_blocks = SHARED ? (shared.n_cols + 15) / 16 : 0, per_expert = (n_cols_in + 15) / 16;
    const bool all = SHARED && (int)blockIdx.x < first_blocks;
    const int b0 = blockIdx.x - first_blocks, e = all ? 0 : SHARED ? b0 / per_expert : blockIdx.y;
    const int c0 = (all ? blockIdx.x : SHARED ? b0 % per_expert : blockIdx.x) * 16;
    const __nv_bfloat16* __restrict__ x = all ? shared.x : x_in;
    const __nv_bfloat16* __restrict__ w = all ? shared.w : w_in;
    __nv_bfloat16* __restrict__ out = all ? shared.out : out_in;
    const int K = all ? shared.K : K_in, n_cols = all ? shared.n_cols : n_cols_in, silu = all ? shared.silu : silu_in, top = all ? 1 : top_in;
    const float alpha = all ? shared.alpha : alpha_in, limit = all ? shared.limit : limit_in;
    if (all) {
        for (int i = threadIdx.x; i < shared.rows; i += 32 * MF_WARPS) list[i] = i;
        if (threadIdx.x == 0) count_s = shared.rows;
    } else if (warp == 0) {
        int n = 0;
        for (int p0 = 0; p0 < n_pairs; p0 += 32) {
            const bool hit = p0 + lane < n_pairs && chosen[p0 + lane] == e;
            const unsigned int mask = __ballot_sync(0xffffffffu, hit);
            if (hit) list[n + __popc(mask & ((1u << lane) - 1u))] = p0 + lane;
            n += __popc(mask);
        }
        if (lane == 0) count_s = n;
    }
    __syncthreads();
    const int count = count_s;
    const __nv_bfloat16* wa[M];     // this lane's two rows of each matrix; rows past the last one read the last and are not stored
    const __nv_bfloat16* wb[M];
#pragma unroll
    for (int m = 0; m < M; ++m) {
        const __nv_bfloat16* base = w + ((long long)e * M + m) * n_cols * K + t * 8;
        wa[m] = base + (long long)min(c0 + g, n_cols - 1) * K;
        wb[m] = base + (long long)min(c0 + g + 8, n_cols - 1) * K;
    }
    for (int first = 0; first < count; first += 8 * MF_NT) {
        const __nv_bfloat16* xr[MF_NT];
        bool have[MF_NT];
#pragma unroll
        for (int i = 0; i < MF_NT; ++i) {
            have[i] = first + i * 8 + g < count;
            const int pair = have[i] ? list[first + i * 8 + g] : 0;
            xr[i] = x + (long long)(GATE_UP ? pair / top : pair) * K + t * 8;
        }
        float acc[M][MF_NT][4];
#pragma unroll
        for (int m = 0; m < M; ++m)
#pragma unroll
            for (int i = 0; i < MF_NT; ++i)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[m][i][q] = 0.f;
        for (int k0 = warp * 32; k0 < K; k0 += MF_DEEP * MF_WARPS * 32) {
            uint4 a[MF_DEEP][M], b[MF_DEEP][M], xv[MF_DEEP][MF_NT];
#pragma unroll
            for (int u = 0; u < MF_DEEP; ++u) {
                const int k = k0 + u * MF_WARPS * 32;
                const bool in = k < K;
#pragma unroll
                for (int m = 0; m < M; ++m) {
                    a[u][m] = in ? mf_load(wa[m] + k) : make_uint4(0u, 0u, 0u, 0u);
                    b[u][m] = in ? mf_load(wb[m] + k) : make_uint4(0u, 0u, 0u, 0u);
                }
#pragma unroll
                for (int i = 0; i < MF_NT; ++i) xv[u][i] = in && have[i] ? mf_load(xr[i] + k) : make_uint4(0u, 0u, 0u, 0u);
            }
#pragma unroll
            for (int u = 0; u < MF_DEEP; ++u)
#pragma unroll
                for (int m = 0; m < M; ++m)
#pragma unroll
                    for (int i = 0; i < MF_NT; ++i) mf_mma(acc[m][i], a[u][m], b[u][m], xv[u][i]);
        }
#pragma unroll
        for (int m = 0; m < M; ++m)
#pragma unroll
            for (int i = 0; i < MF_NT; ++i)
#pragma unroll
                for (int q = 0; q < 4; ++q) red[warp][m][i][g + (q >> 1) * 8][2 * t + (q & 1)] = acc[m][i][q];
        __syncthreads();
#pragma unroll
        for (int i = 0; i < MF_NT; ++i) {
            const int col = threadIdx.x & 15, j = threadIdx.x >> 4, at = first + i * 8 + j, c = c0 + col;
            if (at < count && c < n_cols) {
                float s[M];
#pragma unroll
                for (int m = 0; m < M; ++m) {
                    s[m] = 0.f;
#pragma unroll
                    for (int v = 0; v < MF_WARPS; ++v) s[m] += red[v][m][i][col][j];
                }
                float y = s[0];
                if (GATE_UP) {
                    float gt = rnd<__nv_bfloat16>(s[0]), up = rnd<__nv_bfloat16>(s[M - 1]);
                    if (silu) {
                        const float a = gt / (1.0f + expf(-gt));
                        y = (all ? rnd<__nv_bfloat16>(a) : a) * up;   // a dense feed-forward rounds silu(gate) first
                    } else {
                        gt = fminf(gt, limit);
                        up = fminf(fmaxf(up, -limit), limit);
                        y = gt / (1.0f + expf(-alpha * gt)) * (up + 1.0f);
                    }
                }
                out[(long long)list[at] * n_cols + c] = __float2bfloat16_rn(y);
            }
        }
        __syncthreads();
    }
}

extern "C" {

// h [rows, width], act [n_pairs, ff], down [n_pairs, width]; w_gate_up [experts, 2 ff, width], w_down [experts, width, ff];
// width and ff multiples of 32, everything 16-byte aligned.  s_ff > 0: the shared expert's s_gate_up [2 s_ff, width], s_down [width, s_ff],
// s_act [rows, s_ff] and s_out [rows, width] under the same conditions.
int sb_moe_few(const void* h, const int* chosen, const void* w_gate_up, const void* w_down, void* act, void* down, int n_pairs, int top,
               int n_experts, int width, int ff, float alpha, float limit, int silu, const void* s_gate_up, const void* s_down, void* s_act,
               void* s_out, int s_ff, float s_alpha, float s_limit, int s_silu, cudaStream_t stream) {
    if (n_pairs <= 0 || n_experts <= 0) return 0;
    if (n_pairs > MF_MAX_PAIRS || n_experts > 65535 || width % 32 || ff % 32 || top < 1 || !sb_aligned(16, h, w_gate_up, w_down, act, down) ||
        s_ff < 0 || s_ff % 32 || (s_ff > 0 && !sb_aligned(16, s_gate_up, s_down, s_act, s_out)))
        return (int)cudaErrorInvalidValue;
    typedef __nv_bfloat16 bf;
    const int rows = s_ff > 0 ? n_pairs / top : 0;
    const MfShared up = {(const bf*)h, (const bf*)s_gate_up, (bf*)s_act, rows, width, s_ff, s_silu, s_alpha, s_limit};
    const MfShared dn = {(const bf*)s_act, (const bf*)s_down, (bf*)s_out, rows, s_ff, width, 0, 0.f, 0.f};
    if (rows == 0) {
        sb_launch(moe_few_kernel<true, false>, dim3((ff + 15) / 16, n_experts), 32 * MF_WARPS, 0, stream, (const bf*)h, chosen, (const bf*)w_gate_up,
                  (bf*)act, n_pairs, top, width, ff, alpha, limit, silu, up);
        sb_launch(moe_few_kernel<false, false>, dim3((width + 15) / 16, n_experts), 32 * MF_WARPS, 0, stream, (const bf*)act, chosen, (const bf*)w_down,
                  (bf*)down, n_pairs, top, ff, width, 0.f, 0.f, 0, dn);
        SB_LAUNCH_CHECK();
    }
    const long long b1 = (long long)((ff + 15) / 16) * n_experts + (s_ff + 15) / 16, b2 = (long long)((width + 15) / 16) * (n_experts + 1);
    if (b1 > 0x7fffffff || b2 > 0x7fffffff) return (int)cudaErrorInvalidValue;
    sb_launch(moe_few_kernel<true, true>, dim3((unsigned int)b1), 32 * MF_WARPS, 0, stream, (const bf*)h, chosen, (const bf*)w_gate_up, (bf*)act, n_pairs,
              top, width, ff, alpha, limit, silu, up);
    sb_launch(moe_few_kernel<false, true>, dim3((unsigned int)b2), 32 * MF_WARPS, 0, stream, (const bf*)act, chosen, (const bf*)w_down, (bf*)down, n_pairs,
              top, ff, width, 0.f, 0.f, 0, dn);
    SB_LAUNCH_CHECK();
}

}  // extern "C"
