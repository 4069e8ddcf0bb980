// Prompts through a layer's matrix memory (the "wkv", "gla" and "mlstm" mixers), 64 tokens at a time and all chunks of all
// sequences side by side, where wkv.cu, gla.cu and mlstm.cu walk a sequence token by token.  bfloat16 rows.
//
//   S_t = diag(a_t) S_(t-1) + b_t k_t v_t^T        o_t = q_t^T S_t        (wkv: the state before the token, plus u_i k_i v_t)
//
// (gla, wkv: a decay per key channel, b = 1; mlstm: one decay a = exp(f + m' - m) and one b = exp(i - m) per head.)  Over a chunk
// that starts from S0, with A(j, i) = a_(j+1) ... a_i:
//
//   O = P V + (q A(start, i)) S0        P[i][j] = sum_d q_i k_j b_j A(j, i)        S1 = A(start, end) S0 + sum_j (k_j b_j A(j, end)) v_j^T
//
// chunk_states_kernel leaves every chunk's own share of S1 and its decay, chunk_walk_kernel walks the chunks of a sequence in
// order (a multiplication and an addition per entry of the state) and leaves each chunk's S0, chunk_outputs_kernel takes
// the outputs with the head's norm and the gate.  chunk_gates_kernel first takes the mlstm's gates and running maximum.
//
// What bounds it: a walk token by token is one dependent chain per sequence and head (0.35 to 0.45 us a token, 32 blocks for one
// prompt on 148 SMs).  Here a block's work is a chunk's small products, bound by the instructions that prepare their operands
// (1.3 a clock with 16 warps an SM; the tensor pipe is nearly idle), so a decay is computed once and kept, and as many blocks as
// shared memory allows stand on an SM.  Measured on a B200, us a layer, walk -> this: wkv, 2,048 tokens, 32 heads of 64 x 64: 903
// -> 113 (shares 20, walk 8, outputs 79); gla, 4 sequences of 4,599 tokens, 8 heads of 64 x 128: 735 -> 97; mlstm, 3,333 tokens, 16
// heads of 64 x 128: 1,135 -> 118.
//
// 32 bits throughout: wherever a 32-bit number meets a tensor-core product it is written as three bfloat16 numbers (8 + 8 + 8
// bits: the number itself), against a bfloat16 operand three products, against another 32-bit one the six largest of nine.
// Per-channel decays are multiplied up, never divided out and never taken as differences of summed logarithms: inside 16
// tokens token by token, between groups of 16 by the groups' totals.  The mlstm's log-decays are summed in 64-bit and kept
// as two 32-bit numbers.
#include "common.cuh"
#include "mma_utils.cuh"

#define CM_L 64           // tokens of a chunk
#define CM_THREADS 256    // 8 warps: 4 groups of 16 tokens x 2 halves of the value columns
#define CM_PLD 24         // row stride of a 16 x 16 block of P: float2 reads of 4 rows x 4 lanes meet every bank once
#define CM_P_FLOATS (10 * 16 * CM_PLD)   // the blocks on and below the diagonal
#define CM_LEAST -160.0f  // log2 of a decay that is zero in 32-bit

enum { CM_WKV = 0, CM_GLA = 1, CM_MLSTM = 2 };

struct SbChunkMem {
    const void* q;          // rows `ld` elements apart, bfloat16: H heads of D (q, k) and of V (v, g) columns
    const void* k;
    const void* v;
    const void* g;
    long long ld;
    const float* z;         // wkv, gla: [rows][H D] inputs of the decays; mlstm: [rows, z_ld], gates at i_col + head, f_col + head
    long long z_ld;
    int i_col;
    int f_col;
    const float* bias;      // wkv: w0 [H D]; gla: bias [H D]; mlstm: input gate's [H]
    const float* bias2;     // wkv: u [H D]; mlstm: forget gate's [H]
    const float* norm;
    int norm_stride;        // from a head's norm weights to the next head's
    float eps;
    float inv_tau;
    float cap;
    float q_scale;
    float out_scale;
    float* state;
    long long state_stride;
    const void* last;       // wkv: the layer's input rows [rows][last_width], whose last row goes to the record at last_offset
    int last_width;
    int last_offset;
    void* y;
    long long y_ld;
    float* work;            // sb_chunk_memory_floats() floats
    long long head_floats;  // as given to sb_chunk_memory_floats()
    int H;
    int D;
    int V;
};

// The workspace of a launch over `nh` heads, cells of a step = n_rows / 64 + n_seqs.  Cell (s, c) = cu_q[s] / 64 + s + c.
struct ChunkWork {
    float* add;                 // [cell][nh][DP][VP] a chunk's own share of the state
    __nv_bfloat16* start;       // [cell][nh][3][DP][VP] the state at its start, in three parts
    float* decay;               // [cell][nh][DP] (mlstm: the first number only)
    float* norm;                // [cell][nh][DP] mlstm: the share of the normaliser, then the normaliser at the chunk's start
    float* gates;               // mlstm: [3][rows][H] log2 a, b, exp(-m); others: [rows][H D] the decays
    int head0;
    int nh;
};

__device__ __forceinline__ void cp_async_16_zfill(void* smem_dst, const void* gmem_src, bool valid) {
    const unsigned int s = (unsigned int)__cvta_generic_to_shared(smem_dst);
    const int n = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem_src), "r"(n));
}

// x, y as bfloat16 pairs h + m + l: 24 bits, the 32-bit numbers themselves.
__device__ __forceinline__ void split_three(float x, float y, unsigned int& h, unsigned int& m, unsigned int& l) {
    h = pack_bf16(x, y);
    x -= __uint_as_float(h << 16);
    y -= __uint_as_float(h & 0xffff0000u);
    m = pack_bf16(x, y);
    l = pack_bf16(x - __uint_as_float(m << 16), y - __uint_as_float(m & 0xffff0000u));
}

// The sequence and the chunk of a cell; false where the cell holds no rows.
__device__ __forceinline__ bool find_chunk(const SbBatch& b, int cell, int& s, int& row, int& nt) {
    const int lane = threadIdx.x & 31;
    s = -1;
    for (int base = 0; base < b.n_seqs; base += 32) {
        const int i = base + lane;
        const unsigned int before = __ballot_sync(0xffffffffu, i < b.n_seqs && (b.cu_q[i] >> 6) + i <= cell);
        s += __popc(before);
        if (before != 0xffffffffu) break;
    }
    const int first = b.cu_q[s], end = b.cu_q[s + 1];
    row = first + (cell - (first >> 6) - s) * CM_L;
    nt = min(CM_L, end - row);
    return nt > 0;
}

template <int KIND> __device__ __forceinline__ float channel_decay(float pre, float inv_tau) {
    if (KIND == CM_WKV) return expf(-expf(pre));
    const float ls = pre < 0.f ? pre - log1pf(expf(pre)) : -log1pf(expf(-pre));   // log(sigmoid(pre)) on the side that does not overflow
    return expf(ls * inv_tau);
}

__device__ __forceinline__ void unpack_eight(const uint4& raw, float scale, float* dst) {
    const unsigned int w[4] = {raw.x, raw.y, raw.z, raw.w};
    float f[8];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        f[2 * e] = __uint_as_float(w[e] << 16) * scale;
        f[2 * e + 1] = __uint_as_float(w[e] & 0xffff0000u) * scale;
    }
    *reinterpret_cast<float4*>(dst) = make_float4(f[0], f[1], f[2], f[3]);
    *reinterpret_cast<float4*>(dst + 4) = make_float4(f[4], f[5], f[6], f[7]);
}

// A chunk's rows of D bfloat16 numbers into 32-bit shared memory, zeros for what is not there.
template <int DP, int LD>
__device__ __forceinline__ void load_wide(float* dst, const void* src, long long ld, int row, int nt, int head, int D, float scale, int vec) {
    const __nv_bfloat16* base = (const __nv_bfloat16*)src + (long long)row * ld + (long long)head * D;
    if (vec) {
#pragma unroll 4
        for (int e = threadIdx.x; e < CM_L * DP / 8; e += CM_THREADS) {
            const int r = e / (DP / 8), c = (e % (DP / 8)) * 8;
            const uint4 raw = r < nt && c < D ? *reinterpret_cast<const uint4*>(base + r * ld + c) : make_uint4(0, 0, 0, 0);
            unpack_eight(raw, scale, dst + r * LD + c);
        }
    } else {
#pragma unroll 4
        for (int e = threadIdx.x; e < CM_L * DP; e += CM_THREADS) {
            const int r = e / DP, c = e % DP;
            dst[r * LD + c] = r < nt && c < D ? __bfloat162float(base[r * ld + c]) * scale : 0.f;
        }
    }
}

// The same in bfloat16.
template <int WP, int LD>
__device__ __forceinline__ void load_rows(__nv_bfloat16* dst, const void* src, long long ld, int row, int nt, int head, int W, int vec) {
    const __nv_bfloat16* base = (const __nv_bfloat16*)src + (long long)row * ld + (long long)head * W;
    if (vec) {
        for (int e = threadIdx.x; e < CM_L * WP / 8; e += CM_THREADS) {
            const int r = e / (WP / 8), c = (e % (WP / 8)) * 8;
            const bool ok = r < nt && c < W;
            cp_async_16_zfill(dst + r * LD + c, ok ? base + r * ld + c : base, ok);
        }
    } else {
        for (int e = threadIdx.x; e < CM_L * WP; e += CM_THREADS) {
            const int r = e / WP, c = e % WP;
            dst[r * LD + c] = r < nt && c < W ? base[r * ld + c] : __float2bfloat16_rn(0.f);
        }
    }
}

// The decays of a chunk's tokens per key channel, 1 for what is not there; `keep`: where they are left for load_kept_decays.
template <int KIND, int DP, int LD>
__device__ __forceinline__ void make_decays(float* dst, float* keep, const SbChunkMem& a, int row, int nt, int head, int vec) {
    const int HD = a.H * a.D;
    const float* base = a.z + (long long)row * HD + (long long)head * a.D;
    const float* bias = a.bias + (long long)head * a.D;
    keep += (long long)row * HD + (long long)head * a.D;
    if (vec) {
#pragma unroll 4
        for (int e = threadIdx.x; e < CM_L * DP / 4; e += CM_THREADS) {
            const int r = e / (DP / 4), c = (e % (DP / 4)) * 4;
            float4 d = make_float4(1.f, 1.f, 1.f, 1.f);
            if (r < nt && c < a.D) {
                const float4 z = *reinterpret_cast<const float4*>(base + (long long)r * HD + c);
                d.x = channel_decay<KIND>(z.x + bias[c], a.inv_tau);
                d.y = channel_decay<KIND>(z.y + bias[c + 1], a.inv_tau);
                d.z = channel_decay<KIND>(z.z + bias[c + 2], a.inv_tau);
                d.w = channel_decay<KIND>(z.w + bias[c + 3], a.inv_tau);
                *reinterpret_cast<float4*>(keep + (long long)r * HD + c) = d;
            }
            *reinterpret_cast<float4*>(dst + r * LD + c) = d;
        }
    } else {
        for (int e = threadIdx.x; e < CM_L * DP; e += CM_THREADS) {
            const int r = e / DP, c = e % DP;
            float d = 1.f;
            if (r < nt && c < a.D) {
                d = channel_decay<KIND>(base[(long long)r * HD + c] + bias[c], a.inv_tau);
                keep[(long long)r * HD + c] = d;
            }
            dst[r * LD + c] = d;
        }
    }
}

template <int DP, int LD>
__device__ __forceinline__ void load_kept_decays(float* dst, const float* kept, const SbChunkMem& a, int row, int nt, int head, int vec) {
    const int HD = a.H * a.D;
    const float* base = kept + (long long)row * HD + (long long)head * a.D;
    if (vec) {
#pragma unroll 4
        for (int e = threadIdx.x; e < CM_L * DP / 4; e += CM_THREADS) {
            const int r = e / (DP / 4), c = (e % (DP / 4)) * 4;
            if (r < nt && c < a.D) cp_async_16(dst + r * LD + c, base + (long long)r * HD + c);
            else *reinterpret_cast<float4*>(dst + r * LD + c) = make_float4(1.f, 1.f, 1.f, 1.f);
        }
    } else {
        for (int e = threadIdx.x; e < CM_L * DP; e += CM_THREADS) {
            const int r = e / DP, c = e % DP;
            dst[r * LD + c] = r < nt && c < a.D ? base[(long long)r * HD + c] : 1.f;
        }
    }
}

// mlstm, base 2: c (the sum of log-decays up to a token) as hi + lo, b, exp2(c), exp2(c_last - c) b, exp(-m).
struct alignas(16) GateSums {
    float hi[CM_L], lo[CM_L], b[CM_L], grown[CM_L], left[CM_L], em[CM_L];
    float total;
};

// One warp.
__device__ __forceinline__ void gate_sums(const float* gates, long long plane, int H, int head, int row, int nt, GateSums& c) {
    const int lane = threadIdx.x & 31;
    double step[2];
    float b[2], em[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const int t = 2 * lane + e;
        const long long at = (long long)(row + t) * H + head;
        step[e] = t < nt ? gates[at] : 0.f;
        b[e] = t < nt ? gates[plane + at] : 0.f;
        em[e] = t < nt ? gates[2 * plane + at] : 1.f;
    }
    double run = step[0] + step[1];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double up = __shfl_up_sync(0xffffffffu, run, o);
        if (lane >= o) run += up;
    }
    const double last = __shfl_sync(0xffffffffu, run, 31);
    const double at[2] = {run - step[1], run};
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const int t = 2 * lane + e;
        c.hi[t] = (float)at[e];
        c.lo[t] = (float)(at[e] - (double)(float)at[e]);
        c.b[t] = b[e];
        c.em[t] = em[e];
        c.grown[t] = exp2f((float)at[e]);
        c.left[t] = exp2f((float)(last - at[e])) * b[e];
    }
    if (lane == 0) c.total = exp2f((float)last);
}

// mlstm: gates, running maximum, log2 a, b and exp(-m) of every row.  One block per (sequence, head); 1,024 tokens at a time as a
// scan over (sum of f, maximum of i and what decays into it).  The record's maximum is brought up to date here.
#define CM_GATE_THREADS 1024
__global__ void __launch_bounds__(CM_GATE_THREADS) chunk_gates_kernel(SbChunkMem a, SbBatch batch, ChunkWork w) {
    __shared__ float sum_s[32], top_s[32], m_s[CM_GATE_THREADS + 1];
    const int s = blockIdx.x, head = w.head0 + blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float bi = a.bias[head], bf = a.bias2[head];
    pdl_wait();
    const int row0 = batch.cu_q[s], row1 = batch.cu_q[s + 1];
    if (row1 <= row0) return;
    float* mg = a.state + (long long)batch.seq_slot[s] * a.state_stride + (long long)a.H * a.D * a.V + (long long)a.H * a.D + head;
    const long long plane = (long long)batch.n_rows * a.H;
    if (tid == 0) m_s[0] = *mg;
    for (int t0 = row0; t0 < row1; t0 += CM_GATE_THREADS) {
        const int row = t0 + tid;
        float i = -INFINITY, f = 0.f;
        if (row < row1) {
            const float zi = a.z[(long long)row * a.z_ld + a.i_col + head] + bi, zf = a.z[(long long)row * a.z_ld + a.f_col + head] + bf;
            const float c = a.cap * tanhf(zf / a.cap);
            i = a.cap * tanhf(zi / a.cap);
            f = c < 0.f ? c - log1pf(expf(c)) : -log1pf(expf(-c));
        }
        float sum = f, top = i;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float ps = __shfl_up_sync(0xffffffffu, sum, o), pt = __shfl_up_sync(0xffffffffu, top, o);
            if (lane >= o) {
                top = fmaxf(sum + pt, top);
                sum += ps;
            }
        }
        if (lane == 31) {
            sum_s[warp] = sum;
            top_s[warp] = top;
        }
        __syncthreads();
        float ws = sum_s[lane], wt = top_s[lane];       // every warp scans the warps' totals for itself
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float ps = __shfl_up_sync(0xffffffffu, ws, o), pt = __shfl_up_sync(0xffffffffu, wt, o);
            if (lane >= o) {
                wt = fmaxf(ws + pt, wt);
                ws += ps;
            }
        }
        float m = m_s[0];
        ws = __shfl_sync(0xffffffffu, ws, (warp - 1) & 31);
        wt = __shfl_sync(0xffffffffu, wt, (warp - 1) & 31);
        if (warp > 0) m = fmaxf(ws + m, wt);
        m = fmaxf(sum + m, top);
        m_s[tid + 1] = m;
        __syncthreads();
        const float before = m_s[tid];
        if (row < row1) {
            const long long at = (long long)row * a.H + head;
            const float la = (f + before - m) * 1.4426950408889634f;
            w.gates[at] = la < CM_LEAST ? CM_LEAST : la;
            w.gates[plane + at] = expf(i - m);
            w.gates[2 * plane + at] = expf(-m);
        }
        __syncthreads();
        if (tid == 0) m_s[0] = m_s[min(CM_GATE_THREADS, row1 - t0)];
        __syncthreads();
    }
    if (tid == 0) *mg = m_s[0];
}

// A block per (chunk, head): the chunk's own share of the state after it, [DP][VP], and its decay.
template <int KIND, int DP, int VP>
__global__ void __launch_bounds__(CM_THREADS) chunk_states_kernel(SbChunkMem a, SbBatch batch, ChunkWork w, int vec) {
    constexpr int KLD = DP + 4, VLD = VP + 8;      // KLD: lanes (2 t, g) of a fragment meet every bank once
    constexpr int WM = DP >= 64 ? 4 : 2, WN = 8 / WM, MT = DP / 16 / WM, NT = VP / 8 / WN;
    extern __shared__ __align__(16) unsigned char cm_sm[];
    float* Kf = reinterpret_cast<float*>(cm_sm);                                     // [64][KLD]
    float* Af = Kf + CM_L * KLD;                                                     // [64][KLD] (not mlstm)
    __nv_bfloat16* Vs = reinterpret_cast<__nv_bfloat16*>(KIND == CM_MLSTM ? Af : Af + CM_L * KLD);   // [64][VLD]
    __shared__ alignas(16) float rest[4][DP], totals[4][DP];
    __shared__ GateSums gs;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int head = w.head0 + blockIdx.y;
    pdl_wait();
    int s, row, nt;
    if (!find_chunk(batch, blockIdx.x, s, row, nt)) return;
    load_rows<VP, VLD>(Vs, a.v, a.ld, row, nt, head, a.V, vec);
    cp_async_commit();
    load_wide<DP, KLD>(Kf, a.k, a.ld, row, nt, head, a.D, 1.f, vec);
    const long long cell = (long long)blockIdx.x * w.nh + blockIdx.y;
    if (KIND == CM_MLSTM) {
        if (warp == 0) gate_sums(w.gates, (long long)batch.n_rows * a.H, a.H, head, row, nt, gs);
        __syncthreads();
        if (tid < DP) {
            float n = 0.f;
#pragma unroll 8
            for (int i = 0; i < CM_L; ++i) n = fmaf(Kf[i * KLD + tid], gs.left[i], n);
            w.norm[cell * DP + tid] = n;
        }
        if (tid == 0) w.decay[cell * DP] = gs.total;
    } else {
        make_decays<KIND, DP, KLD>(Af, w.gates, a, row, nt, head, vec);
        __syncthreads();
        for (int e = tid; e < 4 * DP; e += CM_THREADS) {     // 16 tokens of a channel, from the last one back
            const int part = e / DP, d = e % DP;
            float p = 1.f;
#pragma unroll
            for (int i = 15; i >= 0; --i) {
                const int at = (part * 16 + i) * KLD + d;
                Kf[at] *= p;
                p *= Af[at];
            }
            totals[part][d] = p;
        }
        __syncthreads();
        if (tid < DP) {
            float p = 1.f;
#pragma unroll
            for (int part = 3; part >= 0; --part) {
                rest[part][tid] = p;
                p *= totals[part][tid];
            }
            w.decay[cell * DP + tid] = p;
        }
    }
    cp_async_wait<0>();
    __syncthreads();

    const int m0 = (warp % WM) * MT * 16, n0 = (warp / WM) * NT * 8;
    float S[MT][NT][4];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) S[mt][n][e] = 0.f;
    const __nv_bfloat16* vb = Vs + (lane & 15) * VLD + n0 + (lane >> 4) * 8;
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
        if (kk * 16 >= nt) break;
        unsigned int b[NT / 2][4];
#pragma unroll
        for (int i = 0; i < NT / 2; ++i) ldmatrix_x4_trans(b[i], vb + kk * 16 * VLD + i * 16);
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
            unsigned int ah[4], am[4], al[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int d = m0 + mt * 16 + g + (e & 1) * 8, tok = kk * 16 + 2 * t + (e >> 1) * 8;
                float x = Kf[tok * KLD + d], y = Kf[(tok + 1) * KLD + d];
                if (KIND == CM_MLSTM) {
                    x *= gs.left[tok];
                    y *= gs.left[tok + 1];
                } else {
                    x *= rest[kk][d];
                    y *= rest[kk][d];
                }
                split_three(x, y, ah[e], am[e], al[e]);
            }
#pragma unroll
            for (int i = 0; i < NT / 2; ++i) {
                mma_bf16(S[mt][2 * i], al, b[i][0], b[i][1]);
                mma_bf16(S[mt][2 * i + 1], al, b[i][2], b[i][3]);
                mma_bf16(S[mt][2 * i], am, b[i][0], b[i][1]);
                mma_bf16(S[mt][2 * i + 1], am, b[i][2], b[i][3]);
                mma_bf16(S[mt][2 * i], ah, b[i][0], b[i][1]);
                mma_bf16(S[mt][2 * i + 1], ah, b[i][2], b[i][3]);
            }
        }
    }
    float* dst = w.add + cell * DP * VP;
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int d = m0 + mt * 16 + g + half * 8, c = n0 + n * 8 + 2 * t;
                *reinterpret_cast<float2*>(dst + d * VP + c) = make_float2(S[mt][n][2 * half], S[mt][n][2 * half + 1]);
            }
}

// A thread per two neighbouring entries of a sequence's state (mlstm: and per entry of the normaliser): the chunks in order, eight
// of them fetched ahead of the chain.  Leaves the state at each chunk's start and brings the record up to date.
template <int KIND, int DP, int VP>
__global__ void __launch_bounds__(256) chunk_walk_kernel(SbChunkMem a, SbBatch batch, ChunkWork w) {
    const int s = blockIdx.x, head = w.head0 + blockIdx.y, at = blockIdx.z * 256 + threadIdx.x;
    pdl_wait();
    const int first = batch.cu_q[s], n = batch.cu_q[s + 1] - first, count = (n + CM_L - 1) / CM_L;
    if (n <= 0) return;
    float* rec = a.state + (long long)batch.seq_slot[s] * a.state_stride;
    if (KIND == CM_WKV && head == 0) {   // the last token's input: what the next step's first row blends with
        const __nv_bfloat16* last = (const __nv_bfloat16*)a.last + (long long)(first + n - 1) * a.last_width;
        for (int c = at; c < a.last_width; c += gridDim.z * 256) rec[a.last_offset + c] = __bfloat162float(last[c]);
    }
    const long long cell0 = ((long long)(first >> 6) + s) * w.nh + blockIdx.y;
    if (at >= DP * VP / 2) {
        const int d = at - DP * VP / 2;
        if (KIND != CM_MLSTM || d >= DP) return;
        float* ng = rec + (long long)a.H * a.D * a.V + (long long)head * a.D + d;
        float x = d < a.D ? *ng : 0.f;
        for (int c0 = 0; c0 < count; c0 += 8) {
            float add[8], keep[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const long long cell = cell0 + (long long)min(c0 + i, count - 1) * w.nh;
                add[i] = w.norm[cell * DP + d];
                keep[i] = w.decay[cell * DP];
            }
#pragma unroll
            for (int i = 0; i < 8; ++i)
                if (c0 + i < count) {
                    w.norm[(cell0 + (long long)(c0 + i) * w.nh) * DP + d] = x;
                    x = fmaf(keep[i], x, add[i]);
                }
        }
        if (d < a.D) *ng = x;
        return;
    }
    const int d = at / (VP / 2), c = (at % (VP / 2)) * 2;
    const bool in0 = d < a.D && c < a.V, in1 = d < a.D && c + 1 < a.V;
    float* Sg = rec + (long long)head * a.D * a.V + (long long)d * a.V + c;
    float x = in0 ? Sg[0] : 0.f, y = in1 ? Sg[1] : 0.f;
    for (int c0 = 0; c0 < count; c0 += 8) {
        float2 add[8];
        float keep[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const long long cell = cell0 + (long long)min(c0 + i, count - 1) * w.nh;
            add[i] = *reinterpret_cast<const float2*>(w.add + (cell * DP + d) * VP + c);
            keep[i] = w.decay[cell * DP + (KIND == CM_MLSTM ? 0 : d)];
        }
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (c0 + i < count) {
                unsigned int h, m, l;
                split_three(x, y, h, m, l);
                unsigned int* dst = reinterpret_cast<unsigned int*>(w.start + ((cell0 + (long long)(c0 + i) * w.nh) * 3 * DP + d) * VP + c);
                dst[0] = h;
                dst[DP * VP / 2] = m;
                dst[DP * VP] = l;
                x = fmaf(keep[i], x, add[i].x);
                y = fmaf(keep[i], y, add[i].y);
            }
    }
    if (in0) Sg[0] = x;
    if (in1) Sg[1] = y;
}

// Shared memory of chunk_outputs_kernel, in bytes.  Per-channel decays: Q, P, and one region that first holds the decays and the
// keys, then the values and the state at the chunk's start (value columns up to 64: three blocks per SM, else two); mlstm: the
// values, queries and keys in bfloat16, and the state.
template <int KIND, int DP, int VP> constexpr size_t outputs_smem() {
    constexpr size_t start = (size_t)3 * DP * (VP + 8) * 2, v = (size_t)CM_L * (VP + 8) * 2;
    if (KIND == CM_MLSTM) return (size_t)2 * CM_L * (DP + 8) * 2 + v + start;
    constexpr size_t wide = (size_t)CM_L * (DP + 8) * 4;
    return wide + (size_t)CM_P_FLOATS * 4 + (2 * wide > v + start ? 2 * wide : v + start);
}

// A block per (chunk, head): the outputs, the head's norm and the gate.  Warp: 16 tokens x half the value columns.
template <int KIND, int DP, int VP>
__global__ void __launch_bounds__(CM_THREADS, KIND != CM_MLSTM && outputs_smem<KIND, DP, VP>() <= 72 * 1024 ? 3 : (outputs_smem<KIND, DP, VP>() <= 111 * 1024 ? 2 : 1))
chunk_outputs_kernel(SbChunkMem a, SbBatch batch, ChunkWork w, int vec) {
    typedef __nv_bfloat16 bf;
    constexpr int FLD = DP + 8, VLD = VP + 8, NT = VP / 16;
    extern __shared__ __align__(16) unsigned char cm_sm[];
    float* Qf = reinterpret_cast<float*>(cm_sm);               // [64][FLD] queries, then queries times the decays of their 16 tokens
    float* P = Qf + CM_L * FLD;                                // blocks (0,0) (1,0) (1,1) (2,0) ..., [16][CM_PLD] each
    bf* Vs = KIND == CM_MLSTM ? reinterpret_cast<bf*>(cm_sm) : reinterpret_cast<bf*>(P + CM_P_FLOATS);   // [64][VLD]
    bf* Qb = Vs + CM_L * VLD;                                  // mlstm: [64][FLD] each
    bf* Kb = Qb + CM_L * FLD;
    bf* St = KIND == CM_MLSTM ? Kb + CM_L * FLD : Vs + CM_L * VLD;      // [3][DP][VLD]
    float* Kf = P + CM_P_FLOATS;                               // [64][FLD], where the values and the state come later
    float* Af = Kf + CM_L * FLD;                               // [64][FLD]
    __shared__ alignas(16) float totals[4][DP], grown[4][DP], us[DP], ns[DP], red[2][CM_L];
    __shared__ GateSums gs;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int head = w.head0 + blockIdx.y, wr = warp & 3, n0 = (warp >> 2) * (VP / 2);
    pdl_wait();
    int s, row, nt;
    if (!find_chunk(batch, blockIdx.x, s, row, nt)) return;
    const long long cell = (long long)blockIdx.x * w.nh + blockIdx.y;
    auto load_start = [&]() {
        const bf* src = w.start + cell * 3 * DP * VP;
        for (int e = tid; e < 3 * DP * VP / 8; e += CM_THREADS) cp_async_16(St + (e / (VP / 8)) * VLD + (e % (VP / 8)) * 8, src + e * 8);
    };
    float o[NT][4];
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[i][e] = 0.f;
    const int i0 = wr * 16 + g;               // this thread's tokens: i0 and i0 + 8
    float den0 = 1.f, den1 = 1.f;

    if (KIND == CM_MLSTM) {
        load_rows<VP, VLD>(Vs, a.v, a.ld, row, nt, head, a.V, vec);
        load_rows<DP, FLD>(Qb, a.q, a.ld, row, nt, head, a.D, vec);
        load_rows<DP, FLD>(Kb, a.k, a.ld, row, nt, head, a.D, vec);
        cp_async_commit();
        load_start();
        cp_async_commit();
        if (warp == 0) gate_sums(w.gates, (long long)batch.n_rows * a.H, a.H, head, row, nt, gs);
        if (tid >= CM_THREADS - DP) ns[tid - (CM_THREADS - DP)] = w.norm[cell * DP + tid - (CM_THREADS - DP)];
        cp_async_wait<0>();
        __syncthreads();
        float sc[8][4], q0 = 0.f, q1 = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) sc[i][e] = 0.f;
        const bf* qa = Qb + (wr * 16 + (lane & 15)) * FLD + (lane >> 4) * 8;
        const bf* kb = Kb + ((lane & 7) + (lane >> 4) * 8) * FLD + ((lane >> 3) & 1) * 8;
        const bf* sb = St + (lane & 15) * VLD + n0 + (lane >> 4) * 8;
#pragma unroll
        for (int k0 = 0; k0 < DP; k0 += 16) {
            unsigned int qf[4];
            ldmatrix_x4(qf, qa + k0);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float2 nn = *reinterpret_cast<const float2*>(ns + k0 + 2 * t + (e >> 1) * 8);
                float& acc = e & 1 ? q1 : q0;
                acc = fmaf(__uint_as_float(qf[e] << 16), nn.x, acc);
                acc = fmaf(__uint_as_float(qf[e] & 0xffff0000u), nn.y, acc);
            }
#pragma unroll
            for (int i = 0; i < 8; i += 2) {
                if (i <= 2 * wr) {            // keys after this warp's tokens are not seen
                    unsigned int b[4];
                    ldmatrix_x4(b, kb + i * 8 * FLD + k0);
                    mma_bf16(sc[i], qf, b[0], b[1]);
                    mma_bf16(sc[i + 1], qf, b[2], b[3]);
                }
            }
#pragma unroll
            for (int p = 2; p >= 0; --p)
#pragma unroll
                for (int i = 0; i < NT; i += 2) {
                    unsigned int b[4];
                    ldmatrix_x4_trans(b, sb + (p * DP + k0) * VLD + i * 8);
                    mma_bf16(o[i], qf, b[0], b[1]);
                    mma_bf16(o[i + 1], qf, b[2], b[3]);
                }
        }
        const float e0 = gs.grown[i0], e1 = gs.grown[i0 + 8];
        const float h0 = gs.hi[i0], h1 = gs.hi[i0 + 8], l0 = gs.lo[i0], l1 = gs.lo[i0 + 8];
#pragma unroll
        for (int i = 0; i < NT; ++i) {
            o[i][0] *= e0;
            o[i][1] *= e0;
            o[i][2] *= e1;
            o[i][3] *= e1;
        }
        q0 *= e0;
        q1 *= e1;
        const bf* vb = Vs + (lane & 15) * VLD + n0 + (lane >> 4) * 8;
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
            if (kk <= wr) {
                unsigned int ph[4], pm[4], pl[4];
#pragma unroll
                for (int part = 0; part < 2; ++part) {
                    const int i = 2 * kk + part, j = i * 8 + 2 * t;
                    const float2 hj = *reinterpret_cast<const float2*>(gs.hi + j), lj = *reinterpret_cast<const float2*>(gs.lo + j);
                    const float2 bj = *reinterpret_cast<const float2*>(gs.b + j);
                    const float p0 = j <= i0 ? sc[i][0] * exp2f((h0 - hj.x) + (l0 - lj.x)) * bj.x : 0.f;
                    const float p1 = j + 1 <= i0 ? sc[i][1] * exp2f((h0 - hj.y) + (l0 - lj.y)) * bj.y : 0.f;
                    const float p2 = j <= i0 + 8 ? sc[i][2] * exp2f((h1 - hj.x) + (l1 - lj.x)) * bj.x : 0.f;
                    const float p3 = j + 1 <= i0 + 8 ? sc[i][3] * exp2f((h1 - hj.y) + (l1 - lj.y)) * bj.y : 0.f;
                    q0 += p0 + p1;
                    q1 += p2 + p3;
                    split_three(p0, p1, ph[2 * part], pm[2 * part], pl[2 * part]);
                    split_three(p2, p3, ph[2 * part + 1], pm[2 * part + 1], pl[2 * part + 1]);
                }
#pragma unroll
                for (int i = 0; i < NT; i += 2) {
                    unsigned int b[4];
                    ldmatrix_x4_trans(b, vb + kk * 16 * VLD + i * 8);
                    mma_bf16(o[i], pl, b[0], b[1]);
                    mma_bf16(o[i + 1], pl, b[2], b[3]);
                    mma_bf16(o[i], pm, b[0], b[1]);
                    mma_bf16(o[i + 1], pm, b[2], b[3]);
                    mma_bf16(o[i], ph, b[0], b[1]);
                    mma_bf16(o[i + 1], ph, b[2], b[3]);
                }
            }
        }
        q0 += __shfl_xor_sync(0xffffffffu, q0, 1);
        q0 += __shfl_xor_sync(0xffffffffu, q0, 2);
        q1 += __shfl_xor_sync(0xffffffffu, q1, 1);
        q1 += __shfl_xor_sync(0xffffffffu, q1, 2);
        den0 = fmaxf(fabsf(q0 * a.q_scale), gs.em[i0]) + 1e-6f;
        den1 = fmaxf(fabsf(q1 * a.q_scale), gs.em[i0 + 8]) + 1e-6f;
#pragma unroll
        for (int i = 0; i < NT; ++i) {
            o[i][0] = o[i][0] * a.q_scale / den0;
            o[i][1] = o[i][1] * a.q_scale / den0;
            o[i][2] = o[i][2] * a.q_scale / den1;
            o[i][3] = o[i][3] * a.q_scale / den1;
        }
    } else {
        load_kept_decays<DP, FLD>(Af, w.gates, a, row, nt, head, vec);
        cp_async_commit();
        if (KIND == CM_WKV && tid < DP) us[tid] = tid < a.D ? a.bias2[(long long)head * a.D + tid] : 0.f;
        load_wide<DP, FLD>(Qf, a.q, a.ld, row, nt, head, a.D, KIND == CM_GLA ? a.q_scale : 1.f, vec);
        load_wide<DP, FLD>(Kf, a.k, a.ld, row, nt, head, a.D, 1.f, vec);
        cp_async_wait<0>();
        __syncthreads();
        {   // P inside 16 tokens: four lanes per key j carry k_j times the decays since, token after token
            const int blk = warp >> 1, jj = (warp & 1) * 8 + (lane >> 2), j = blk * 16 + jj;
            float* Pd = P + (blk * (blk + 3) / 2 * 16) * CM_PLD + jj;      // block (blk, blk), column j
            float4 cur[DP / 16];
#pragma unroll
            for (int e = 0; e < DP / 16; ++e) cur[e] = *reinterpret_cast<const float4*>(Kf + j * FLD + e * 16 + t * 4);
            if ((warp & 1) && t == 0)
#pragma unroll
                for (int i = 0; i < 8; ++i) Pd[i * CM_PLD] = 0.f;
            if (blk * 16 < nt) {
#pragma unroll 2
                for (int ii = (warp & 1) * 8; ii < 16; ++ii) {
                    const float* qi = Qf + (blk * 16 + ii) * FLD + t * 4;
                    const float* ai = Af + (blk * 16 + ii) * FLD + t * 4;
                    float2 acc = make_float2(0.f, 0.f), acc2 = acc;
#pragma unroll
                    for (int e = 0; e < DP / 16; ++e) {
                        const float4 q4 = *reinterpret_cast<const float4*>(qi + e * 16);
                        float4 x = cur[e];
                        if (KIND == CM_GLA) {
                            if (ii > jj) {
                                const float4 a4 = *reinterpret_cast<const float4*>(ai + e * 16);
                                x = make_float4(x.x * a4.x, x.y * a4.y, x.z * a4.z, x.w * a4.w);
                                cur[e] = x;
                            }
                        } else {
                            if (ii == jj) {
                                const float4 u4 = *reinterpret_cast<const float4*>(us + e * 16 + t * 4);
                                x = make_float4(x.x * u4.x, x.y * u4.y, x.z * u4.z, x.w * u4.w);
                            } else if (ii > jj) {
                                const float4 a4 = *reinterpret_cast<const float4*>(ai + e * 16);
                                cur[e] = make_float4(x.x * a4.x, x.y * a4.y, x.z * a4.z, x.w * a4.w);
                            }
                        }
                        acc = fma_pair(make_float2(q4.x, q4.y), make_float2(x.x, x.y), acc);
                        acc2 = fma_pair(make_float2(q4.z, q4.w), make_float2(x.z, x.w), acc2);
                    }
                    float p = (acc.x + acc.y) + (acc2.x + acc2.y);
                    p += __shfl_xor_sync(0xffffffffu, p, 1);
                    p += __shfl_xor_sync(0xffffffffu, p, 2);
                    if (t == 0) Pd[ii * CM_PLD] = ii >= jj ? p : 0.f;
                }
            }
        }
        __syncthreads();
        for (int e = tid; e < 4 * DP; e += CM_THREADS) {     // q times the decays since its 16 tokens began, k times those until they end
            const int part = e / DP, d = e % DP;
            float p = 1.f;
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const int at = (part * 16 + i) * FLD + d;
                if (KIND == CM_GLA) p *= Af[at];
                Qf[at] *= p;
                if (KIND == CM_WKV) p *= Af[at];
            }
            totals[part][d] = p;
            p = 1.f;
#pragma unroll
            for (int i = 15; i >= 0; --i) {
                const int at = (part * 16 + i) * FLD + d;
                Kf[at] *= p;
                p *= Af[at];
            }
        }
        __syncthreads();
        if (tid < DP) {
            float p = 1.f;
#pragma unroll
            for (int part = 0; part < 4; ++part) {
                grown[part][tid] = p;
                p *= totals[part][tid];
            }
        }
        if (warp < 6) {   // P between groups of 16 tokens: (1,0) (2,1) (3,2) (2,0) (3,1) (3,0)
            const int qi = warp < 3 ? warp + 1 : (warp == 3 ? 2 : 3), kj = warp < 3 ? warp : (warp == 4 ? 1 : 0);
            if (qi * 16 < nt) {
                float c[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll 2
                for (int k0 = 0; k0 < DP; k0 += 16) {
                    unsigned int ah[4], am[4], al[4], bh[4], bm[4], bl[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int col = k0 + 2 * t + (e >> 1) * 8;
                        float2 x = *reinterpret_cast<const float2*>(Qf + (qi * 16 + g + (e & 1) * 8) * FLD + col);
                        for (int between = kj + 1; between < qi; ++between) {
                            const float2 f = *reinterpret_cast<const float2*>(&totals[between][col]);
                            x.x *= f.x;
                            x.y *= f.y;
                        }
                        split_three(x.x, x.y, ah[e], am[e], al[e]);
                    }
#pragma unroll
                    for (int e = 0; e < 4; ++e) {   // two groups of 8 keys, two halves of 16 channels
                        const float2 x = *reinterpret_cast<const float2*>(Kf + (kj * 16 + (e >> 1) * 8 + g) * FLD + k0 + 2 * t + (e & 1) * 8);
                        split_three(x.x, x.y, bh[e], bm[e], bl[e]);
                    }
#pragma unroll
                    for (int n = 0; n < 2; ++n) {
                        mma_bf16(c[n], ah, bl[2 * n], bl[2 * n + 1]);
                        mma_bf16(c[n], al, bh[2 * n], bh[2 * n + 1]);
                        mma_bf16(c[n], am, bm[2 * n], bm[2 * n + 1]);
                        mma_bf16(c[n], ah, bm[2 * n], bm[2 * n + 1]);
                        mma_bf16(c[n], am, bh[2 * n], bh[2 * n + 1]);
                        mma_bf16(c[n], ah, bh[2 * n], bh[2 * n + 1]);
                    }
                }
#pragma unroll
                for (int n = 0; n < 2; ++n)
#pragma unroll
                    for (int half = 0; half < 2; ++half)
                        *reinterpret_cast<float2*>(P + ((qi * (qi + 1) / 2 + kj) * 16 + g + half * 8) * CM_PLD + n * 8 + 2 * t) =
                            make_float2(c[n][2 * half], c[n][2 * half + 1]);
            }
        }
        __syncthreads();                      // keys and decays are done with: the values and the state take their place
        load_rows<VP, VLD>(Vs, a.v, a.ld, row, nt, head, a.V, vec);
        cp_async_commit();
        load_start();
        cp_async_commit();
        cp_async_wait<1>();                   // the values are there (for this thread; the barrier makes it everybody's)
        __syncthreads();
        const bf* vb = Vs + (lane & 15) * VLD + n0 + (lane >> 4) * 8;
        if (wr * 16 < nt) {
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
                if (kk <= wr) {
                    unsigned int ph[4], pm[4], pl[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float2 x = *reinterpret_cast<const float2*>(P + ((wr * (wr + 1) / 2 + kk) * 16 + g + (e & 1) * 8) * CM_PLD + 2 * t + (e >> 1) * 8);
                        split_three(x.x, x.y, ph[e], pm[e], pl[e]);
                    }
#pragma unroll
                    for (int i = 0; i < NT; i += 2) {
                        unsigned int b[4];
                        ldmatrix_x4_trans(b, vb + kk * 16 * VLD + i * 8);
                        mma_bf16(o[i], pl, b[0], b[1]);
                        mma_bf16(o[i + 1], pl, b[2], b[3]);
                        mma_bf16(o[i], pm, b[0], b[1]);
                        mma_bf16(o[i + 1], pm, b[2], b[3]);
                        mma_bf16(o[i], ph, b[0], b[1]);
                        mma_bf16(o[i + 1], ph, b[2], b[3]);
                    }
                }
            }
        }
        cp_async_wait<0>();
        __syncthreads();
        const bf* sb = St + (lane & 15) * VLD + n0 + (lane >> 4) * 8;
        if (wr * 16 < nt) {
#pragma unroll 2
            for (int k0 = 0; k0 < DP; k0 += 16) {
                unsigned int qh[4], qm[4], ql[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int col = k0 + 2 * t + (e >> 1) * 8;
                    const float2 x = *reinterpret_cast<const float2*>(Qf + (i0 + (e & 1) * 8) * FLD + col);
                    const float2 f = *reinterpret_cast<const float2*>(&grown[wr][col]);
                    split_three(x.x * f.x, x.y * f.y, qh[e], qm[e], ql[e]);
                }
#pragma unroll
                for (int i = 0; i < NT; i += 2) {
                    unsigned int bh[4], bm[4], bl[4];
                    ldmatrix_x4_trans(bl, sb + (2 * DP + k0) * VLD + i * 8);
                    ldmatrix_x4_trans(bm, sb + (DP + k0) * VLD + i * 8);
                    ldmatrix_x4_trans(bh, sb + k0 * VLD + i * 8);
                    mma_bf16(o[i], qh, bl[0], bl[1]);
                    mma_bf16(o[i + 1], qh, bl[2], bl[3]);
                    mma_bf16(o[i], ql, bh[0], bh[1]);
                    mma_bf16(o[i + 1], ql, bh[2], bh[3]);
                    mma_bf16(o[i], qm, bm[0], bm[1]);
                    mma_bf16(o[i + 1], qm, bm[2], bm[3]);
                    mma_bf16(o[i], qh, bm[0], bm[1]);
                    mma_bf16(o[i + 1], qh, bm[2], bm[3]);
                    mma_bf16(o[i], qm, bh[0], bh[1]);
                    mma_bf16(o[i + 1], qm, bh[2], bh[3]);
                    mma_bf16(o[i], qh, bh[0], bh[1]);
                    mma_bf16(o[i + 1], qh, bh[2], bh[3]);
                }
            }
        }
    }

    // the head's root mean square over its value columns, the norm's weight and the gate
    float ss0 = 0.f, ss1 = 0.f;
#pragma unroll
    for (int i = 0; i < NT; ++i) {
        ss0 = fmaf(o[i][0], o[i][0], fmaf(o[i][1], o[i][1], ss0));
        ss1 = fmaf(o[i][2], o[i][2], fmaf(o[i][3], o[i][3], ss1));
    }
    ss0 += __shfl_xor_sync(0xffffffffu, ss0, 1);
    ss0 += __shfl_xor_sync(0xffffffffu, ss0, 2);
    ss1 += __shfl_xor_sync(0xffffffffu, ss1, 1);
    ss1 += __shfl_xor_sync(0xffffffffu, ss1, 2);
    if (t == 0) {
        red[warp >> 2][i0] = ss0;
        red[warp >> 2][i0 + 8] = ss1;
    }
    __syncthreads();
    const float* nw = a.norm + (long long)head * a.norm_stride;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const int i = i0 + half * 8;
        if (i >= nt) continue;
        const float mul = (KIND == CM_MLSTM ? a.out_scale : 1.f) / sqrtf((red[0][i] + red[1][i]) / (float)a.V + a.eps);
        const bf* gr = (const bf*)a.g + (long long)(row + i) * a.ld + (long long)head * a.V;
        bf* yr = (bf*)a.y + (long long)(row + i) * a.y_ld + (long long)head * a.V;
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            const int c = n0 + n * 8 + 2 * t;
            float2 gv = make_float2(0.f, 0.f);
            if (vec && c < a.V) gv = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(gr + c));
            else {
                if (c < a.V) gv.x = __bfloat162float(gr[c]);
                if (c + 1 < a.V) gv.y = __bfloat162float(gr[c + 1]);
            }
            float gx = 1.0f / (1.0f + expf(-gv.x)), gy = 1.0f / (1.0f + expf(-gv.y));
            if (KIND != CM_MLSTM) {
                gx *= gv.x;
                gy *= gv.y;
            }
            if (vec && c < a.V) {
                const float2 nn = make_float2(nw[c], nw[c + 1]);
                *reinterpret_cast<__nv_bfloat162*>(yr + c) =
                    __floats2bfloat162_rn(o[n][2 * half] * mul * nn.x * gx, o[n][2 * half + 1] * mul * nn.y * gy);
            } else {
                if (c < a.V) yr[c] = __float2bfloat16_rn(o[n][2 * half] * mul * nw[c] * gx);
                if (c + 1 < a.V) yr[c + 1] = __float2bfloat16_rn(o[n][2 * half + 1] * mul * nw[c + 1] * gy);
            }
        }
    }
}

static int cm_key_pad(int D) { return D <= 32 ? 32 : (D <= 64 ? 64 : 128); }
static int cm_value_pad(int V) { return V <= 64 ? 64 : 128; }
static long long cm_head_floats(long long cells, int D, int V) {
    const long long dp = cm_key_pad(D), vp = cm_value_pad(V);
    return cells * (dp * vp + 3 * dp * vp / 2 + 2 * dp);
}

static long long cm_gate_floats(int kind, long long rows, int H, int D) { return (rows * H * (kind == CM_MLSTM ? 3 : D) + 3) / 4 * 4; }

// Heads that are worked on together: as many as keep their share of the workspace, states and normalisers, within head_floats (at
// least one).  The gates or decays of all rows and heads, cm_gate_floats, come on top.
static int cm_heads(long long head_floats, long long cells, int H, int D, int V) {
    const long long fit = head_floats / cm_head_floats(cells, D, V);
    return fit < 1 ? 1 : (fit < H ? (int)fit : H);
}

template <int KIND, int DP, int VP>
static int launch_chunk_memory(SbChunkMem a, SbBatch batch, int vec, cudaStream_t stream) {
    const long long cells = batch.n_rows / CM_L + batch.n_seqs;
    const int per = cm_heads(a.head_floats, cells, a.H, a.D, a.V);
    constexpr size_t states_smem = (size_t)CM_L * (DP + 4) * 4 * (KIND == CM_MLSTM ? 1 : 2) + (size_t)CM_L * (VP + 8) * 2;
    constexpr size_t out_smem = outputs_smem<KIND, DP, VP>();
    cudaError_t err = cudaFuncSetAttribute(chunk_states_kernel<KIND, DP, VP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)states_smem);
    if (err == cudaSuccess)
        err = cudaFuncSetAttribute(chunk_outputs_kernel<KIND, DP, VP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)out_smem);
    if (err != cudaSuccess) return (int)err;
    ChunkWork w;
    w.gates = a.work;
    w.add = a.work + cm_gate_floats(KIND, batch.n_rows, a.H, a.D);
    w.start = reinterpret_cast<__nv_bfloat16*>(w.add + cells * per * DP * VP);
    w.decay = reinterpret_cast<float*>(w.start + cells * per * 3 * DP * VP);
    w.norm = w.decay + cells * per * DP;
    const int walk = (DP * VP / 2 + (KIND == CM_MLSTM ? DP : 0) + 255) / 256;
    for (int h = 0; h < a.H; h += per) {
        w.head0 = h;
        w.nh = a.H - h < per ? a.H - h : per;
        const dim3 grid((unsigned int)cells, w.nh);
        if (KIND == CM_MLSTM) sb_launch(chunk_gates_kernel, dim3(batch.n_seqs, w.nh), CM_GATE_THREADS, 0, stream, a, batch, w);
        sb_launch(chunk_states_kernel<KIND, DP, VP>, grid, CM_THREADS, states_smem, stream, a, batch, w, vec);
        sb_launch(chunk_walk_kernel<KIND, DP, VP>, dim3(batch.n_seqs, w.nh, walk), 256, 0, stream, a, batch, w);
        sb_launch(chunk_outputs_kernel<KIND, DP, VP>, grid, CM_THREADS, out_smem, stream, a, batch, w, vec);
        err = cudaGetLastError();
        if (err != cudaSuccess) return (int)err;
    }
    return 0;
}

extern "C" {

// Floats of workspace for a step of n_rows rows of n_seqs sequences whose heads may take head_floats of them together, or -1 for heads
// that these kernels do not take.
long long sb_chunk_memory_floats(int kind, int n_rows, int n_seqs, int H, int D, int V, long long head_floats) {
    if (n_rows < 1 || n_seqs < 1 || H < 1 || H > 65535 || D < 1 || V < 1 || D > 128 || V > 128 || (kind == CM_WKV && D != V)) return -1;
    const long long cells = n_rows / CM_L + n_seqs;
    return cm_gate_floats(kind, n_rows, H, D) + cm_heads(head_floats, cells, H, D, V) * cm_head_floats(cells, D, V);
}

// Kernels that such a step launches.
int sb_chunk_memory_launches(int kind, int n_rows, int n_seqs, int H, int D, int V, long long head_floats) {
    const int per = cm_heads(head_floats, n_rows / CM_L + n_seqs, H, D, V);
    return (H + per - 1) / per * (kind == CM_MLSTM ? 4 : 3);   // the gates, the chunks' shares, the walk over them, the outputs
}

int sb_chunk_memory(int kind, SbChunkMem a, SbBatch batch, cudaStream_t stream) {
    if (batch.n_seqs <= 0 || batch.n_rows <= 0) return 0;
    if (sb_chunk_memory_floats(kind, batch.n_rows, batch.n_seqs, a.H, a.D, a.V, a.head_floats) < 0 || a.work == nullptr
        || (kind == CM_GLA && !(a.inv_tau > 0.f)) || (kind == CM_MLSTM && !(a.cap > 0.f)))
        return (int)cudaErrorInvalidValue;
    const auto aligned = [](const void* p, size_t n) { return (reinterpret_cast<size_t>(p) & (n - 1)) == 0; };
    const int vec = a.D % 8 == 0 && a.V % 8 == 0 && a.ld % 8 == 0 && a.y_ld % 2 == 0 && aligned(a.q, 16) && aligned(a.k, 16) && aligned(a.v, 16)
                    && aligned(a.g, 4) && aligned(a.y, 4) && (kind == CM_MLSTM || aligned(a.z, 16));
    const int dp = cm_key_pad(a.D), vp = cm_value_pad(a.V);
#define SB_CM(KIND, DP, VP) if (kind == KIND && dp == DP && vp == VP) return launch_chunk_memory<KIND, DP, VP>(a, batch, vec, stream)
    SB_CM(CM_WKV, 32, 64);
    SB_CM(CM_WKV, 64, 64);
    SB_CM(CM_WKV, 128, 128);
    SB_CM(CM_GLA, 32, 64);
    SB_CM(CM_GLA, 64, 64);
    SB_CM(CM_GLA, 128, 64);
    SB_CM(CM_GLA, 32, 128);
    SB_CM(CM_GLA, 64, 128);
    SB_CM(CM_GLA, 128, 128);
    SB_CM(CM_MLSTM, 32, 64);
    SB_CM(CM_MLSTM, 64, 64);
    SB_CM(CM_MLSTM, 128, 64);
    SB_CM(CM_MLSTM, 32, 128);
    SB_CM(CM_MLSTM, 64, 128);
    SB_CM(CM_MLSTM, 128, 128);
#undef SB_CM
    return (int)cudaErrorInvalidValue;
}

}  // extern "C"
