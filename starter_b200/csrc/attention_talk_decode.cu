// Decoding with scores that meet across heads (attention_talk.cu says what is computed), on the tensor cores: bfloat16 queries
// and cache, key and value widths of 64 or 128, up to 5 query heads per key/value head and up to 16 key/value heads.
//
// A block takes a row and a share of its key pages; warp c owns key/value head c with its query heads.  Per page of 64 keys:
//   scores   S[16 keys x 8 heads] by mma.sync with the keys as the left operand, straight from the cache into registers: a
//            lane reads 16 bytes of a key row, and the columns stand in the product in the order in which the lanes hold them
//            (the queries' registers in the same order)
//   mixing   all heads' capped scores meet in shared memory, a thread per key and some heads, 32-bit
//   softmax  a warp per its own heads, 32-bit
//   values   O[16 x V] by mma.sync with the values as the right operand; a weight is three bfloat16 numbers (8 + 8 + 8
//            bits: the 32-bit weight itself) that stand as three rows of the left operand, so that the exact product
//            costs no more than the rounded one would (up to 5 heads fill 15 of its 16 rows)
// Masked keys of a page weigh nothing and their values are not read, so what lies in a page's free rows does not matter.
//
// What bounds it: the cache's bytes.  The block-per-row kernel spent its time on a turn of 32 keys at a time, each a read of
// the keys, two barriers and a read of the values one after another, with lanes that each walked a key row of their own (a
// line per lane and load).  Measured on a B200, 16 heads on 8 of 128, 2,049 keys a row, us a layer with the merge: 8 rows 74 -> 30 (67
// MB: 10 us at the copy bandwidth); the whole step of six layers at 1 / 8 / 32 rows: 798 -> 500, 920 -> 697, 2,249 -> 1,248.
#include "attention_flex.cuh"
#include "mma_utils.cuh"

#define TD_KEYS SB_PAGE
#define TD_LD (TD_KEYS + 4)

__device__ __forceinline__ uint4 td_load(const __nv_bfloat16* p) { return *reinterpret_cast<const uint4*>(p); }

// One of the three bfloat16 numbers that make up x.
__device__ __forceinline__ float td_piece(float x, int piece) {
    const float h = __bfloat162float(__float2bfloat16_rn(x));
    if (piece == 0) return h;
    x -= h;
    const float m = __bfloat162float(__float2bfloat16_rn(x));
    return piece == 1 ? m : x - m;
}

template <int D, int V>
__global__ void __launch_bounds__(512) talking_decode_kernel(SbFlex p, SbBatch batch, __nv_bfloat16* __restrict__ out, int n_splits,
                                                             float* __restrict__ partial) {
    typedef __nv_bfloat16 bf;
    constexpr int KJ = D / 32, NT = V / 8;
    extern __shared__ __align__(16) float td_sm[];
    const int H = p.n_heads, G = p.n_kv_heads, per = H / G;
    float* tb = td_sm;                       // [H][H]
    float* raw = tb + (H * H + 3) / 4 * 4;   // [H][TD_LD] capped scores
    float* mix = raw + H * TD_LD;            // [H][TD_LD] mixed scores, then weights
    float* sums = mix + H * TD_LD;           // [G][3 per][V]
    const int row = blockIdx.x, tid = threadIdx.x, lane = tid & 31, c = tid >> 5, g = lane >> 2, t = lane & 3;
    const int threads = blockDim.x;
    if (p.talk != nullptr)                   // weights: they do not depend on the kernel before
        for (int e = tid; e < H * H; e += threads) tb[e] = p.talk[e];
    pdl_wait();
    int slot, pos;
    row_place(batch, row, slot, pos);
    const int lo = p.window > 0 ? max(0, pos - p.window + 1) : 0, kept_end = min(p.keep_first, lo);
    const int first_page = lo / TD_KEYS, kept_pages = min((kept_end + TD_KEYS - 1) / TD_KEYS, first_page);
    const int pages = kept_pages + pos / TD_KEYS - first_page + 1;
    const int share = (pages + n_splits - 1) / n_splits, page_lo = blockIdx.y * share, page_hi = min(pages, page_lo + share);

    unsigned int qf[KJ][4];
    {
        const bf* qr = (const bf*)p.q + (long long)row * p.q_row + (long long)(c * per + min(g, per - 1)) * p.q_head;
#pragma unroll
        for (int j = 0; j < KJ; ++j) {
            const uint4 x = g < per ? td_load(qr + j * 32 + t * 8) : make_uint4(0, 0, 0, 0);
            qf[j][0] = x.x, qf[j][1] = x.y, qf[j][2] = x.z, qf[j][3] = x.w;
        }
    }
    float o[NT][4];
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[i][e] = 0.f;
    float run_m = -INFINITY, run_l = 0.f;    // lane j: of the warp's head j

    // A block to itself on an SM waits for every read: it asks for its page ahead (one sequence of 2,049 keys, the whole step: 530 ->
    // 500 us); where blocks hide one another's reads the extra requests cost (8 sequences: 24.4 -> 27.7 us a layer).
    const bool few = gridDim.x * gridDim.y <= 74;
    for (int pg = page_lo; pg < page_hi; ++pg) {
        const int lp = pg < kept_pages ? pg : first_page + pg - kept_pages, n0 = lp * TD_KEYS;
        const long long tok = flex_token(p, slot, n0, c);
        if (tok < 0) continue;               // a page that the slot does not have: the same for every head
        const auto seen = [&](int i) { return n0 + i <= pos && (n0 + i >= lo || n0 + i < kept_end); };
        if (few && lane == 0) {              // the visible rows of the page are asked for in one go
            const int from = lp < kept_pages ? 0 : max(0, lo - n0), to = min(TD_KEYS, (lp < kept_pages && n0 + TD_KEYS <= lo ? kept_end : pos + 1) - n0);
            l2_prefetch((const bf*)p.k + (tok + from) * D, (to - from) * D * 2);
            l2_prefetch((const bf*)p.v + (tok + from) * p.v_row, (to - from) * p.v_row * 2);
        }
        const bf* kp = (const bf*)p.k + tok * D + g * D + t * 8;
        const bf* vp = (const bf*)p.v + tok * p.v_row + g * 8;
#pragma unroll 1
        for (int k16 = 0; k16 < TD_KEYS / 16; ++k16) {
            uint4 ka[KJ], kb[KJ];
#pragma unroll
            for (int j = 0; j < KJ; ++j) {
                ka[j] = td_load(kp + (k16 * 16) * D + j * 32);
                kb[j] = td_load(kp + (k16 * 16 + 8) * D + j * 32);
            }
            float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int j = 0; j < KJ; ++j) {
                const unsigned int a0[4] = {ka[j].x, kb[j].x, ka[j].y, kb[j].y}, a1[4] = {ka[j].z, kb[j].z, ka[j].w, kb[j].w};
                mma_bf16(s, a0, qf[j][0], qf[j][1]);
                mma_bf16(s, a1, qf[j][2], qf[j][3]);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (2 * t + (e & 1) < per) raw[(c * per + 2 * t + (e & 1)) * TD_LD + k16 * 16 + g + (e >> 1) * 8] = s[e];
        }
        __syncwarp();
        for (int e = lane; e < per * TD_KEYS; e += 32) {   // the warp's scores, dealt out evenly
            float* r = raw + (c * per + e / TD_KEYS) * TD_LD + e % TD_KEYS;
            float s = *r * p.scale;
            if (p.softcap > 0.f) s = p.softcap * tanhf(s / p.softcap);
            *r = seen(e % TD_KEYS) ? s : 0.f;
        }
        __syncthreads();
        const float* scores = raw;
        if (p.talk != nullptr) {
            const int key = tid % TD_KEYS, group = tid / TD_KEYS, groups = threads >= TD_KEYS ? threads / TD_KEYS : 1;
            if (group < groups)
                for (int k2 = key; k2 < TD_KEYS; k2 += threads >= TD_KEYS ? TD_KEYS : threads)
                    for (int h0 = group; h0 < H; h0 += 4 * groups) {
                        float x[4] = {0.f, 0.f, 0.f, 0.f};
                        for (int i = 0; i < H; ++i) {
                            const float s = raw[i * TD_LD + k2];
#pragma unroll
                            for (int j = 0; j < 4; ++j)
                                if (h0 + j * groups < H) x[j] = fmaf(tb[(h0 + j * groups) * H + i], s, x[j]);
                        }
#pragma unroll
                        for (int j = 0; j < 4; ++j)
                            if (h0 + j * groups < H) mix[(h0 + j * groups) * TD_LD + k2] = x[j];
                    }
            scores = mix;
        }
        __syncthreads();
        float alpha = 1.f;                   // lane j: of the warp's head j
        for (int j = 0; j < per; ++j) {
            const int at = (c * per + j) * TD_LD + 2 * lane;
            const float2 x = *reinterpret_cast<const float2*>(scores + at);
            const bool s0 = seen(2 * lane), s1 = seen(2 * lane + 1);
            const float m_old = __shfl_sync(0xffffffffu, run_m, j);
            const float m_new = fmaxf(m_old, warp_max(fmaxf(s0 ? x.x : -INFINITY, s1 ? x.y : -INFINITY)));
            const bool any = m_new != -INFINITY;
            const float w0 = s0 && any ? expf(x.x - m_new) : 0.f, w1 = s1 && any ? expf(x.y - m_new) : 0.f;
            const float sum = warp_sum(w0 + w1);
            if (lane == j && any) {
                alpha = expf(m_old - m_new);
                run_m = m_new;
                run_l = run_l * alpha + sum;
            }
            *reinterpret_cast<float2*>(mix + at) = make_float2(w0, w1);
        }
        __syncwarp();
        const int j0 = g % per, j1 = (g + 8) % per, piece0 = g / per, piece1 = (g + 8) / per;   // rows g and g + 8 of the left operand
        const float al0 = __shfl_sync(0xffffffffu, alpha, j0), al1 = __shfl_sync(0xffffffffu, alpha, j1);
        if (pg > page_lo) {
#pragma unroll
            for (int i = 0; i < NT; ++i) {
                o[i][0] *= al0;
                o[i][1] *= al0;
                o[i][2] *= al1;
                o[i][3] *= al1;
            }
        }
#pragma unroll 1
        for (int k16 = 0; k16 < TD_KEYS / 16; ++k16) {
            unsigned int a[4] = {0u, 0u, 0u, 0u};
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int i = k16 * 16 + 2 * t + half * 8;
                if (piece0 < 3) {
                    const float2 w = *reinterpret_cast<const float2*>(mix + (c * per + j0) * TD_LD + i);
                    a[2 * half] = pack_bf16(td_piece(w.x, piece0), td_piece(w.y, piece0));
                }
                if (piece1 < 3) {
                    const float2 w = *reinterpret_cast<const float2*>(mix + (c * per + j1) * TD_LD + i);
                    a[2 * half + 1] = pack_bf16(td_piece(w.x, piece1), td_piece(w.y, piece1));
                }
            }
#pragma unroll
            for (int vb = 0; vb < V / 64; ++vb) {
                uint4 r[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int i = k16 * 16 + 2 * t + (e & 1) + (e >> 1) * 8;
                    r[e] = seen(i) ? td_load(vp + (long long)i * p.v_row + vb * 64) : make_uint4(0, 0, 0, 0);
                }
                const unsigned int lo0[4] = {r[0].x, r[0].y, r[0].z, r[0].w}, lo1[4] = {r[1].x, r[1].y, r[1].z, r[1].w};
                const unsigned int hi0[4] = {r[2].x, r[2].y, r[2].z, r[2].w}, hi1[4] = {r[3].x, r[3].y, r[3].z, r[3].w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {   // columns g * 8 + 2 i and + 1 of this half of the row
                    mma_bf16(o[vb * 8 + 2 * i], a, __byte_perm(lo0[i], lo1[i], 0x5410), __byte_perm(hi0[i], hi1[i], 0x5410));
                    mma_bf16(o[vb * 8 + 2 * i + 1], a, __byte_perm(lo0[i], lo1[i], 0x7632), __byte_perm(hi0[i], hi1[i], 0x7632));
                }
            }
        }
    }

    float* mine = sums + (size_t)c * 3 * per * V;
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int r = g + (e >> 1) * 8;
            if (r < 3 * per) mine[r * V + (i / 8) * 64 + (2 * t + (e & 1)) * 8 + i % 8] = o[i][e];
        }
    __syncwarp();
    for (int j = 0; j < per; ++j) {
        const int h = c * per + j;
        const float m = __shfl_sync(0xffffffffu, run_m, j);
        float l = __shfl_sync(0xffffffffu, run_l, j);
        if (n_splits > 1) {
            float* dst = partial + (((long long)row * H + h) * n_splits + blockIdx.y) * (V + 2);
            for (int d = lane; d < V; d += 32) dst[d] = (mine[(2 * per + j) * V + d] + mine[(per + j) * V + d]) + mine[j * V + d];
            if (lane == 0) {
                dst[V] = m;
                dst[V + 1] = l;
            }
        } else {
            float scale = 1.f;
            if (p.sink != nullptr) {   // one more term in the denominator, no value behind it
                const float sk = p.sink[h], m_new = fmaxf(m, sk);
                scale = expf(m - m_new);
                l = l * scale + expf(sk - m_new);
            }
            const float inv = scale / l;
            bf* orow = out + ((long long)row * H + h) * V;
            for (int d = lane; d < V; d += 32)
                orow[d] = __float2bfloat16_rn(((mine[(2 * per + j) * V + d] + mine[(per + j) * V + d]) + mine[j * V + d]) * inv);
        }
    }
}

void sb_talking_merge_bf16(const float* partial, void* out, const float* sink, int n_rows, int n_heads, int n_splits, int v_dim,
                           cudaStream_t stream);   // attention_talk.cu

extern "C" {

// Bytes of shared memory of a block, or -1 for sizes that this kernel does not take.
long long sb_talking_decode_smem(int n_heads, int n_kv_heads, int k_dim, int v_dim) {
    if (n_heads < 1 || n_kv_heads < 1 || n_heads % n_kv_heads || n_kv_heads > 16 || n_heads / n_kv_heads > 5 || (k_dim != 64 && k_dim != 128)
        || (v_dim != 64 && v_dim != 128))
        return -1;
    return ((long long)(n_heads * n_heads + 3) / 4 * 4 + 2ll * n_heads * TD_LD + 3ll * n_heads * v_dim) * 4;
}

int sb_talking_decode(SbFlex p, SbBatch batch, void* out, int n_splits, float* partial, cudaStream_t stream) {
    if (batch.n_rows <= 0) return 0;
    const long long smem = sb_talking_decode_smem(p.n_heads, p.n_kv_heads, p.k_dim, p.v_dim);
    if (smem < 0 || smem > 227 * 1024 || n_splits < 1 || n_splits > 64 || (n_splits > 1 && partial == nullptr) || p.q_row % 8 || p.q_head % 8
        || p.v_row % 8 || (p.v_heads > 0 && p.v_heads != p.n_kv_heads))
        return (int)cudaErrorInvalidValue;
#define SB_TD(D, V)                                                                                                                 \
    if (p.k_dim == D && p.v_dim == V) {                                                                                             \
        const cudaError_t err =                                                                                                     \
            cudaFuncSetAttribute(talking_decode_kernel<D, V>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);              \
        if (err != cudaSuccess) return (int)err;                                                                                    \
        sb_launch(talking_decode_kernel<D, V>, dim3(batch.n_rows, n_splits), 32 * p.n_kv_heads, (size_t)smem, stream, p, batch,    \
                  (__nv_bfloat16*)out, n_splits, partial);                                                                          \
    }
    SB_TD(64, 64)
    SB_TD(64, 128)
    SB_TD(128, 64)
    SB_TD(128, 128)
#undef SB_TD
    if (n_splits > 1) sb_talking_merge_bf16(partial, out, p.sink, batch.n_rows, p.n_heads, n_splits, p.v_dim, stream);
    SB_LAUNCH_CHECK();
}

}  // extern "C"
