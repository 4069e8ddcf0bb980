// The attention of attention_flex.cu for prompts on the Blackwell tensor cores: S = Q K^T and O = P V by tcgen05.mma, S, P
// and O in tensor memory, keys and values brought in by TMA, bfloat16.  Two entries:
//   sb_flex_attention_tc        cache pages, key widths of 64 or 128 columns, values of 64 or 128; any number of query heads per
//                               key/value head; every option of the call (scale, per-head temperature, distance penalty, window,
//                               chunk, sink, fewer value heads than key heads, values inside the key rows) but pinned pages;
//   sb_flex_attention_tc_rows   the step's own rows, one key head per query head, 64 + 32 key columns with values of 64 or 128 + 64
//                               with values of 128; scale and sink.  Other widths have no such form here.
//
// The work is laid out as in attn_prefill_tc.cu, where the reasons are measured: a block owns 128 (position, query head of
// the group) rows of one sequence and key/value head, one row per thread and per lane of tensor memory; one thread of a
// fifth warp issues every product, one of a sixth every copy; S of the next 64 keys is computed while the rows work on the
// last ones; O stays in tensor memory and is rescaled only when a row's reference maximum moves by more than 2^8; blocks
// start longest first across all heads.  What differs:
//   * a weight w meets its value as two bfloat16 numbers hi + lo (hi = bf16(w), lo = bf16(w - hi)), so that it keeps 16
//     bits, as in attention_flex_mma.cu: hi and lo take the two halves of the S buffer they came from, and eight products
//     (instead of four) read them from there.  w is one instruction (ex2.approx, 2^-22) where that kernel calls expf: next to the
//     weight's 16 bits the difference is nothing.  Errors against 64 bits over 200 to 3,333 rows, up to 9,200 keys, scores of
//     size 1 to 8, with sink, window, temperature and penalty: that kernel / this / this with expf 1.607334e-3 / 1.607334e-3 /
//     1.607334e-3, 1.656125e-3 / 1.656126e-3 / 1.656126e-3, at most 1.645750e-3 / 1.645765e-3 / 1.645770e-3 (200 rows behind 9,000
//     keys), the largest error the same in all; with expf a call takes 14 to 28% longer (2,048 rows of 16 heads on 8 of
//     128 47.6 -> 54.7 us, with temperature and penalty 57.9 -> 72.4);
//   * with a temperature or a penalty per head (BIASED) the scores are finished before their maximum is taken;
//   * DENSE: keys and values are not in cache pages but rows of the step itself, every sequence at its start: a key is a
//     head's own columns of one matrix beside columns of another that all heads share (a latent layer's plain and rotated
//     parts), so that nothing has to be copied together first.
// Key width 192 keeps one stage of values instead of two: with two, a second block would not fit the SM.
//
// Bound: the row threads' instructions (exponentials, the split of the weights, trips to tensor memory), not the tensor
// core.  Measured (B200, us a call with its launch, 64-row mma.sync kernel / this one): one prompt, 16 heads on 8 of 128 with
// temperature, penalty and chunks of 2,048: 500 tokens 39 / 26, 2,048 tokens 220 / 52, 8,192 tokens 673 / 129; without them
// 8,192 tokens 2,342 / 334; 16 heads on 4 of 64: 143 / 39 at 2,048, 1,436 / 269 at 8,192; six prompts of 700 160 / 45.
#include "attention_flex.cuh"
#include "tc_maps.cuh"
#include "tc_utils.cuh"

#define FT_ROWS 128
#define FT_IDS 128       // one per row thread
#define FT_THREADS 256   // the rows; and a group of four warps of which one thread issues products and one copies

// Where a DENSE call's keys and values lie (column offsets are in the maps' matrices).
struct FlexRows {
    int key_cols;    // columns of a head in the matrix of plain keys
    int shared_col;  // first column of the shared part in its matrix
    int value_cols;  // columns of a head in the matrix of values
};

template <int KD, int VD, bool DENSE, bool BIASED>
__global__ void __launch_bounds__(FT_THREADS, 2)
flex_attention_tc_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_s,
                         const __grid_constant__ CUtensorMap map_v, SbFlex p, SbBatch batch, __nv_bfloat16* __restrict__ out,
                         FlexRows dense, int* status) {
    constexpr int ATOMS = (KD + 63) / 64, V_ATOMS = VD / 64, V_STAGES = KD > 128 ? 1 : 2;
    static_assert(DENSE || V_STAGES == 2, "the refill of the page ids counts on values being asked for before the keys after them");
    constexpr int SHARED_ATOM = DENSE ? ATOMS - 1 : ATOMS;   // the last block of 64 columns comes from the shared matrix
    constexpr int Q_ATOM = FT_ROWS * 128;          // bytes of a [128 rows][64 columns] block of Q
    constexpr int KV_ATOM = SB_PAGE * 128;         // bytes of a [64 keys][64 columns] block of K or V
    constexpr int K_STAGE = ATOMS * KV_ATOM, V_STAGE = V_ATOMS * KV_ATOM;
    extern __shared__ __align__(1024) unsigned char smem[];
    unsigned char* q_s = smem;
    unsigned char* k_s = q_s + ATOMS * Q_ATOM;     // [2 stages]
    unsigned char* v_s = k_s + 2 * K_STAGE;        // [V_STAGES]
    uint64_t* bars = (uint64_t*)(v_s + V_STAGES * V_STAGE);
    uint64_t* k_full = bars;                       // [2] keys of a page have landed in stage i & 1
    uint64_t* v_full = bars + 2;                   // [V_STAGES] values likewise
    uint64_t* s_done = bars + 4;                   // [2] S of page i is in S buffer i & 1
    uint64_t* o_done = bars + 6;                   // [2] O += P V of page i is done
    uint64_t* p_ready = bars + 8;                  // every row has read S of page i and written its P (128 arrivals)
    uint32_t* tmem_slot = (uint32_t*)(bars + 9);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
    int* s_pages = (int*)(tmem_slot + 4);          // [FT_IDS] ids of the block's next pages
    if ((smem_u32(smem) & 1023u) != 0) {           // the swizzled tiles need it; never seen, but never assumed
        if (threadIdx.x == 0) atomicOr(status, SB_STATUS_TIMEOUT);
        return;
    }

    const int seq = blockIdx.z, kvh = blockIdx.x;
    const int tid = threadIdx.x, warp = tid >> 5;
    const int G = p.n_heads / p.n_kv_heads;
    const int slot = DENSE ? 0 : batch.seq_slot[seq];
    const int row0 = batch.cu_q[seq];
    const int q_len = batch.cu_q[seq + 1] - row0;
    const int start = DENSE ? 0 : batch.lengths[slot];
    const int total = q_len * G;
    const int tile = gridDim.y - 1 - blockIdx.y;   // latest rows (most keys) first, across all heads
    const int t0 = tile * FT_ROWS;
    if (t0 >= total) return;
    const int t_last = min(t0 + FT_ROWS, total) - 1;
    const int pos_min = start + t0 / G, pos_max = start + t_last / G;
    const int lo_min = flex_first_key(p, pos_min), lo_max = flex_first_key(p, pos_max);
    const int first_page = lo_min / SB_PAGE, last_page = pos_max / SB_PAGE;
    const int n_pages = last_page - first_page + 1;

    const int* table = DENSE ? nullptr : p.table + (long long)slot * p.table_width;
    auto page_id = [&](int lp) {
        if (p.ring_pages) lp %= p.ring_pages;
        return lp < p.table_width ? max(table[lp], 0) : 0;
    };
    // Copies of one page's keys (or values), given what the page is: its id, or its first row among the step's.
    auto copy_k = [&](int i, int place) {
        unsigned char* to = k_s + (i & 1) * K_STAGE;
        uint64_t* bar = &k_full[i & 1];
        mbar_expect_tx(bar, K_STAGE);
#pragma unroll
        for (int a = 0; a < ATOMS; ++a) {
            if (DENSE && a == SHARED_ATOM) tma_load_2d(to + a * KV_ATOM, &map_s, dense.shared_col, place, bar);
            else if (DENSE) tma_load_2d(to + a * KV_ATOM, &map_k, kvh * dense.key_cols + 64 * a, place, bar);
            else tma_load_2d(to + a * KV_ATOM, &map_k, 64 * a, (place * p.n_kv_heads + kvh) * SB_PAGE, bar);
        }
    };
    auto copy_v = [&](int i, int place) {
        const int st = i % V_STAGES;
        uint64_t* bar = &v_full[st];
        mbar_expect_tx(bar, V_STAGE);
#pragma unroll
        for (int a = 0; a < V_ATOMS; ++a)
            tma_load_2d(v_s + st * V_STAGE + a * KV_ATOM, &map_v, (DENSE ? kvh * dense.value_cols : 0) + 64 * a,
                        DENSE ? place : (int)flex_value_page(p, place, kvh), bar);
    };
    auto place_now = [&](int i) { return DENSE ? row0 + (first_page + i) * SB_PAGE : page_id(first_page + i); };
    pdl_wait();
    if (tid == FT_ROWS) {   // barriers, and the first keys and values at once
#pragma unroll
        for (int b = 0; b < 8; ++b) mbar_init(&bars[b], 1);
        mbar_init(p_ready, FT_ROWS);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        for (int i = 0; i < 2 && i < n_pages; ++i) {
            const int place = place_now(i);
            copy_k(i, place);
            if (i == 0) copy_v(0, place);
        }
    }
    if (warp == 0) tmem_alloc(tmem_slot, 256u);
    // This thread's query row into shared memory, in the swizzled K-major layout the tensor core reads.
    const bool owns_row = tid < FT_ROWS;
    const int t = t0 + tid;
    const int head = kvh * G + (t < total ? t % G : 0);
    const long long grow = row0 + (t < total ? t / G : 0);
    const int pos = t < total ? start + t / G : -1;
    const int lo = t < total ? flex_first_key(p, pos) : 0;
    if (owns_row) {
        const __nv_bfloat16* src = (const __nv_bfloat16*)p.q + grow * p.q_row + (long long)head * p.q_head;
#pragma unroll
        for (int c = 0; c < KD / 8; ++c) {
            uint4 v = make_uint4(0u, 0u, 0u, 0u);
            if (t < total) v = *reinterpret_cast<const uint4*>(src + c * 8);
            *reinterpret_cast<uint4*>(q_s + (c >> 3) * Q_ATOM + tid * 128 + (((c & 7) ^ (tid & 7)) << 4)) = v;
        }
    }
    // Ids of the block's pages: a ring of FT_IDS entries in two halves.  Both are filled at the start; every 64 pages the rows
    // refill the half behind them with the pages 64 to 127 ahead (below).
    if (!DENSE && owns_row && tid < n_pages) s_pages[tid] = page_id(first_page + tid);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // Q was written by ordinary stores
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const uint32_t tmem_row = tmem + ((uint32_t)((warp & 3) * 32) << 16);   // this warp's 32 lanes
    const uint32_t idesc_s = umma_idesc(SB_PAGE, 0), idesc_o = umma_idesc(VD, 1);
    constexpr uint32_t O_COL = 2 * SB_PAGE;        // tensor memory: S buffers at columns 0 and 64, O from 128

    if (!owns_row) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 56;" ::: "memory");
        if (tid == FT_ROWS) {   // the products
            const uint64_t q_desc0 = desc_k_major(q_s), k_desc0 = desc_k_major(k_s), v_desc0 = desc_mn_major(v_s, KV_ATOM);
            auto issue_s = [&](int i) {   // S of page i into S buffer i & 1
                mbar_wait(&k_full[i & 1], (i >> 1) & 1, abort_flag, status);
                tc_fence_after();
#pragma unroll
                for (int ks = 0; ks < KD / 16; ++ks)
                    tc_mma(tmem + (i & 1) * SB_PAGE, q_desc0 + (ks >> 2) * (Q_ATOM >> 4) + 2 * (ks & 3),
                           k_desc0 + (i & 1) * (K_STAGE >> 4) + (ks >> 2) * (KV_ATOM >> 4) + 2 * (ks & 3), idesc_s, ks > 0 ? 1u : 0u);
                tc_commit(&s_done[i & 1]);
            };
            issue_s(0);
            for (int i = 0; i < n_pages && !*abort_flag; ++i) {
                const int b = i & 1, st = i % V_STAGES;
                if (i + 1 < n_pages) issue_s(i + 1);   // its buffer was read by the rows before p_ready of i - 1
                mbar_wait(p_ready, i & 1, abort_flag, status);
                mbar_wait(&v_full[st], (i / V_STAGES) & 1, abort_flag, status);
                if (*abort_flag) break;
                tc_fence_after();
#pragma unroll
                for (int part = 0; part < 2; ++part)   // the weights' upper and lower halves
#pragma unroll
                    for (int ks = 0; ks < SB_PAGE / 16; ++ks)
                        tc_mma_ts(tmem + O_COL, tmem + b * SB_PAGE + 32 * part + 8 * ks, v_desc0 + st * (V_STAGE >> 4) + ks * (2048 >> 4),
                                  idesc_o, (i > 0 || part > 0 || ks > 0) ? 1u : 0u);
                tc_commit(&o_done[b]);
            }
        } else if (tid == FT_ROWS + 32) {   // the copies
            for (int i = 0; i < n_pages && !*abort_flag; ++i) {
                auto next_v = [&]() {   // into the stage of page i + 1 - V_STAGES, once its product is done
                    if (i + 1 >= n_pages) return;
                    const int before = i + 1 - V_STAGES;
                    if (before >= 0) mbar_wait(&o_done[before & 1], (before >> 1) & 1, abort_flag, status);
                    if (*abort_flag) return;
                    copy_v(i + 1, DENSE ? place_now(i + 1) : s_pages[(i + 1) & (FT_IDS - 1)]);
                };
                if (V_STAGES == 2) next_v();
                if (i + 2 < n_pages && !*abort_flag) {   // keys two pages ahead go into the stage of page i, once S of page i has read it
                    mbar_wait(&s_done[i & 1], (i >> 1) & 1, abort_flag, status);
                    if (!*abort_flag) copy_k(i + 2, DENSE ? place_now(i + 2) : s_pages[(i + 2) & (FT_IDS - 1)]);
                }
                if (V_STAGES == 1 && !*abort_flag) next_v();
            }
            if (*abort_flag) {   // leaving early: give the copies in flight a bounded time to land
                const long long t_abort = clock64();
                while (clock64() - t_abort < (1ll << 22)) {}
            }
        }
        tc_fence_before();
        __syncthreads();   // the block's last meeting: the rows free tensor memory after it
        return;
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 200;" ::: "memory");
        constexpr float LOG2E = 1.4426950408889634f;
        const float scale2 = (p.head_scale != nullptr ? p.scale * p.head_scale[head] : p.scale) * LOG2E;
        const float slope2 = p.slopes != nullptr ? p.slopes[head] * LOG2E : 0.f;
        float m_ref = -INFINITY, l_run = 0.f;
        for (int i = 0; i < n_pages; ++i) {
            const int b = i & 1;
            // The half of pages i - 64 to i - 1 may be overwritten once S of page i is done: that took the keys of page i, which
            // the copying thread asked for after the values of page i - 1, the last id it reads there.  The fetch of the new ids
            // needs no such wait, and is under way during it.
            const bool refill = !DENSE && i > 0 && (i & 63) == 0 && tid < 64 && i + 64 + tid < n_pages;
            const int next_id = refill ? page_id(first_page + i + 64 + tid) : 0;
            mbar_wait(&s_done[b], (i >> 1) & 1, abort_flag, status);
            if (*abort_flag) break;
            if (refill) s_pages[(i + 64 + tid) & (FT_IDS - 1)] = next_id;
            tc_fence_after();
            const int key0 = (first_page + i) * SB_PAGE;
            float s[SB_PAGE];
            {
                uint32_t* raw = reinterpret_cast<uint32_t*>(s);
                tc_ld32_async(tmem_row + b * SB_PAGE, raw);
                tc_ld32_async(tmem_row + b * SB_PAGE + 32, raw + 32);
                tc_wait_ld();
            }
            if (BIASED) {   // in the log2 domain, penalty included
                const float2 sc = make_float2(scale2, scale2), sl = make_float2(slope2, slope2);
                const float far = (float)(key0 - pos);
#pragma unroll
                for (int c = 0; c < SB_PAGE; c += 2) {
                    const float2 bias = fma_pair(sl, add_pair(make_float2(far, far), make_float2((float)c, (float)(c + 1))), make_float2(0.f, 0.f));
                    const float2 x = fma_pair(make_float2(s[c], s[c + 1]), sc, bias);
                    s[c] = x.x;
                    s[c + 1] = x.y;
                }
            }
            const bool whole_page_visible = key0 + SB_PAGE - 1 <= pos_min && key0 >= lo_max && t_last == t0 + FT_ROWS - 1;
            if (!whole_page_visible) {
#pragma unroll
                for (int c = 0; c < SB_PAGE; ++c) {
                    const int n = key0 + c;
                    if (!(n <= pos && n >= lo)) s[c] = -INFINITY;
                }
            }
            float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int c = 0; c < SB_PAGE; c += 8) {
                mx4[0] = max_of_three(mx4[0], s[c], s[c + 1]); mx4[1] = max_of_three(mx4[1], s[c + 2], s[c + 3]);
                mx4[2] = max_of_three(mx4[2], s[c + 4], s[c + 5]); mx4[3] = max_of_three(mx4[3], s[c + 6], s[c + 7]);
            }
            float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
            if (!BIASED) mx *= scale2;   // scale2 > 0 here: the maximum commutes with it
            float alpha = 1.0f;
            if (mx > m_ref + 8.0f || m_ref == -INFINITY) {
                const float m_new = fmaxf(m_ref, mx);
                alpha = m_new == -INFINITY ? 1.0f : exp2f(m_ref - m_new);   // 0 when the reference was -inf
                m_ref = m_new;
            }
            const float m_use = m_ref == -INFINITY ? 0.f : m_ref;
            uint32_t hi[SB_PAGE / 2], lo2[SB_PAGE / 2];
            const float2 sc = make_float2(BIASED ? 1.f : scale2, BIASED ? 1.f : scale2), shift = make_float2(-m_use, -m_use);
            float2 sum2[4] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
            for (int c = 0; c < SB_PAGE; c += 2) {
                const float2 sv = make_float2(s[c], s[c + 1]);
                const float2 x = BIASED ? add_pair(sv, shift) : fma_pair(sv, sc, shift);
                const float2 pr = make_float2(fast_exp2(x.x), fast_exp2(x.y));
                sum2[(c >> 1) & 3] = add_pair(sum2[(c >> 1) & 3], pr);
                const __nv_bfloat162 h2 = __floats2bfloat162_rn(pr.x, pr.y);
                const uint32_t h = *reinterpret_cast<const uint32_t*>(&h2);
                const float2 rest = add_pair(pr, make_float2(-__uint_as_float(h << 16), -__uint_as_float(h & 0xffff0000u)));
                const __nv_bfloat162 l2 = __floats2bfloat162_rn(rest.x, rest.y);
                hi[c >> 1] = h;
                lo2[c >> 1] = *reinterpret_cast<const uint32_t*>(&l2);
            }
            l_run = l_run * alpha + (((sum2[0].x + sum2[0].y) + (sum2[1].x + sum2[1].y)) + ((sum2[2].x + sum2[2].y) + (sum2[3].x + sum2[3].y)));

            if (i > 0 && __any_sync(0xffffffffu, alpha != 1.0f)) {   // O of the earlier pages moves to the new reference
                mbar_wait(&o_done[(i - 1) & 1], ((i - 1) >> 1) & 1, abort_flag, status);
                if (*abort_flag) break;
                tc_fence_after();
#pragma unroll
                for (int d0 = 0; d0 < VD; d0 += 32) {
                    float o[32];
                    tc_ld32(tmem_row + O_COL + d0, o);
#pragma unroll
                    for (int d = 0; d < 32; ++d) o[d] *= alpha;
                    tc_st32(tmem_row + O_COL + d0, o);
                }
            }
            // Values of keys that no row of this block may see are whatever a former owner left (or another sequence's): they
            // meet weights of exactly zero, but zero times an infinity or a NaN would not be zero.  Only a block's last
            // (and, with a window or chunk, first) page has such rows; thread k clears the row of key k.
            if (key0 + SB_PAGE - 1 > pos_max || key0 < lo_min) {
                const int st = i % V_STAGES;
                mbar_wait(&v_full[st], (i / V_STAGES) & 1, abort_flag, status);
                if (*abort_flag) break;
                if (tid < SB_PAGE && (key0 + tid > pos_max || key0 + tid < lo_min)) {
                    unsigned char* vt = v_s + st * V_STAGE;
#pragma unroll
                    for (int c = 0; c < V_ATOMS * 8; ++c)
                        *reinterpret_cast<uint4*>(vt + (c >> 3) * KV_ATOM + tid * 128 + ((c & 7) << 4)) = make_uint4(0u, 0u, 0u, 0u);
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                }
            }
            tc_st32_u32(tmem_row + b * SB_PAGE, hi);
            tc_st32_u32(tmem_row + b * SB_PAGE + 32, lo2);
            tc_fence_before();
            mbar_arrive(p_ready);
        }
        if (!*abort_flag) {
            mbar_wait(&o_done[(n_pages - 1) & 1], ((n_pages - 1) >> 1) & 1, abort_flag, status);
            tc_fence_after();
        }
        if (!*abort_flag) {
            float mul = 1.0f / l_run;
            if (p.sink != nullptr) {
                const float sk = p.sink[head] * LOG2E, mf = fmaxf(m_ref, sk), a = exp2f(m_ref - mf);
                mul = a / (l_run * a + exp2f(sk - mf));
            }
            __nv_bfloat16* o_row = out + (grow * p.n_heads + head) * VD;
#pragma unroll
            for (int d0 = 0; d0 < VD; d0 += 32) {
                float o[32];
                tc_ld32(tmem_row + O_COL + d0, o);
                if (t < total) {
#pragma unroll
                    for (int d = 0; d < 32; d += 8) {
                        uint4 packed;
                        __nv_bfloat162* h2 = reinterpret_cast<__nv_bfloat162*>(&packed);
#pragma unroll
                        for (int e = 0; e < 4; ++e) h2[e] = __floats2bfloat162_rn(o[d + 2 * e] * mul, o[d + 2 * e + 1] * mul);
                        *reinterpret_cast<uint4*>(o_row + d0 + d) = packed;
                    }
                }
            }
        }
        tc_fence_before();
        __syncthreads();
        if (warp == 0) tmem_dealloc(tmem, 256u);
    }
}

// ---- host side ----------------------------------------------------------------------------------

template <int KD, int VD, bool DENSE, bool BIASED>
static int launch_flex_tc(const CUtensorMap& mk, const CUtensorMap& ms, const CUtensorMap& mv, SbFlex p, SbBatch batch, void* out,
                          FlexRows dense, int max_q_len, int* status, cudaStream_t stream) {
    constexpr int atoms = (KD + 63) / 64, v_stages = KD > 128 ? 1 : 2;
    constexpr int smem = atoms * FT_ROWS * 128 + 2 * atoms * SB_PAGE * 128 + v_stages * (VD / 64) * SB_PAGE * 128 + 96 + FT_IDS * 4;
    static bool configured[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        const cudaError_t e = cudaFuncSetAttribute(flex_attention_tc_kernel<KD, VD, DENSE, BIASED>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return (int)e;
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    const int G = p.n_heads / p.n_kv_heads;
    const long long tiles = ((long long)max_q_len * G + FT_ROWS - 1) / FT_ROWS;
    if (tiles > 65535 || batch.n_seqs > 65535) return (int)cudaErrorInvalidValue;
    const dim3 grid(p.n_kv_heads, (unsigned int)tiles, batch.n_seqs);
    sb_launch(flex_attention_tc_kernel<KD, VD, DENSE, BIASED>, grid, FT_THREADS, smem, stream, mk, ms, mv, p, batch, (__nv_bfloat16*)out, dense,
              status);
    return (int)cudaGetLastError();
}

extern "C" {

// Whether the kernel takes these sizes.  `dense`: keys of k_dim columns of which the last block of 64 (or fewer) is shared.
int sb_flex_attention_tc_takes(int k_dim, int v_dim, int dense) {
    if (v_dim != 64 && v_dim != 128) return 0;
    if (dense) return (k_dim == 96 && v_dim == 64) || (k_dim == 192 && v_dim == 128);
    return k_dim == 64 || k_dim == 128;
}

// Keys and values in the layer's pages; n_pages: pages in its pool (the null page included).
int sb_flex_attention_tc(SbFlex p, SbBatch batch, void* out, int max_q_len, int n_pages, int* status, cudaStream_t stream) {
    if (batch.n_rows <= 0) return 0;
    const bool biased = p.head_scale != nullptr || p.slopes != nullptr;
    if (!sb_flex_attention_tc_takes(p.k_dim, p.v_dim, 0) || max_q_len < 1 || n_pages < 1 || p.pinned_pages || (!biased && !(p.scale > 0.f)))
        return (int)cudaErrorInvalidValue;
    const int v_heads = p.v_heads > 0 ? p.v_heads : p.n_kv_heads;
    CUtensorMap mk, mv;
    int e = make_rows_map(&mk, p.k, (long long)n_pages * p.n_kv_heads * SB_PAGE, p.k_dim, p.k_dim, SB_PAGE);
    if (!e) e = make_rows_map(&mv, p.v, (long long)n_pages * v_heads * SB_PAGE, p.v_dim, p.v_row, SB_PAGE);
    if (e) return e;
    const FlexRows none = {0, 0, 0};
#define FT_CASE(KD, VD)                                                                                                       \
    if (p.k_dim == KD && p.v_dim == VD)                                                                                       \
        return biased ? launch_flex_tc<KD, VD, false, true>(mk, mk, mv, p, batch, out, none, max_q_len, status, stream)       \
                      : launch_flex_tc<KD, VD, false, false>(mk, mk, mv, p, batch, out, none, max_q_len, status, stream);
    FT_CASE(64, 64)
    FT_CASE(64, 128)
    FT_CASE(128, 64)
    FT_CASE(128, 128)
#undef FT_CASE
    return (int)cudaErrorInvalidValue;
}

// Keys and values among the step's own rows, every sequence from its first token on: plain keys [rows, heads * keep] (keep
// a multiple of 64) plain_ld apart, the part that all heads share at shared[row * shared_ld .. + k_dim - keep], values
// [rows, heads * v_dim] values_ld apart.  p: queries, scale, sink; one key/value head per query head.
int sb_flex_attention_tc_rows(SbFlex p, SbBatch batch, const void* plain, long long plain_ld, const void* shared, long long shared_ld,
                              const void* values, long long values_ld, void* out, int max_q_len, int* status, cudaStream_t stream) {
    if (batch.n_rows <= 0) return 0;
    if (!sb_flex_attention_tc_takes(p.k_dim, p.v_dim, 1) || max_q_len < 1 || p.n_heads != p.n_kv_heads || !(p.scale > 0.f) ||
        p.head_scale != nullptr || p.slopes != nullptr)
        return (int)cudaErrorInvalidValue;
    const int keep = (p.k_dim - 1) / 64 * 64, rest = p.k_dim - keep;
    CUtensorMap mk, ms, mv;
    int e = make_rows_map(&mk, plain, batch.n_rows, (long long)p.n_heads * keep, plain_ld, SB_PAGE);
    if (!e) e = make_rows_map(&ms, shared, batch.n_rows, rest, shared_ld, SB_PAGE);
    if (!e) e = make_rows_map(&mv, values, batch.n_rows, (long long)p.n_heads * p.v_dim, values_ld, SB_PAGE);
    if (e) return e;
    const FlexRows dense = {keep, 0, p.v_dim};
    if (p.k_dim == 96) return launch_flex_tc<96, 64, true, false>(mk, ms, mv, p, batch, out, dense, max_q_len, status, stream);
    return launch_flex_tc<192, 128, true, false>(mk, ms, mv, p, batch, out, dense, max_q_len, status, stream);
}

}  // extern "C"
