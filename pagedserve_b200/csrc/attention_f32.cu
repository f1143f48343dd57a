// Paged causal attention in float32 on CUDA cores, for head sizes that are multiples of 4 up to 128 (other sizes run on the
// general kernel of attention_simt.cu, whose cache layout, masks, cap, sink and all_values these share).
//
// prompt_attention_f32_kernel: prompt portions, 64 queries of one head per CTA, key tiles of 64 aligned to absolute positions (head sizes of
//                              36 to 64 run on tensor cores instead: attention_f32_tc.cu).
// token_attention_f32_kernel:  single tokens (decode steps, short portions), one CTA per (token, head).
// Scores, softmax and results are float32 throughout (expf, tanhf).  Within each kernel the order of every sum depends only on a
// query's position (reference: src/model/paged_attention.py:262-295): its bits are the same whatever else is in the step and, of
// portions that all run on one kernel, wherever a prompt was cut.  The two add in different orders (the prompt kernel key by key with a
// running maximum, the token kernel in states per lane group that are merged), so a query of a short portion differs from the same query of
// a long one by the rounding of float32 sums.  One order for both (states per tile of 64 keys, joined in order) was measured: 12 heads of 64,
// one token, 100 keys 4.2 -> 7.2 us, 1,000 keys 18.2 -> 23.7.
#include "common.cuh"

namespace ps {
namespace af32 {

// position -> offset of its row (of head g) in the pool, or -1 where the request has no page there; pages are 1 << shift long
__device__ __forceinline__ long long row_offset(const int* bt, int key, int shift, long long page_stride, int g, int head_dim) {
    const int page = bt[key >> shift];
    return page < 0 ? -1 : (long long)page * page_stride + (long long)(((g << shift) + (key & ((1 << shift) - 1))) * head_dim);
}
__device__ __forceinline__ void copy16(float* dst, const float* src, bool ok) {        // not ok: zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
                 ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(ok ? 16 : 0) : "memory");
}
__device__ __forceinline__ void commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT> __device__ __forceinline__ void wait_copies() { asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory"); }
__device__ __forceinline__ float capped(float score, float softcap) {
    return softcap > 0.f ? softcap * tanhf(score / softcap) : score;
}

constexpr int BQ = 64, BKEY = 64, PROMPT_THREADS = 128;

template <int HD> struct PromptTiles {
    static constexpr int ROW = HD + 4;             // pitch of Q, K and V: eight neighbouring rows on eight groups of four banks
    static constexpr int PROW = BKEY + 8;          // pitch of the weights
    static constexpr int K = BQ * ROW, V = K + BKEY * ROW, P = V + BKEY * ROW;
    static constexpr size_t BYTES = (size_t)(P + BQ * PROW) * sizeof(float);
};

// o += weights . values of one tile of keys; EDGE: rows pos + 4 i leave out the keys that they do not see
template <int HD, bool EDGE>
__device__ __forceinline__ void add_values(float (&o)[4][HD / 8], const float* p_row, const float* v_row, int key0, int pos,
                                           const int (&low)[4]) {
    using T = PromptTiles<HD>;
#pragma unroll 4
    for (int key = 0; key < BKEY; key += 4) {
        float p[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float4 four = *reinterpret_cast<const float4*>(p_row + 4 * i * T::PROW + key);
            p[i][0] = four.x; p[i][1] = four.y; p[i][2] = four.z; p[i][3] = four.w;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int c = 0; c < HD / 32; ++c) {
                const float4 v = *reinterpret_cast<const float4*>(v_row + (key + k) * T::ROW + 32 * c);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (EDGE && (key0 + key + k > pos + 4 * i || key0 + key + k < low[i])) continue;
                    o[i][4 * c] = fmaf(p[i][k], v.x, o[i][4 * c]);
                    o[i][4 * c + 1] = fmaf(p[i][k], v.y, o[i][4 * c + 1]);
                    o[i][4 * c + 2] = fmaf(p[i][k], v.z, o[i][4 * c + 2]);
                    o[i][4 * c + 3] = fmaf(p[i][k], v.w, o[i][4 * c + 3]);
                }
            }
    }
}

// What bounds it: multiply-adds (128 per clock and SM) beside the reads of their operands from shared memory.  A warp owns 16
// queries, so the weights of a row never leave it; a thread computes 4 x 8 scores (queries ty + 4 i, keys tx + 8 j) and
// 4 x HD / 8 results (4 tx + 32 c + 0..3).  One buffer each for keys and values: the next keys are on their way while the
// weights meet the values, the next values while the scores are formed.  Head sizes below HD are filled up with zeros.
// Blocks late in their prompt see the most keys and go first.
template <int HD>
__global__ void __launch_bounds__(PROMPT_THREADS, HD <= 32 ? 3 : 1)
prompt_attention_f32_kernel(const float* __restrict__ q, int q_stride, float* __restrict__ out, int out_stride,
                            const float* __restrict__ k_pool, const float* __restrict__ v_pool, long long page_stride,
                            const int* __restrict__ q_start, const int* __restrict__ kv_len, const int* __restrict__ block_table,
                            int bt_stride, const int* __restrict__ item_row, int first_item, int n_items, int n_heads,
                            int n_kv_heads, int head_dim, int page_size, int window, float scale, float softcap,
                            const float* __restrict__ sink, int all_values) {
    using T = PromptTiles<HD>;
    constexpr int ROW = T::ROW, PIECES = HD / 4, CHUNKS = HD / 32;
    extern __shared__ __align__(16) float smem[];
    float *q_s = smem, *k_s = smem + T::K, *v_s = smem + T::V, *p_s = smem + T::P;
    pdl_prologue();
    q = pdl_fresh(q);
    k_pool = pdl_fresh(k_pool);
    v_pool = pdl_fresh(v_pool);
    int block = blockIdx.y, item = -1, qb = 0;
    for (int i = first_item; i < first_item + n_items; ++i) {
        const int blocks = (q_start[i + 1] - q_start[i] + BQ - 1) / BQ;
        if (block < blocks) { item = i; qb = blocks - 1 - block; break; }
        block -= blocks;
    }
    if (item < 0) return;
    const int column = blockIdx.x, h = all_values ? column / n_kv_heads : column, g = h / (n_heads / n_kv_heads);
    const long long to_value = all_values ? (long long)(column % n_kv_heads - g) * page_size * head_dim : 0;
    const int q_len = q_start[item + 1] - q_start[item];
    const int pos0 = kv_len[item] - q_len + qb * BQ, tok0 = q_start[item] + qb * BQ;
    const int rows = min(BQ, q_len - qb * BQ), hi = pos0 + rows - 1;
    const int lo = first_visible_key(pos0, window);
    const int* bt = block_table + (size_t)(item_row ? item_row[item] : item) * bt_stride;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, ty = lane >> 3, tx = lane & 7;
    const int shift = 31 - __clz(page_size);

    for (int c = tid; c < BQ * PIECES; c += PROMPT_THREADS) {
        const int r = c / PIECES, d = (c % PIECES) * 4;
        const bool ok = r < rows && d < head_dim;
        copy16(q_s + r * ROW + d, q + (ok ? (size_t)(tok0 + r) * q_stride + h * head_dim + d : 0), ok);
    }
    auto load = [&](int tile, const float* pool, long long beyond, float* to) {
        for (int c = tid; c < BKEY * PIECES; c += PROMPT_THREADS) {
            const int r = c / PIECES, d = (c % PIECES) * 4, key = tile * BKEY + r;
            const long long at = key >= lo && key <= hi && d < head_dim ? row_offset(bt, key, shift, page_stride, g, head_dim) : -1;
            copy16(to + r * ROW + d, pool + (at >= 0 ? at + beyond + d : 0), at >= 0);
        }
    };
    const int first = lo / BKEY, last = hi / BKEY;
    load(first, k_pool, 0, k_s);
    commit();
    load(first, v_pool, to_value, v_s);
    commit();

    float o[4][4 * CHUNKS], m[4], l[4];
    int low[4];                                                // a row's first visible key
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        m[i] = -INFINITY;
        l[i] = 0.f;
        low[i] = first_visible_key(pos0 + warp * 16 + ty + 4 * i, window);
#pragma unroll
        for (int d = 0; d < 4 * CHUNKS; ++d) o[i][d] = 0.f;
    }
    const float* q_row = q_s + (warp * 16 + ty) * ROW;
    float* p_row = p_s + (warp * 16 + ty) * T::PROW;
    for (int tile = first; tile <= last; ++tile) {
        wait_copies<1>();
        __syncthreads();                                       // the keys (and, at first, the queries) are there
        unsigned long long pair[4][8];                         // sums over even and over odd dimensions
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) pair[i][j] = 0ull;
#pragma unroll
        for (int d = 0; d < HD; d += 4) {
            ulonglong2 a[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(q_row + 4 * i * ROW + d);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(k_s + (tx + 8 * j) * ROW + d);
#pragma unroll
                for (int i = 0; i < 4; ++i) pair[i][j] = pair_fma(a[i].x, b.x, pair[i][j]);
#pragma unroll
                for (int i = 0; i < 4; ++i) pair[i][j] = pair_fma(a[i].y, b.y, pair[i][j]);
            }
        }
        __syncthreads();                                       // everyone is done with the keys
        if (tile < last) load(tile + 1, k_pool, 0, k_s);
        commit();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int pos = pos0 + warp * 16 + ty + 4 * i;
            float s[8], top = -INFINITY;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                float even, odd;
                pair_split(pair[i][j], even, odd);
                const int key = tile * BKEY + tx + 8 * j;
                s[j] = key <= pos && key >= low[i] ? capped((even + odd) * scale, softcap) : -INFINITY;
                top = fmaxf(top, s[j]);
            }
#pragma unroll
            for (int x = 1; x < 8; x <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, x));
            const float m_new = fmaxf(m[i], top);
            const float base = m_new == -INFINITY ? 0.f : m_new;       // a row that sees no key of this tile or before it
            const float shrink = expf(m[i] - base);
            m[i] = m_new;
            l[i] *= shrink;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float p = expf(s[j] - base);
                l[i] += p;
                p_row[4 * i * T::PROW + tx + 8 * j] = p;
            }
#pragma unroll
            for (int d = 0; d < 4 * CHUNKS; ++d) o[i][d] *= shrink;
        }
        wait_copies<1>();
        __syncthreads();                                       // the values are there (and the warp's weights)
        // A tile that some row of the warp sees only in part: what is not seen stays out of the sums (a weight of zero would
        // make a NaN of an infinity that stands in a later token's values).
        const int warp_pos = pos0 + warp * 16;
        if (tile * BKEY + BKEY - 1 > warp_pos || (window != 0 && tile * BKEY < first_visible_key(warp_pos + 15, window))) {
            add_values<HD, true>(o, p_row, v_s + 4 * tx, tile * BKEY, warp_pos + ty, low);
        } else {
            add_values<HD, false>(o, p_row, v_s + 4 * tx, tile * BKEY, warp_pos + ty, low);
        }
        __syncthreads();                                       // everyone is done with the values
        if (tile < last) load(tile + 1, v_pool, to_value, v_s);
        commit();
    }
    wait_copies<0>();
    const float sink_h = sink ? sink[h] : -INFINITY;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = warp * 16 + ty + 4 * i;
        float total = l[i];
#pragma unroll
        for (int x = 1; x < 8; x <<= 1) total += __shfl_xor_sync(0xffffffffu, total, x);
        float scale_out = 1.f;
        if (sink) {
            const float big = fmaxf(m[i], sink_h);
            scale_out = expf(m[i] - big);
            total = total * scale_out + expf(sink_h - big);
        }
        scale_out /= total;
        if (r >= rows) continue;
        float* to = out + (size_t)(tok0 + r) * out_stride + column * head_dim;
#pragma unroll
        for (int c = 0; c < CHUNKS; ++c) {
            const int d = 32 * c + 4 * tx;
            if (d < head_dim)
                *reinterpret_cast<float4*>(to + d) = make_float4(o[i][4 * c] * scale_out, o[i][4 * c + 1] * scale_out,
                                                                 o[i][4 * c + 2] * scale_out, o[i][4 * c + 3] * scale_out);
        }
    }
}

constexpr int TOKEN_WARPS = 8;

// What bounds it: the latency of a token's keys and values, then their bytes.  HD / 4 lanes hold a row (16 bytes each), so a
// warp reads 128 / HD whole rows at once and has UNROLL of them per lane group, keys and values, on their way together.
// Every lane group keeps a softmax state of its own; the CTA's states are merged in order at the end.
template <int HD>
__global__ void __launch_bounds__(TOKEN_WARPS * 32)
token_attention_f32_kernel(const float* __restrict__ q, int q_stride, float* __restrict__ out, int out_stride,
                           const float* __restrict__ k_pool, const float* __restrict__ v_pool, long long page_stride,
                           const int* __restrict__ token_row, const int* __restrict__ positions,
                           const int* __restrict__ block_table, int bt_stride, int n_heads, int n_kv_heads, int head_dim,
                           int page_size, int window, float scale, float softcap, const float* __restrict__ sink,
                           int all_values) {
    constexpr int LANES = HD / 4, GROUPS = 32 / LANES, UNROLL = 4, STATES = TOKEN_WARPS * GROUPS;
    constexpr int SPAN = STATES * UNROLL;                      // keys of one round of the CTA
    __shared__ float acc_s[STATES][HD];
    __shared__ float m_s[STATES], l_s[STATES];
    pdl_prologue();
    q = pdl_fresh(q);
    k_pool = pdl_fresh(k_pool);
    v_pool = pdl_fresh(v_pool);
    const int t = blockIdx.x, column = blockIdx.y, h = all_values ? column / n_kv_heads : column, g = h / (n_heads / n_kv_heads);
    const long long to_value = all_values ? (long long)(column % n_kv_heads - g) * page_size * head_dim : 0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, group = lane / LANES, d = (lane % LANES) * 4;
    const int p = positions[t], lo = first_visible_key(p, window);
    const int* bt = block_table + (size_t)token_row[t] * bt_stride;
    const bool inside = d < head_dim;
    const int shift = 31 - __clz(page_size);
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 query = inside ? *reinterpret_cast<const float4*>(q + (size_t)t * q_stride + h * head_dim + d) : zero;
    float m = -INFINITY, l = 0.f;
    float4 acc = zero;
    for (int round = lo / SPAN * SPAN; round <= p; round += SPAN) {
        float4 k[UNROLL], v[UNROLL];
        bool seen[UNROLL];
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
            const int key = round + (u * TOKEN_WARPS + warp) * GROUPS + group;
            seen[u] = key >= lo && key <= p;
            const long long at = seen[u] ? row_offset(bt, key, shift, page_stride, g, head_dim) : -1;
            k[u] = at >= 0 && inside ? *reinterpret_cast<const float4*>(k_pool + at + d) : zero;
            v[u] = at >= 0 && inside ? *reinterpret_cast<const float4*>(v_pool + at + to_value + d) : zero;
        }
        float s[UNROLL], top = m;
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
            float dot = fmaf(query.w, k[u].w, fmaf(query.z, k[u].z, fmaf(query.y, k[u].y, query.x * k[u].x)));
#pragma unroll
            for (int x = 1; x < LANES; x <<= 1) dot += __shfl_xor_sync(0xffffffffu, dot, x);
            s[u] = seen[u] ? capped(dot * scale, softcap) : -INFINITY;
            top = fmaxf(top, s[u]);
        }
        const float base = top == -INFINITY ? 0.f : top;
        const float shrink = expf(m - base);
        m = top;
        l *= shrink;
        acc.x *= shrink; acc.y *= shrink; acc.z *= shrink; acc.w *= shrink;
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
            const float w = expf(s[u] - base);
            l += w;
            acc.x = fmaf(w, v[u].x, acc.x);
            acc.y = fmaf(w, v[u].y, acc.y);
            acc.z = fmaf(w, v[u].z, acc.z);
            acc.w = fmaf(w, v[u].w, acc.w);
        }
    }
    const int state = warp * GROUPS + group;
    *reinterpret_cast<float4*>(&acc_s[state][d]) = acc;
    if (lane % LANES == 0) { m_s[state] = m; l_s[state] = l; }
    __syncthreads();
    if (threadIdx.x >= head_dim) return;
    const float sink_h = sink ? sink[h] : -INFINITY;
    float big = sink_h;
#pragma unroll
    for (int i = 0; i < STATES; ++i) big = fmaxf(big, m_s[i]);
    float total = sink ? expf(sink_h - big) : 0.f, sum = 0.f;
#pragma unroll
    for (int i = 0; i < STATES; ++i) {
        const float w = m_s[i] == -INFINITY ? 0.f : expf(m_s[i] - big);
        total = fmaf(l_s[i], w, total);
        sum = fmaf(acc_s[i][threadIdx.x], w, sum);
    }
    out[(size_t)t * out_stride + column * head_dim + threadIdx.x] = sum / total;
}

template <int HD>
int launch_prompt(const float* q, int q_stride, float* out, int out_stride, const float* k_pool, const float* v_pool,
                  long long page_stride, const int* q_start, const int* kv_len, const int* block_table, int bt_stride,
                  const int* item_row, int first_item, int n_items, int max_blocks, int n_heads, int n_kv_heads, int head_dim,
                  int page_size, int window, float scale, float softcap, const float* sink, int all_values, cudaStream_t s) {
    auto kernel = prompt_attention_f32_kernel<HD>;
    static size_t raised[MAX_DEVICES] = {0};
    if (!ensure_dynamic_smem((const void*)kernel, PromptTiles<HD>::BYTES, raised)) return PS_ERR_LAUNCH;
    return launch_pdl(kernel, dim3(all_values ? n_heads * n_kv_heads : n_heads, max_blocks), dim3(PROMPT_THREADS),
                      PromptTiles<HD>::BYTES, s, q, q_stride, out, out_stride, k_pool, v_pool, page_stride, q_start, kv_len,
                      block_table, bt_stride, item_row, first_item, n_items, n_heads, n_kv_heads, head_dim, page_size, window,
                      scale, softcap, sink, all_values);
}

int check(const void* q, int q_stride, const void* out, int out_stride, const void* k_pool, const void* v_pool,
          long long page_stride, int n_heads, int n_kv_heads, int head_dim, int page_size, int all_values) {
    if (n_heads <= 0 || n_kv_heads <= 0 || n_heads % n_kv_heads || (long long)n_heads * (all_values ? n_kv_heads : 1) > 65535)
        return PS_ERR_BAD_ARGUMENT;
    if (head_dim <= 0 || head_dim > 128 || head_dim % 4 || q_stride % 4 || out_stride % 4 || page_stride % 4) return PS_ERR_UNSUPPORTED;
    if (page_size <= 0 || page_size > 64 || (page_size & (page_size - 1))) return PS_ERR_UNSUPPORTED;
    if (((uintptr_t)q | (uintptr_t)out | (uintptr_t)k_pool | (uintptr_t)v_pool) & 15) return PS_ERR_UNSUPPORTED;
    return PS_OK;
}

}  // namespace af32
}  // namespace ps

// Items first_item .. of the step (prompt portions; q_start, kv_len and item_row by item), max_blocks >= the number of 64-query
// blocks that they make up.  Everything float32; 16-byte aligned rows.
PS_EXPORT int ps_prompt_attention_f32(const float* q, int q_stride, float* out, int out_stride, const float* k_pool,
                                      const float* v_pool, long long page_stride, const int* q_start, const int* kv_len,
                                      const int* block_table, int bt_stride, const int* item_row, int first_item, int n_items,
                                      int max_blocks, int n_heads, int n_kv_heads, int head_dim, int page_size, int window,
                                      float scale, float softcap, const float* sink, int all_values, void* stream) {
    if (n_items <= 0 || max_blocks <= 0) return PS_OK;
    const int rc = ps::af32::check(q, q_stride, out, out_stride, k_pool, v_pool, page_stride, n_heads, n_kv_heads, head_dim,
                                   page_size, all_values);
    if (rc) return rc;
    if (max_blocks > 65535) return PS_ERR_UNSUPPORTED;
    auto launch = head_dim <= 32 ? ps::af32::launch_prompt<32> : ps::af32::launch_prompt<128>;
    return launch(q, q_stride, out, out_stride, k_pool, v_pool, page_stride, q_start, kv_len, block_table, bt_stride, item_row,
                  first_item, n_items, max_blocks, n_heads, n_kv_heads, head_dim, page_size, window, scale, softcap, sink,
                  all_values, (cudaStream_t)stream);
}

// T single tokens at positions[t], which read the pages of block-table row token_row[t].
PS_EXPORT int ps_token_attention_f32(const float* q, int q_stride, float* out, int out_stride, const float* k_pool,
                                     const float* v_pool, long long page_stride, const int* token_row, const int* positions,
                                     const int* block_table, int bt_stride, int T, int n_heads, int n_kv_heads, int head_dim,
                                     int page_size, int window, float scale, float softcap, const float* sink, int all_values,
                                     void* stream) {
    if (T <= 0) return PS_OK;
    const int rc = ps::af32::check(q, q_stride, out, out_stride, k_pool, v_pool, page_stride, n_heads, n_kv_heads, head_dim,
                                   page_size, all_values);
    if (rc) return rc;
    auto kernel = head_dim <= 32 ? ps::af32::token_attention_f32_kernel<32> : head_dim <= 64 ? ps::af32::token_attention_f32_kernel<64>
                                                                                             : ps::af32::token_attention_f32_kernel<128>;
    return ps::launch_pdl(kernel, dim3(T, all_values ? n_heads * n_kv_heads : n_heads), dim3(ps::af32::TOKEN_WARPS * 32), 0,
                          (cudaStream_t)stream, q, q_stride, out, out_stride, k_pool, v_pool, page_stride, token_row, positions,
                          block_table, bt_stride, n_heads, n_kv_heads, head_dim, page_size, window, scale, softcap, sink,
                          all_values);
}
