// Paged attention of single tokens (decode steps, short portions), bfloat16, on CUDA cores: one CTA per (token, head), the whole context.
//
// HD / 8 lanes hold a row of a key (16 bytes each), so that a warp reads 256 / HD whole rows at once, and UNROLL of them per lane group, keys and
// values straight to registers; nothing passes through shared memory until the warps' states are merged.  A warp's keys of a round share one
// maximum; scores, weights and sums are float32 (the weights are not rounded to bfloat16 as they are where they are an operand of mma.sync).
//   round r: keys r * SPAN + (u * WARPS + warp) * GROUPS + lane group, u < UNROLL, SPAN = UNROLL * WARPS * GROUPS
// A round's rows are asked for while the round before is worked on, and their pages a round earlier.  Rows that are older than the step
// are asked for before the wait for the kernel in front (as in attention_decode.cu, which says why that is allowed).
//
// What bounds it: the latency of a round's rows where there are few (token, head) pairs, so a CTA has as many warps as leave all CTAs resident;
// with many pairs the bytes (six CTAs of 4 warps, 80 KB in flight on an SM).  Against attention_decode.cu, whose chunks pass through shared
// memory behind four barriers, us, other / here (heads of 64, 12 a token): 1 token behind 48 keys 4.0 / 2.1, 500 4.4 / 3.4, 1,000 7.8 / 5.6; 8
// tokens, 300 keys 5.2 / 3.7, 600 8.3 / 6.5; 16, 300 9.8 / 6.2; 64, 160 9.4 / 8.3, 640 33.8 / 28.6 (25 heads 58.7 / 51.1); 256, 160 32.5 / 26.9.
#include "common.cuh"

namespace ps {
namespace lanes {

constexpr int UNROLL = 4;

__device__ __forceinline__ uint4 load_row(const __nv_bfloat16* p) {          // past L1: a row of this step must not come from an older line
    uint4 v;
    asm volatile("ld.global.cg.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ void unpack(const uint4& raw, float (&x)[8]) {
    const uint32_t word[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        x[2 * i] = __uint_as_float(word[i] << 16);
        x[2 * i + 1] = __uint_as_float(word[i] & 0xffff0000u);
    }
}

template <int HD, int WARPS, int RESIDENT>
__global__ void __launch_bounds__(WARPS * 32, RESIDENT)
attention_lanes_kernel(const __nv_bfloat16* __restrict__ q, int q_stride, __nv_bfloat16* __restrict__ out, int out_stride,
                       const __nv_bfloat16* __restrict__ k_pool, const __nv_bfloat16* __restrict__ v_pool, long long page_stride,
                       const int* __restrict__ token_item, const int* __restrict__ token_row, const int* __restrict__ positions,
                       const int* __restrict__ block_table, int bt_stride, const int* __restrict__ q_start,
                       const int* __restrict__ kv_len, int n_heads, int n_kv_heads, int head_dim, int page_log2, int window,
                       float scale_log2, SoftmaxExtras extras, int all_values) {
    constexpr int LANES = HD / 8, GROUPS = 32 / LANES, SPAN = UNROLL * WARPS * GROUPS;
    __shared__ float acc_s[WARPS][HD];
    __shared__ float m_s[WARPS], l_s[WARPS];
    const int t = blockIdx.x, column = blockIdx.y, h = all_values ? column / n_kv_heads : column, g = h / (n_heads / n_kv_heads);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, group = lane / LANES, d = (lane % LANES) * 8;
    // ---- before the wait: only what no kernel of this step writes (positions, tables, older keys)
    const int item = token_item[t], p = positions[t], lo = first_visible_key(p, window);
    const int first_new = (q_start && kv_len) ? kv_len[item] - (q_start[item + 1] - q_start[item]) : 0;
    const int* bt = block_table + (size_t)(token_row ? token_row[t] : item) * bt_stride;
    const int page_size = 1 << page_log2;
    // from a key's place to its value's in the other pool
    const long long to_value = (all_values ? (long long)(column % n_kv_heads - g) * page_size * head_dim : 0);
    const bool inside = d < head_dim;
    const int first = lo / SPAN * SPAN;
    auto key_of = [&](int round, int u) { return round + (u * WARPS + warp) * GROUPS + group; };
    auto seen = [&](int key) { return key >= lo && key <= p; };
    auto fetch_pages = [&](int round, int (&page)[UNROLL]) {
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
            const int key = key_of(round, u);
            page[u] = seen(key) ? bt[key >> page_log2] : -1;
        }
    };
    uint4 k[UNROLL], v[UNROLL];
    // rows of a round: those with keys in [from, to); what is not there is zero
    auto fetch_rows = [&](int round, const int (&page)[UNROLL], int from, int to) {
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
            const int key = key_of(round, u);
            if (key >= from && key < to && page[u] >= 0 && inside) {
                const long long at = (long long)page[u] * page_stride + (long long)((g << page_log2) + (key & (page_size - 1))) * head_dim + d;
                k[u] = load_row(k_pool + at);
                v[u] = load_row(v_pool + at + to_value);
            }
        }
    };
    auto clear_rows = [&]() {
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) k[u] = v[u] = make_uint4(0, 0, 0, 0);
    };
    int page[UNROLL];
    fetch_pages(first, page);
    clear_rows();
    fetch_rows(first, page, 0, first_new);
    const float sink_log2 = extras.sink ? extras.sink[h] * 1.4426950408889634f : -INFINITY;

    pdl_prologue();
    q = pdl_fresh(q);
    k_pool = pdl_fresh(k_pool);
    v_pool = pdl_fresh(v_pool);
    float query[8];
    {
        uint4 raw = make_uint4(0, 0, 0, 0);
        if (inside) raw = *reinterpret_cast<const uint4*>(q + (size_t)t * q_stride + h * head_dim + d);
        unpack(raw, query);
    }
    fetch_rows(first, page, first_new, p + 1);
    fetch_pages(first + SPAN, page);
    float m = -INFINITY, l = 0.f, acc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = 0.f;
    for (int round = first; round <= p; round += SPAN) {
        float s[UNROLL], top = m;
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
            float x[8];
            unpack(k[u], x);
            float dot = x[0] * query[0];
#pragma unroll
            for (int i = 1; i < 8; ++i) dot = fmaf(x[i], query[i], dot);
            s[u] = dot;
        }
#pragma unroll
        for (int o = 1; o < LANES; o <<= 1)
#pragma unroll
            for (int u = 0; u < UNROLL; ++u) s[u] += __shfl_xor_sync(0xffffffffu, s[u], o);
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
            s[u] = seen(key_of(round, u)) ? score_log2(s[u], scale_log2, extras) : -INFINITY;
            top = fmaxf(top, s[u]);
        }
#pragma unroll
        for (int o = LANES; o < 32; o <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
        const float base = top == -INFINITY ? 0.f : top, shrink = ex2(m - base);
        m = top;
        l *= shrink;
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] *= shrink;
        uint4 value[UNROLL];
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) value[u] = v[u];
        if (round + SPAN <= p) {                                  // the next round's rows go out, and the pages of the one behind it
            clear_rows();
            fetch_rows(round + SPAN, page, 0, p + 1);
            fetch_pages(round + 2 * SPAN, page);
        }
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
            const float w = ex2(s[u] - base);                     // (what is not seen: a weight and a row of zeros)
            float x[8];
            unpack(value[u], x);
            l += w;
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[i] = fmaf(w, x[i], acc[i]);
        }
    }
    // the lane groups of a warp have one maximum: their sums add up
#pragma unroll
    for (int o = LANES; o < 32; o <<= 1) {
        l += __shfl_xor_sync(0xffffffffu, l, o);
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], o);
    }
    if (group == 0) {
        *reinterpret_cast<float4*>(&acc_s[warp][d]) = make_float4(acc[0], acc[1], acc[2], acc[3]);
        *reinterpret_cast<float4*>(&acc_s[warp][d + 4]) = make_float4(acc[4], acc[5], acc[6], acc[7]);
        if (lane == 0) { m_s[warp] = m; l_s[warp] = l; }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < head_dim; i += WARPS * 32) {
        float big = sink_log2;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) big = fmaxf(big, m_s[w]);
        float total = extras.sink ? ex2(sink_log2 - big) : 0.f, sum = 0.f;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) {
            const float weight = m_s[w] == -INFINITY ? 0.f : ex2(m_s[w] - big);
            total = fmaf(l_s[w], weight, total);
            sum = fmaf(acc_s[w][i], weight, sum);
        }
        // (no weight at all: zero; a NaN in the total, from the query, a key or infinite scores, stays one)
        store_result(out, (size_t)t * out_stride + column * head_dim + i, total == 0.f ? sum * 0.f : sum / total, extras);
    }
}

template <int HD, int WARPS, int RESIDENT>
int launch(const void* q, int q_stride, void* out, int out_stride, const void* k_pool, const void* v_pool, long long page_stride,
           const int* token_item, const int* token_row, const int* positions, const int* block_table, int bt_stride, const int* q_start,
           const int* kv_len, int T, int n_heads, int n_kv_heads, int head_dim, int page_size, int window, float scale, float softcap,
           const float* sink, int all_values, int wide, cudaStream_t s) {
    return launch_pdl(attention_lanes_kernel<HD, WARPS, RESIDENT>, dim3(T, all_values ? n_heads * n_kv_heads : n_heads), dim3(WARPS * 32), 0, s,
                      (const __nv_bfloat16*)q, q_stride, (__nv_bfloat16*)out, out_stride, (const __nv_bfloat16*)k_pool,
                      (const __nv_bfloat16*)v_pool, page_stride, token_item, token_row, positions, block_table, bt_stride, q_start, kv_len,
                      n_heads, n_kv_heads, head_dim, 31 - __builtin_clz(page_size), window, scale * 1.4426950408889634f,
                      softmax_extras(scale, softcap, sink, wide), all_values);
}

}  // namespace lanes
}  // namespace ps

// Arguments as for ps_paged_attention_decode_ex; head sizes that are multiples of 8 up to 128, pages of a power of two; max_kv_len: the longest context that a token
// may have (for the choice of the warps only); warps 4, 8 or 16 (0: chosen here).
PS_EXPORT int ps_attention_lanes(const void* q, int q_stride, void* out, int out_stride, const void* k_pool, const void* v_pool,
                                 long long page_stride, const int* token_item, const int* token_row, const int* positions,
                                 const int* block_table, int bt_stride, const int* q_start, const int* kv_len, int T, int n_heads,
                                 int n_kv_heads, int head_dim, int page_size, int window, float scale, int max_kv_len, int warps, float softcap,
                                 const float* sink, int all_values, int wide, void* stream) {
    if (T <= 0) return PS_OK;
    if (n_heads <= 0 || n_kv_heads <= 0 || n_heads % n_kv_heads || (long long)n_heads * (all_values ? n_kv_heads : 1) > 65535) return PS_ERR_BAD_ARGUMENT;
    if (!q || !out || !k_pool || !v_pool || !token_item || !positions || !block_table) return PS_ERR_BAD_ARGUMENT;
    if (head_dim <= 0 || head_dim > 128 || head_dim % 8 || q_stride % 8 || page_stride % 8 || page_stride <= 0 || page_stride > 0x7fffffff)
        return PS_ERR_UNSUPPORTED;
    if (page_size <= 0 || (page_size & (page_size - 1)) || (((uintptr_t)q | (uintptr_t)k_pool | (uintptr_t)v_pool) & 15)) return PS_ERR_UNSUPPORTED;
    if (warps != 0 && warps != 4 && warps != 8 && warps != 16) return PS_ERR_BAD_ARGUMENT;
    // As many warps as leave all CTAs resident (heads of 64, us with 16 / 8 / 4 warps: 96 pairs of token and head, 300 keys each 5.3 / 5.6 / 7.5; 192
    // pairs 9.9 / 6.4 / 7.7; 768 pairs, 150 keys 20.0 / 14.8 / 8.5).  Where contexts may be long, one long one among short ones decides, which more
    // warps walk faster.
    // 297 to 444 pairs take 8 beyond 256 keys, three CTAs on an SM.  384 pairs, us with three / with two on an SM / 4 warps: 30 keys each 3.0 / - / 2.2,
    // 60 keys 3.4 / 5.0 / 3.7, 300 keys 8.5 / 12.7 / 9.1, all of 1,000 18.8 / 26.1 / 23.5; one of 500 among 60s 7.7 / 9.2 / 10.8, one of 1,000 among 60s
    // 12.1 / 14 / 19.0, a fourth of 1,000 among 100s 16.6 / 16.7 / 20.8.  Beyond 1,280 keys two: a third takes more from the long ones than it gives (a
    // fourth of 4,000 among 100s 57 / 45).
    // 445 to 592 pairs take 4 where contexts end at 1,280 (480 pairs, 60 keys 5.7 with 8 warps, 4.3 with 4, 300 keys 13.2 / 12.0, one of 1,000 among 60s 14 / 19.3).
    // Heads of 128, whose round has half as many keys, take 8 up to 592 pairs from short contexts on (384 pairs, 300 keys 12.6 / 17.8 / 15.1, one of 1,000
    // among 60s 21.4 / 22 / 33.0; 512 pairs, two on an SM, 300 keys 19.1, with 4 warps 21.5, one of 500 among 60s 14.7 / 19.0).
    const long long pairs = (long long)T * n_heads * (all_values ? n_kv_heads : 1);
    const bool three = pairs > 296 && pairs <= 444 && max_kv_len <= 1280;
    if (warps == 0) {
        const bool large = head_dim > 64;
        if (pairs <= 148) warps = 16;
        else if (pairs <= 296) warps = 8;
        else if (pairs <= 444) warps = large || max_kv_len > 256 ? 8 : 4;
        else warps = pairs <= 592 && (large || max_kv_len > 1280) ? 8 : 4;
    }
#define PS_LANES(HD, WARPS, RESIDENT)                                                                                                     \
    return ps::lanes::launch<HD, WARPS, RESIDENT>(q, q_stride, out, out_stride, k_pool, v_pool, page_stride, token_item, token_row, positions,      \
                                        block_table, bt_stride, q_start, kv_len, T, n_heads, n_kv_heads, head_dim, page_size, window,     \
                                        scale, softcap, sink, all_values, wide, (cudaStream_t)stream)
#define PS_LANES_HEADS(HD)                                                                                                                \
    if (warps == 16) PS_LANES(HD, 16, 1);                                                                                                 \
    if (warps == 8 && three) PS_LANES(HD, 8, 3);                                                                                          \
    if (warps == 8) PS_LANES(HD, 8, 2);                                                                                                   \
    PS_LANES(HD, 4, 6)
    if (head_dim <= 64) { PS_LANES_HEADS(64); }
    PS_LANES_HEADS(128);
#undef PS_LANES_HEADS
#undef PS_LANES
}
