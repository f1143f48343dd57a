// Causal attention of prompt portions over the paged cache in float32 on tcgen05, to float32 accuracy, for head sizes of 36 to 64 (multiples
// of 4; smaller than 64 are filled up with zeros).  Cache layout, masks, cap, sink and all_values as in attention_f32.cu, whose kernels take
// the other sizes and the single tokens.
//
// Queries, keys, values and weights are cut into three bfloat16 pieces each, and six of the nine products of two numbers'
// pieces are formed, the small ones first, as in gemm_f32_tc.cu (which says what the terms left out and the sums that tcgen05 cuts off amount to).
// One CTA per (128 queries of an entry, head), key tiles of 128 aligned to absolute positions:
//
//   warps 0..15  bring keys and values in (cp.async through the block table, each thread its own pieces of rows), cut them into pieces in
//                shared memory, and are four threads to a query row: softmax over 32 keys each in float32 (expf, tanhf), weights as pieces into
//                tensor memory, 16 columns of the result each in registers
//   warp 16      issues per tile S = Q K^T (24 MMAs of 128 x 128 x 16, Q's pieces in tensor memory) and P V (48 of 128 x 64 x 16)
//
// An accumulator takes one tile's values only (128 keys); tiles are added up in registers with rounding.  While P V of a tile runs, the next
// tile's keys and values are cut into pieces; its scores are queued behind.
//
// Infinities and NaNs: a value that is not finite counts as zero in the product (0 * infinity would reach rows that do not see it), and a row
// that sees one, or whose results are not finite or below 2^-80, is computed again at the end, term by term.
//
// The order of a row's sums depends on its position alone (reference: src/model/paged_attention.py:262-295).
//
// What bounds a tile: the chain of softmax (the workers), P V and the next S (72 MMAs, 74 clocks and more each), which follow one another; a CTA
// fills an SM, so only cutting into pieces overlaps.  In the last tile the products stop at the last key (in steps of 16), and a warp whose rows
// see none of its 32 keys forms no weights (16 tokens 10.4 -> 6.3 us, 4 x 64 12.6 -> 9.9, 5 x 128 14.7 -> 13.8).  Us, multiply-adds (as
// attention_f32.cu's, for heads of 64) / here, 12 heads of 64: 2 x 1,024 tokens 187 / 51, 5 x 128 18.4 / 13.8, 8 x 20 tokens behind 280
// 39.5 / 20.4, 2 x 16 behind 984 116 / 48, 16 tokens 9.8 / 6.3, 64 10.5 / 9.6, 4 x 64 10.9 / 9.9.  Error against 64 bits: 2 x 16 behind 984
// 6.0e-7 / 2.7e-7, 5 x 128 1.6e-7 / 1.4e-7.
#include <type_traits>

#include "f32_pieces.cuh"

namespace ps {
namespace f32tc {

constexpr int BQ = 128, BKEY = 128, HD = 64;
constexpr int WORKERS = 512, THREADS = WORKERS + 32;
constexpr int PLANE = BKEY * HD * 2, OPS_BYTES = 3 * PLANE;      // pieces of a tile of keys or of values
constexpr int RAW_BYTES = BKEY * HD * 4;
constexpr int K_OPS = 0, V_OPS = OPS_BYTES, K_RAW = 3 * OPS_BYTES, V_RAW = K_RAW + RAW_BYTES, EXCHANGE = V_RAW + RAW_BYTES;
constexpr int EXCHANGE_BYTES = 2 * 4 * BQ * 4;                   // [2][4 threads of a row][128 rows] floats
constexpr size_t SMEM = (size_t)EXCHANGE + EXCHANGE_BYTES + 128 /*barriers*/ + 1024 /*alignment*/;
constexpr int TMEM_COLS = 512, S_COL = 0, O_COL = 128, Q_COL = 192, P_COL = 288;       // Q: 3 x 32 columns, P: 3 x 64
static_assert(P_COL + 3 * 64 <= TMEM_COLS && SMEM <= 227 * 1024, "they fit");
constexpr float LARGEST = 3.402823466e38f;

struct Call {
    const float *q, *k_pool, *v_pool, *sink;
    float* out;
    long long page_stride, to_value;                             // to_value: from a key's place in its pool to its value's in the other
    const int* bt;
    int q_stride, out_stride, head_dim, shift, g;
    float scale, softcap;
};

// position -> offset of its row (of head g) in the pool, or -1 where the request has no page there; pages are 1 << shift long
__device__ __forceinline__ long long row_offset(const int* bt, int key, int shift, long long page_stride, int g, int head_dim) {
    const int page = bt[key >> shift];
    return page < 0 ? -1 : (long long)page * page_stride + (long long)(((g << shift) + (key & ((1 << shift) - 1))) * head_dim);
}
__device__ __forceinline__ void copy16(void* dst, const float* src, bool ok) {         // not ok: zeros
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(ok ? 16 : 0) : "memory");
}
__device__ __forceinline__ float capped(float score, float softcap) {
    return softcap > 0.f ? softcap * tanhf(score / softcap) : score;
}
__device__ __forceinline__ bool finite(float v) { return fabsf(v) <= LARGEST; }

// columns [d0, d0 + 16) of a row of the result, term by term: the query at `q` sees the keys low .. pos
__device__ __noinline__ void plain_row(const Call& c, const float* q, float* out, int low, int pos, int d0, const float* sink) {
    auto score = [&](int key) {
        const long long at = row_offset(c.bt, key, c.shift, c.page_stride, c.g, c.head_dim);
        float dot = 0.f;
        for (int d = 0; d < c.head_dim && at >= 0; ++d) dot = fmaf(q[d], c.k_pool[at + d], dot);
        return capped(dot * c.scale, c.softcap);
    };
    float top = sink ? *sink : -INFINITY;
#pragma unroll 1
    for (int key = low; key <= pos; ++key) top = fmaxf(top, score(key));
    const float base = top == -INFINITY ? 0.f : top;
    float total = sink ? expf(*sink - base) : 0.f, sum[16];
#pragma unroll
    for (int d = 0; d < 16; ++d) sum[d] = 0.f;
#pragma unroll 1
    for (int key = low; key <= pos; ++key) {
        const float p = expf(score(key) - base);
        const long long at = row_offset(c.bt, key, c.shift, c.page_stride, c.g, c.head_dim);
        total += p;
#pragma unroll
        for (int d = 0; d < 16; ++d)
            if (d0 + d < c.head_dim && at >= 0) sum[d] = fmaf(p, c.v_pool[at + c.to_value + d0 + d], sum[d]);
    }
#pragma unroll
    for (int d = 0; d < 16; ++d)
        if (d0 + d < c.head_dim) out[d0 + d] = sum[d] / total;
}
// whether the row sees a value that is not finite in these columns
__device__ __noinline__ bool sees_infinity(const Call& c, int low, int pos, int d0) {
    bool bad = false;
#pragma unroll 1
    for (int key = low; key <= pos; ++key) {
        const long long at = row_offset(c.bt, key, c.shift, c.page_stride, c.g, c.head_dim);
        for (int d = d0; d < min(d0 + 16, c.head_dim) && at >= 0; ++d) bad |= !finite(c.v_pool[at + c.to_value + d]);
    }
    return bad;
}

__global__ void __launch_bounds__(THREADS, 1)
prompt_attention_f32_tc_kernel(const float* __restrict__ q, int q_stride, float* __restrict__ out, int out_stride,
                               const float* __restrict__ k_pool, const float* __restrict__ v_pool, long long page_stride,
                               const int* __restrict__ q_start, const int* __restrict__ kv_len, const int* __restrict__ block_table,
                               int bt_stride, const int* __restrict__ item_row, int first_item, int n_items, int n_heads, int n_kv_heads,
                               int head_dim, int page_size, int window, float scale, float softcap, const float* __restrict__ sink,
                               int all_values, int* __restrict__ status) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* base = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    float* exchange = reinterpret_cast<float*>(base + EXCHANGE);
    uint64_t* bars = reinterpret_cast<uint64_t*>(base + EXCHANGE + EXCHANGE_BYTES);
    uint64_t *k_ready = bars, *s_full = bars + 1, *p_ready = bars + 2, *o_full = bars + 3;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 4);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    volatile int* infinities = abort_flag + 1;                   // a value of the CTA's tiles is not finite

    pdl_prologue();
    q = pdl_fresh(q);
    k_pool = pdl_fresh(k_pool);
    v_pool = pdl_fresh(v_pool);
    // which (item, query block) is this CTA? late blocks see most keys: they come first
    int block = blockIdx.y, item = -1, qb = 0;
    for (int i = first_item; i < first_item + n_items; ++i) {
        int blocks = (q_start[i + 1] - q_start[i] + BQ - 1) / BQ;
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
    const int first = lo / BKEY, last = hi / BKEY;
    const int* bt = block_table + (size_t)(item_row ? item_row[item] : item) * bt_stride;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

    if (tid == 0) {
        *abort_flag = 0;
        *infinities = 0;
        mbar_init(k_ready, WORKERS / 32);
        mbar_init(s_full, 1);
        mbar_init(p_ready, WORKERS / 32);
        mbar_init(o_full, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == WORKERS / 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(tmem_slot)), "r"((uint32_t)TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == WORKERS / 32) {
        if (elect_one()) {
            // D = f32, A = B = bf16, M = 128; keys K-major, N = 128 or what is left of the last tile; values MN-major (bit 16), N = 64
            constexpr uint32_t kind = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BQ >> 4) << 24);
            constexpr uint32_t idesc_o = kind | (1u << 16) | ((uint32_t)(HD >> 3) << 17);
            // the six products, the small ones first: pieces of the first and of the second operand
            constexpr int piece_a[6] = {2, 1, 0, 1, 0, 0}, piece_b[6] = {0, 1, 2, 0, 1, 0};
            const uint64_t keys = umma_desc(smem_u32(base + K_OPS));
            for (int it = 0; it <= last - first; ++it) {
                if (!mbar_wait(k_ready, it & 1, abort_flag)) { atomicExch(status, 61); break; }
                tc_fence_after();
                // 16-key steps that anyone sees: the others' scores are masked whatever they are, and their weights and values are zeros
                const int steps = (min(BKEY, hi - (first + it) * BKEY + 1) + 15) / 16;
                const uint32_t idesc_s = kind | ((uint32_t)(2 * steps) << 17);
#pragma unroll
                for (int product = 0; product < 6; ++product)
#pragma unroll
                    for (int k = 0; k < HD / 16; ++k)
                        umma_ts(tmem + S_COL, tmem + Q_COL + 32 * piece_a[product] + 8 * k, keys + piece_b[product] * (PLANE >> 4) + 2 * k, idesc_s,
                                (product | k) ? 1u : 0u);
                umma_commit(s_full);
                if (!mbar_wait(p_ready, it & 1, abort_flag)) { atomicExch(status, 62); break; }
                tc_fence_after();
                const uint64_t values = umma_desc(smem_u32(base + V_OPS + (it & 1) * OPS_BYTES));
                auto step = [&](int product, int k) {            // 16 keys: 2,048 bytes of values
                    umma_ts(tmem + O_COL, tmem + P_COL + 64 * piece_a[product] + 8 * k, values + piece_b[product] * (PLANE >> 4) + 128 * k, idesc_o,
                            (product | k) ? 1u : 0u);
                };
                if (steps == BKEY / 16) {
#pragma unroll
                    for (int product = 0; product < 6; ++product)
#pragma unroll
                        for (int k = 0; k < BKEY / 16; ++k) step(product, k);
                } else {
#pragma unroll
                    for (int product = 0; product < 6; ++product)
#pragma unroll 1
                        for (int k = 0; k < steps; ++k) step(product, k);
                }
                umma_commit(o_full);
            }
        }
        __syncwarp();
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)TMEM_COLS) : "memory");
        return;
    }

    const int quarter = warp & 3, team = warp >> 2;              // tensor memory lanes 32 quarter.., keys 32 team.. and columns 16 team..
    const int row = 32 * quarter + lane, pos = pos0 + row;
    const int low = first_visible_key(pos, window);
    const uint32_t tmem_row = tmem + ((uint32_t)(32 * quarter) << 16);
    const int shift = 31 - __clz(page_size);
    // A wait that runs out is noted and the work goes on: nobody leaves a barrier of the workers, and no later wait lasts.
    bool ok = true;
    auto await = [&](uint64_t* bar, int phase, int code) {
        if (!mbar_wait(bar, phase, abort_flag)) {
            ok = false;
            if (lane == 0) atomicExch(status, code);
        }
        tc_fence_after();
    };
    // Of a tile's rows a thread has the 8 columns from 8 (tid & 7) of rows tid / 8 and 64 + tid / 8, in slots of its own: what it copies
    // in it alone reads, and no barrier stands between.
    auto bring = [&](int tile, const float* pool, long long beyond, int raw) {
        if (tile <= last) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int key = tile * BKEY + 64 * i + (tid >> 3), d = 8 * (tid & 7);
                const long long at = key >= lo && key <= hi && d < head_dim ? row_offset(bt, key, shift, page_stride, g, head_dim) : -1;
                const float* from = at >= 0 ? pool + at + beyond + d : pool;
                copy16(base + raw + ((2 * i) * WORKERS + tid) * 16, from, at >= 0);
                copy16(base + raw + ((2 * i + 1) * WORKERS + tid) * 16, at >= 0 && d + 4 < head_dim ? from + 4 : pool, at >= 0 && d + 4 < head_dim);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto cut = [&](int tile, int raw, unsigned char* to, bool values) {          // the older of the two groups on their way has come
        asm volatile("cp.async.wait_group 1;" ::: "memory");
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            if (tile * BKEY + 64 * i > hi) break;                // (no step of the products reads these rows)
            float4 v[2];
#pragma unroll
            for (int half = 0; half < 2; ++half) v[half] = *reinterpret_cast<const float4*>(base + raw + ((2 * i + half) * WORKERS + tid) * 16);
            if (values) {
                float most = 0.f, *x = &v[0].x;
#pragma unroll
                for (int j = 0; j < 8; ++j) most = __uint_as_float(max(__float_as_uint(most), __float_as_uint(x[j]) & 0x7fffffffu));
                if (!finite(most)) {
#pragma unroll
                    for (int j = 0; j < 8; ++j) x[j] = finite(x[j]) ? x[j] : 0.f;
                    *infinities = 1;
                }
            }
            uint32_t piece[3][4];
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                split(v[half].x, v[half].y, piece[0][2 * half], piece[1][2 * half], piece[2][2 * half]);
                split(v[half].z, v[half].w, piece[0][2 * half + 1], piece[1][2 * half + 1], piece[2][2 * half + 1]);
            }
            const int r = 64 * i + (tid >> 3);
#pragma unroll
            for (int p = 0; p < 3; ++p)
                *reinterpret_cast<uint4*>(to + p * PLANE + r * 128 + (((tid & 7) ^ (r & 7)) << 4)) =
                    make_uint4(piece[p][0], piece[p][1], piece[p][2], piece[p][3]);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    };
    auto arrive = [&](uint64_t* bar) {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar);
    };

    bring(first, k_pool, 0, K_RAW);
    bring(first, v_pool, to_value, V_RAW);
    {
        // the row's query, 16 numbers of it, as pieces into tensor memory
        uint32_t piece[3][8];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int d = 16 * team + 4 * i;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (row < rows && d < head_dim) v = *reinterpret_cast<const float4*>(q + (size_t)(tok0 + row) * q_stride + h * head_dim + d);
            split(v.x, v.y, piece[0][2 * i], piece[1][2 * i], piece[2][2 * i]);
            split(v.z, v.w, piece[0][2 * i + 1], piece[1][2 * i + 1], piece[2][2 * i + 1]);
        }
#pragma unroll
        for (int p = 0; p < 3; ++p) tmem_st8(tmem_row + Q_COL + 32 * p + 8 * team, piece[p]);
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    }
    cut(first, K_RAW, base + K_OPS, false);
    arrive(k_ready);
    bring(first + 1, k_pool, 0, K_RAW);
    cut(first, V_RAW, base + V_OPS, true);
    bring(first + 1, v_pool, to_value, V_RAW);

    float o[16], m = -INFINITY, l = 0.f;                         // l: of this thread's keys
#pragma unroll
    for (int d = 0; d < 16; ++d) o[d] = 0.f;
    auto drain = [&](int it) {                                   // the product of tile `it` joins the row's sums
        await(o_full, it & 1, 64);
        uint32_t r[16];
        tmem_ld16(tmem_row + O_COL + 16 * team, r);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int d = 0; d < 16; ++d) o[d] += __uint_as_float(r[d]);
    };
    // A tile.  LAST: the last one, of whose keys a warp's rows may see none (a team's keys begin beyond the diagonal or the end): it forms no
    // weights then and stores zeros.  (Every rounding is written out, so that both forms have the same bits.)
    auto work = [&](int tile, auto last_tile) {
        constexpr bool LAST = decltype(last_tile)::value;
        const int it = tile - first;
        if (it > 0) drain(it - 1);
        await(s_full, it & 1, 63);
        float s[32], top = -INFINITY;
        const int key0 = tile * BKEY + 32 * team;
        const bool seen = !LAST || key0 <= min(pos0 + 32 * quarter + 31, hi);
        if (seen) {
            uint32_t r[16];
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                tmem_ld16(tmem_row + S_COL + 32 * team + 16 * half, r);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int j = 0; j < 16; ++j) s[16 * half + j] = __fmul_rn(__uint_as_float(r[j]), scale);
            }
            if (softcap > 0.f) {
#pragma unroll 4
                for (int j = 0; j < 32; ++j) s[j] = capped(s[j], softcap);
            }
            if (key0 + 31 > pos || key0 < low) {
#pragma unroll
                for (int j = 0; j < 32; ++j) s[j] = key0 + j <= pos && key0 + j >= low ? s[j] : -INFINITY;
            }
#pragma unroll
            for (int j = 0; j < 32; ++j) top = fmaxf(top, s[j]);
        }
        float* shared_top = exchange + (it & 1) * 4 * BQ + row;  // (two buffers: one barrier a tile is enough)
        shared_top[team * BQ] = top;
        asm volatile("bar.sync %0, 128;" ::"r"(2 + quarter) : "memory");
#pragma unroll
        for (int i = 0; i < 4; ++i) top = fmaxf(top, shared_top[i * BQ]);
        const float m_new = fmaxf(m, top);
        const float m_base = m_new == -INFINITY ? 0.f : m_new;   // a row that sees no key of this tile or before it
        const float shrink = expf(m - m_base);
        m = m_new;
        if (!seen) l = __fmul_rn(l, shrink);
#pragma unroll
        for (int d = 0; d < 16; ++d) o[d] = __fmul_rn(o[d], shrink);
        if (seen) {
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                uint32_t piece[3][8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const float even = expf(__fsub_rn(s[16 * half + 2 * j], m_base)), odd = expf(__fsub_rn(s[16 * half + 2 * j + 1], m_base));
                    l = half == 0 && j == 0 ? fmaf(l, shrink, even) : l + even;
                    l += odd;
                    split(even, odd, piece[0][j], piece[1][j], piece[2][j]);
                }
#pragma unroll
                for (int p = 0; p < 3; ++p) tmem_st8(tmem_row + P_COL + 64 * p + 16 * team + 8 * half, piece[p]);
            }
        } else if (key0 <= hi) {
            const uint32_t none[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
#pragma unroll 1
            for (int i = 0; i < 6; ++i) tmem_st8(tmem_row + P_COL + 64 * (i >> 1) + 16 * team + 8 * (i & 1), none);
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        arrive(p_ready);
        if constexpr (!LAST) {
            cut(tile + 1, K_RAW, base + K_OPS, false);
            arrive(k_ready);
            bring(tile + 2, k_pool, 0, K_RAW);
            cut(tile + 1, V_RAW, base + V_OPS + ((it + 1) & 1) * OPS_BYTES, true);
            bring(tile + 2, v_pool, to_value, V_RAW);
        }
    };
#pragma unroll 1
    for (int tile = first; tile < last; ++tile) work(tile, std::false_type());
    work(last, std::true_type());
    drain(last - first);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    // the row's sum is that of its four threads, in order; both buffers of the exchange are free behind the barrier
    asm volatile("bar.sync 1, %0;" ::"n"(WORKERS) : "memory");
    exchange[team * BQ + row] = l;
    asm volatile("bar.sync 1, %0;" ::"n"(WORKERS) : "memory");
    float total = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) total += exchange[i * BQ + row];
    if (ok && row < rows) {
        const float* sink_h = sink ? sink + h : nullptr;
        float scale_out = 1.f;
        if (sink_h) {
            const float big = fmaxf(m, *sink_h);
            scale_out = expf(m - big);
            total = total * scale_out + expf(*sink_h - big);
        }
        scale_out /= total;
        float* to = out + (size_t)(tok0 + row) * out_stride + column * head_dim;
        bool again = !finite(scale_out);
#pragma unroll
        for (int d = 0; d < 16; ++d) {
            o[d] *= scale_out;
            again |= doubtful(o[d]);
        }
        if (again || *infinities) {
            const Call call{q, k_pool, v_pool, sink_h, out, page_stride, to_value, bt, q_stride, out_stride, head_dim, shift, g, scale, softcap};
            if (again || sees_infinity(call, low, pos, 16 * team)) {
                plain_row(call, q + (size_t)(tok0 + row) * q_stride + h * head_dim, to, low, pos, 16 * team, sink_h);
                again = true;
            }
        }
        if (!again) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int d = 16 * team + 4 * i;
                if (d < head_dim) *reinterpret_cast<float4*>(to + d) = make_float4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
}

}  // namespace f32tc
}  // namespace ps

// As ps_prompt_attention_f32 (attention_f32.cu), for head sizes of 36 to 64; max_blocks >= the number of 128-query blocks that the items
// make up.  status: device int32 that a bounded wait sets when it runs out (must not be null).
PS_EXPORT int ps_prompt_attention_f32_tc(const float* q, int q_stride, float* out, int out_stride, const float* k_pool, const float* v_pool,
                                         long long page_stride, const int* q_start, const int* kv_len, const int* block_table, int bt_stride,
                                         const int* item_row, int first_item, int n_items, int max_blocks, int n_heads, int n_kv_heads,
                                         int head_dim, int page_size, int window, float scale, float softcap, const float* sink,
                                         int all_values, int* status, void* stream) {
    using namespace ps::f32tc;
    if (n_items <= 0 || max_blocks <= 0) return PS_OK;
    if (!status || n_heads <= 0 || n_kv_heads <= 0 || n_heads % n_kv_heads) return PS_ERR_BAD_ARGUMENT;
    if (head_dim <= 32 || head_dim > HD || head_dim % 4 || q_stride % 4 || out_stride % 4 || page_stride % 4) return PS_ERR_UNSUPPORTED;
    if (page_size <= 0 || page_size > 64 || (page_size & (page_size - 1)) || max_blocks > 65535) return PS_ERR_UNSUPPORTED;
    if (((uintptr_t)q | (uintptr_t)out | (uintptr_t)k_pool | (uintptr_t)v_pool) & 15) return PS_ERR_UNSUPPORTED;
    static size_t raised[ps::MAX_DEVICES] = {0};
    if (!ps::ensure_dynamic_smem((const void*)prompt_attention_f32_tc_kernel, SMEM, raised)) return PS_ERR_LAUNCH;
    return ps::launch_pdl(prompt_attention_f32_tc_kernel, dim3(all_values ? n_heads * n_kv_heads : n_heads, max_blocks), dim3(THREADS), SMEM,
                          (cudaStream_t)stream, q, q_stride, out, out_stride, k_pool, v_pool, page_stride, q_start, kv_len, block_table,
                          bt_stride, item_row, first_item, n_items, n_heads, n_kv_heads, head_dim, page_size, window, scale, softcap, sink,
                          all_values, status);
}
