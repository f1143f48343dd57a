// float32 products of many rows on the tensor cores, to float32 accuracy: out[M,N] = epilogue(A[M,K] W[N,K]^T + bias).
//
// A float32 number is the sum of three bfloat16 numbers (24 bits of mantissa: 8 + 8 + 8), a = a0 + a1 + a2, and a product
// of two is a0 b0 + (a0 b1 + a1 b0) + (a0 b2 + a1 b1 + a2 b0) but for terms below 2^-22 of it, of either sign (f32_pieces.cuh).  tcgen05.mma forms the six
// bfloat16 products exactly and adds them up in float32.  It cuts its sums off instead of rounding them (64 x 64 x 16 terms after
// one another: 1 + 0.75 * 2^-23 gives 1), an error that grows with every MMA on one accumulator: over K = 768 of normal numbers 7.4e-7 of the
// result's size, where float32 additions one after the other are off by 2.1e-7.  So an accumulator takes 64 k's only, the small
// terms ahead of the large ones (what is cut off is then a part of a small sum), and the blocks are added in registers with rounding.
//
//   warp 0       TMA: boxes of 32 k's x 128 rows of A and of W (float32, 128-byte swizzle) into a ring of slots
//   warps 4..19  turn a stage of 64 k's (two slots, half of the warps each) into pieces, A's into tensor memory (as the MMA's first operand it
//                costs no shared memory bandwidth), W's into shared memory; then they add the accumulator of the stage before to their sums
//   warp 1       issues 24 MMAs of 128 x 128 x 16 a stage into two accumulators in turn
//
// K is cut into `parts` (by K alone) whose sums are added in order.  A cluster of so many CTAs forms one part each and adds them
// through distributed shared memory, or one of half as many CTAs two each, or one CTA forms all of them one after the other, whichever is
// modelled to be faster for the tiles at hand.  All give the same bits (a cluster's later CTAs keep their two parts' sums apart), so that a row's
// result does not depend on the rows beside it.
//
// A stage takes 1.44 us, its MMAs 0.93 (74 clocks each).  Bound by shared memory: a stage brings 64 KB in, reads 64 KB, writes 48 KB of
// pieces of W and the MMAs read 96 KB, 2,130 of about 2,700 clocks at 128 bytes each; around the stages a CTA takes 7 us (first operands 0.6,
// first pieces 1.1, the last MMAs and sums 1.8, results through shared memory to global 3).  Us, float32 multiply-adds / here: 2,048 x 2,304 x 768
// 152 / 51, 2,048 x 768 x 3,072 259 / 80 (121 TFLOP/s), 384 x 2,304 x 768 41 / 17, 651 x 1,024 x 1,024 53 / 20, 17 x 768 x 768 10.4 / 9.3.  With stages
// of 32 k's (half as much work between barriers, twice the additions of accumulators) 70 / 112 in the first two.
//
// Infinities and NaNs: the pieces of an infinity are an infinity and NaNs.  A result that is not finite, or below 2^-80, is computed again, term by
// term, from the operands themselves.
//
// Stands where the reference has cuBLAS nn.Linear calls in float32 (src/model/paged_decoder.py:49-50, 178-179, 295-299).
#include "f32_pieces.cuh"

namespace ps {
namespace f32tc {

constexpr int BM = 128, BN = 128, BK = 64;
constexpr int SLOT = 32;                                         // k's of a slot of float32 operands: 128 bytes
constexpr int RAW = 4, OPS = 2;                                  // slots of float32 operands, stages of pieces
constexpr int SPLITTERS = 16;                                    // warps that form pieces and sums
constexpr int THREADS = 128 + 32 * SPLITTERS;
// Registers: 96 a thread at launch (five warps a scheduler), of which the first warps, which only issue, hand most to the splitters.  (The
// compiler keeps to the 96 all the same and spills 17 words.)
constexpr int REGS = 96, FEW_REGS = 32, MANY_REGS = 112;
static_assert(128 * FEW_REGS + 32 * SPLITTERS * MANY_REGS <= THREADS * REGS, "no more than the block was launched with");
constexpr int OPERAND = BM * SLOT * 4, RAW_BYTES = 2 * OPERAND;
constexpr int PLANE = BN * BK * 2, OPS_BYTES = 3 * PLANE;
constexpr int PITCH = BN + 4;                                    // floats of a row of results in shared memory
constexpr size_t SMEM = (size_t)RAW * RAW_BYTES + OPS * OPS_BYTES + 1024 /*alignment*/ + 256 /*barriers*/;
constexpr int RESULTS = BM * PITCH;
static_assert(2 * RESULTS * 4 <= RAW * RAW_BYTES + OPS * OPS_BYTES, "results lie where the operands were");
constexpr float FIXED = 7.f, PER_SPLIT = .3f, PER_STAGE = 1.44f;  // microseconds of a CTA, measured
constexpr int TMEM_COLS = 512, TMEM_A = 256;                     // accumulators at columns 0 and 128, pieces of A from 256, 128 a stage

// the doubtful ones among the sums of up to `count` of four neighbouring columns again, one product after the other
__device__ __noinline__ float4 plain_dots(float4 sums, const float* a, const float* w, int ldw, int K, int count) {
    float v[4] = {sums.x, sums.y, sums.z, sums.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        if (j >= count || !doubtful(v[j])) continue;
        v[j] = 0.f;
#pragma unroll 1
        for (int k = 0; k < K; ++k) v[j] = fmaf(a[k], w[(size_t)j * ldw + k], v[j]);
    }
    return make_float4(v[0], v[1], v[2], v[3]);
}

// grid (column tiles * splits, row tiles), clusters of `splits` CTAs in x; splits is 1, parts / 2 or parts
__global__ void __launch_bounds__(THREADS, 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, const float* __restrict__ A,
                   int lda, const float* __restrict__ W, int ldw, const float* __restrict__ bias, float* __restrict__ out, int ldo,
                   int M, int N, int K, int act, int accumulate, int parts, int splits, int* __restrict__ status) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* raw = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* ops = raw + RAW * RAW_BYTES;
    uint64_t* bars = reinterpret_cast<uint64_t*>(ops + OPS * OPS_BYTES);
    uint64_t* raw_full = bars;                     // [RAW]  TMA -> splitters
    uint64_t* raw_empty = raw_full + RAW;          // [RAW]  splitters -> TMA
    uint64_t* ops_full = raw_empty + RAW;          // [OPS]  splitters -> MMA
    uint64_t* ops_empty = ops_full + OPS;          // [OPS]  MMA -> splitters
    uint64_t* acc_full = ops_empty + OPS;          // [2]    MMA -> splitters
    uint64_t* acc_empty = acc_full + 2;            // [2]    splitters -> MMA
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tile_n = blockIdx.x / splits, rank = blockIdx.x - tile_n * splits;
    const int m0 = blockIdx.y * BM, n0 = tile_n * BN;
    const int blocks = (K + BK - 1) / BK;
    auto part_start = [&](int part) { return (int)((long long)blocks * part / parts); };
    const int first_part = rank * (parts / splits), last_part = first_part + parts / splits;
    const bool two_sums = splits > 1 && splits < parts && rank > 0;    // this CTA's two parts are not added up here
    const int kb0 = part_start(first_part), stages = part_start(last_part) - kb0;

    __shared__ __align__(16) float columns[BN];    // the tile's bias or factors
    if (threadIdx.x == 0) {
        *abort_flag = 0;
        for (int s = 0; s < RAW; ++s) { mbar_init(&raw_full[s], 1); mbar_init(&raw_empty[s], SPLITTERS / 2); }
        for (int s = 0; s < OPS; ++s) { mbar_init(&ops_full[s], SPLITTERS); mbar_init(&ops_empty[s], 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], SPLITTERS); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(tmem_slot)), "r"((uint32_t)TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    // all of the block (of the cluster) are there
    auto meet = [&]() {
        if (splits > 1) cluster_sync_all();
        else asm volatile("bar.sync 0;" ::: "memory");
    };

    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(FEW_REGS));
        if (warp == 0) {
            if (elect_one()) {
                // the first stages' weights go out before the wait, if nothing of this step makes them
                const int slots = stages * (BK / SLOT), early = (accumulate & PS_WEIGHTS_READY) ? min(RAW, slots) : 0;
                for (int it = 0; it < early; ++it) {
                    mbar_expect_tx(&raw_full[it], RAW_BYTES);
                    tma_load_2d(raw + it * RAW_BYTES + OPERAND, &map_w, kb0 * BK + it * SLOT, n0, &raw_full[it]);
                }
                pdl_prologue();
                for (int it = 0; it < slots; ++it) {
                    const int s = it % RAW, x = kb0 * BK + it * SLOT;
                    unsigned char* to = raw + s * RAW_BYTES;
                    if (it >= early) {
                        if (!mbar_wait(&raw_empty[s], ((it / RAW) & 1) ^ 1, abort_flag)) { atomicExch(status, 51); break; }
                        mbar_expect_tx(&raw_full[s], RAW_BYTES);
                        tma_load_2d(to + OPERAND, &map_w, x, n0, &raw_full[s]);
                    }
                    tma_load_2d(to, &map_a, x, m0, &raw_full[s]);
                }
            } else {
                pdl_prologue();
            }
            __syncwarp();
        } else if (warp == 1) {
            pdl_prologue();
            if (elect_one()) {
                // D = f32, A = B = bf16, both K-major, N = 128, M = 128
                constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
                // pieces of A and of W of the six products, the small ones first
                constexpr int piece_a[6] = {2, 1, 0, 1, 0, 0}, piece_w[6] = {0, 1, 2, 0, 1, 0};
                for (int it = 0; it < stages; ++it) {
                    const int s = it % OPS, buf = it & 1;
                    if (!mbar_wait(&acc_empty[buf], ((it >> 1) & 1) ^ 1, abort_flag)) { atomicExch(status, 52); break; }
                    if (!mbar_wait(&ops_full[s], (it / OPS) & 1, abort_flag)) { atomicExch(status, 53); break; }
                    tc_fence_after();
                    const uint32_t d = tmem + buf * BN, a = tmem + TMEM_A + 128 * s;
                    const uint64_t w = umma_desc(smem_u32(ops + s * OPS_BYTES));
#pragma unroll
                    for (int product = 0; product < 6; ++product)
#pragma unroll
                        for (int k = 0; k < BK / 16; ++k)      // 16 bf16: 8 columns of tensor memory, 32 bytes = 2 units of the address field
                            umma_ts(d, a + 32 * piece_a[product] + 8 * k, w + piece_w[product] * (PLANE >> 4) + 2 * k, idesc, (product | k) ? 1u : 0u);
                    umma_commit(&ops_empty[s]);
                    umma_commit(&acc_full[buf]);
                }
            }
            __syncwarp();
        } else {
            pdl_prologue();
        }
        tc_fence_before();
        meet();
        if (warp == 1) {
            tc_fence_after();
            asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)TMEM_COLS) : "memory");
        }
        if (splits > 1) cluster_sync_all();
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(MANY_REGS));
        pdl_prologue();
        const int quarter = warp & 3, team = (warp - 4) >> 2;          // TMEM lanes 32 quarter.. (rows), k's 8 team.. and columns 32 team..
        const int row = 32 * quarter + lane;
        // (behind the wait: the kernel in front may have made the vector; it is there long before the first operands are pieces)
        if (team == 0) columns[row] = bias && n0 + row < N ? pdl_fresh(bias)[n0 + row] : 0.f;
        const uint32_t tmem_row = tmem + ((uint32_t)(32 * quarter) << 16);
        const int half = team >> 1, sub = team & 1;                    // slot of a stage, 16 k's of the slot
        unsigned long long sum[16], total[16];                         // pairs of columns: of the part, of the parts before it
#pragma unroll
        for (int j = 0; j < 16; ++j) sum[j] = total[j] = 0ull;
        int part = first_part, part_end = part_start(first_part + 1) - kb0;
        bool ok = true;
        auto drain = [&](int it) {                                     // the accumulator of stage `it` joins the sums
            const int buf = it & 1;
            if (!mbar_wait(&acc_full[buf], (it >> 1) & 1, abort_flag)) { ok = false; if (lane == 0) atomicExch(status, 54); return; }
            tc_fence_after();
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                uint32_t r[16];
                tmem_ld16(tmem_row + buf * BN + 32 * team + 16 * half, r);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (half == 1) {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&acc_empty[buf]);
                }
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    unsigned long long& to = sum[8 * half + j];
                    to = pair_add(to, pair_of(__uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1])));
                }
            }
            if (it + 1 == part_end && !(two_sums && part > first_part)) {
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    total[j] = pair_add(total[j], sum[j]);
                    sum[j] = 0ull;
                }
                ++part;
                part_end = part < last_part ? part_start(part + 1) - kb0 : -1;
            }
        };
        for (int it = 0; it < stages && ok; ++it) {
            const int o = it % OPS;
            const int slot = it * (BK / SLOT) + half, s = slot % RAW;
            if (!mbar_wait(&raw_full[s], (slot / RAW) & 1, abort_flag)) { ok = false; if (lane == 0) atomicExch(status, 55); break; }
            const unsigned char* from = raw + s * RAW_BYTES + row * 128;
            float4 v[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] = *reinterpret_cast<const float4*>(from + (((4 * sub + i) ^ (row & 7)) << 4));
            if (!mbar_wait(&ops_empty[o], ((it / OPS) & 1) ^ 1, abort_flag)) { ok = false; if (lane == 0) atomicExch(status, 56); break; }
            tc_fence_after();
            uint32_t piece[3][8];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                split(v[i].x, v[i].y, piece[0][2 * i], piece[1][2 * i], piece[2][2 * i]);
                split(v[i].z, v[i].w, piece[0][2 * i + 1], piece[1][2 * i + 1], piece[2][2 * i + 1]);
            }
#pragma unroll
            for (int q = 0; q < 3; ++q) tmem_st8(tmem_row + TMEM_A + 128 * o + 32 * q + 16 * half + 8 * sub, piece[q]);
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] = *reinterpret_cast<const float4*>(from + OPERAND + (((4 * sub + i) ^ (row & 7)) << 4));
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                split(v[i].x, v[i].y, piece[0][2 * i], piece[1][2 * i], piece[2][2 * i]);
                split(v[i].z, v[i].w, piece[0][2 * i + 1], piece[1][2 * i + 1], piece[2][2 * i + 1]);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&raw_empty[s]);
            unsigned char* to = ops + o * OPS_BYTES + row * 128;
#pragma unroll
            for (int q = 0; q < 3; ++q)
#pragma unroll
                for (int i = 0; i < 2; ++i)
                    *reinterpret_cast<uint4*>(to + q * PLANE + (((4 * half + 2 * sub + i) ^ (row & 7)) << 4)) =
                        make_uint4(piece[q][4 * i], piece[q][4 * i + 1], piece[q][4 * i + 2], piece[q][4 * i + 3]);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&ops_full[o]);
            if (it >= 1) drain(it - 1);
        }
        if (ok) drain(stages - 1);
        // every stage has been brought in and read: its memory takes the results
        asm volatile("bar.sync 1, %0;" ::"n"(32 * SPLITTERS) : "memory");
        float* staged = reinterpret_cast<float*>(raw) + row * PITCH + 32 * team;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            float4 v;
            pair_split(total[2 * j], v.x, v.y);
            pair_split(total[2 * j + 1], v.z, v.w);
            *reinterpret_cast<float4*>(staged + 4 * j) = v;
            if (two_sums) {
                pair_split(sum[2 * j], v.x, v.y);
                pair_split(sum[2 * j + 1], v.z, v.w);
                *reinterpret_cast<float4*>(staged + RESULTS + 4 * j) = v;
            }
        }
        tc_fence_before();
        meet();

    // ---- the rows rank, rank + splits, ... of the tile: the parts in order, the epilogue, four columns a lane
        const float* results = reinterpret_cast<const float*>(raw) + 4 * lane;
        const int n = n0 + 4 * lane;
        const bool vector_out = N % 4 == 0 && ldo % 4 == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0;
        const float4 column = *reinterpret_cast<const float4*>(columns + 4 * lane);
        auto row_of = [&](int i) { return rank + splits * (warp - 4 + SPLITTERS * i); };
        auto here = [&](int r) { return r < BM && m0 + r < M && n < N; };
        auto fetch = [&](int r) {                                      // what a result is added to
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (!(accumulate & PS_ACCUMULATE) || !here(r)) return v;
            const float* at = out + (size_t)(m0 + r) * ldo + n;
            if (vector_out) return *reinterpret_cast<const float4*>(at);
            v.x = at[0];
            if (n + 1 < N) v.y = at[1];
            if (n + 2 < N) v.z = at[2];
            if (n + 3 < N) v.w = at[3];
            return v;
        };
        auto finish = [&](int r, const float4& before) {
            if (!here(r)) return;
            float4 v = before, sums = make_float4(0.f, 0.f, 0.f, 0.f);
            auto add = [&](const float4& p) { sums.x += p.x; sums.y += p.y; sums.z += p.z; sums.w += p.w; };
            if (splits == 1) {
                add(*reinterpret_cast<const float4*>(results + r * PITCH));
            } else {
                for (int q = 0; q < splits; ++q) {
                    add(ld_cluster_f32x4(results + r * PITCH, q));
                    if (q > 0 && splits < parts) add(ld_cluster_f32x4(results + RESULTS + r * PITCH, q));
                }
            }
            if (doubtful(sums.x) || doubtful(sums.y) || doubtful(sums.z) || doubtful(sums.w))
                sums = plain_dots(sums, pdl_fresh(A) + (size_t)(m0 + r) * lda, W + (size_t)n * ldw, ldw, K, N - n);
            if (bias && (accumulate & PS_COLUMN_FACTOR)) { sums.x *= column.x; sums.y *= column.y; sums.z *= column.z; sums.w *= column.w; }
            else if (bias) { sums.x += column.x; sums.y += column.y; sums.z += column.z; sums.w += column.w; }
            if (act != PS_ACT_NONE) {
                sums.x = apply_act(sums.x, act); sums.y = apply_act(sums.y, act);
                sums.z = apply_act(sums.z, act); sums.w = apply_act(sums.w, act);
            }
            v.x += sums.x; v.y += sums.y; v.z += sums.z; v.w += sums.w;
            float* at = out + (size_t)(m0 + r) * ldo + n;
            if (vector_out) {
                *reinterpret_cast<float4*>(at) = v;
            } else {
                at[0] = v.x;
                if (n + 1 < N) at[1] = v.y;
                if (n + 2 < N) at[2] = v.z;
                if (n + 3 < N) at[3] = v.w;
            }
        };
        // (kept short: an instruction that no CTA of the SM has run yet costs more to fetch than to run)
        float4 next = fetch(row_of(0));
#pragma unroll 1
        for (int i = 0; row_of(i) < BM; ++i) {
            const float4 before = next;
            next = fetch(row_of(i + 1));
            finish(row_of(i), before);
        }
        if (splits > 1) cluster_sync_all();                            // the others have read this CTA's results
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
    static const EncodeTiledFn fn = [] {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult result;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &result) != cudaSuccess ||
            result != cudaDriverEntryPointSuccess)
            ptr = nullptr;
        return reinterpret_cast<EncodeTiledFn>(ptr);
    }();
    return fn;
}

// A row-major [rows, K] float32 matrix in boxes of 128 rows x 32 columns (128 bytes), 128-byte swizzle
static bool make_map(CUtensorMap* map, const void* base, int rows, int K, int ld) {
    const EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)ld * 4};
    const cuuint32_t box[2] = {(cuuint32_t)SLOT, (cuuint32_t)BM}, elem[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The parts that K is cut into: by K alone
inline int parts_of(int K) { return K < 512 ? 2 : (K < 2048 ? 4 : 6); }

static void launch_config(cudaLaunchConfig_t* config, cudaLaunchAttribute* attribute, int splits) {
    config->gridDim = dim3(splits);
    config->blockDim = dim3(THREADS);
    config->dynamicSmemBytes = SMEM;
    attribute->id = cudaLaunchAttributeClusterDimension;
    attribute->val.clusterDim.x = splits;
    attribute->val.clusterDim.y = attribute->val.clusterDim.z = 1;
    config->attrs = attribute;
    config->numAttrs = 1;
}

// How many clusters of `splits` CTAs (one per SM) are resident at once: a cluster lies within one group of SMs, so that larger ones leave more
// SMs idle.  Asked of the driver once per size and process.
static int resident_clusters(int splits) {
    static std::mutex lock;
    static int known[9] = {0};
    std::lock_guard<std::mutex> guard(lock);
    if (known[splits] == 0) {
        cudaLaunchConfig_t config = {};
        cudaLaunchAttribute attribute[1];
        launch_config(&config, attribute, splits);
        int count = 0;
        if (cudaOccupancyMaxActiveClusters(&count, (const void*)gemm_f32_tc_kernel, &config) != cudaSuccess || count <= 0) {
            cudaGetLastError();
            count = 128 / splits;
        }
        known[splits] = count;
    }
    return known[splits];
}

}  // namespace f32tc
}  // namespace ps

// The parts of K whose sums ps_gemm_f32_tc adds in order.
PS_EXPORT int ps_gemm_f32_tc_parts(int K) { return ps::f32tc::parts_of(K); }

// float32 products on tcgen05: K at least 256; K and both leading dimensions multiples of 4, A and W on 16-byte boundaries.  accumulate as
// for ps_gemm_simt.  splits: 0 = choose, 1, half of ps_gemm_f32_tc_parts(K) or as many: the CTAs that share K; the bits are the same.
// status: device int32 that a bounded wait sets when it runs out (must not be null).
PS_EXPORT int ps_gemm_f32_tc(const float* A, int lda, const float* W, int ldw, const float* bias, float* out, int ldo, int M, int N, int K,
                             int act, int accumulate, int splits, int* status, void* stream) {
    using namespace ps::f32tc;
    if (M <= 0 || N <= 0) return PS_OK;
    if (!status || K <= 0 || lda < K || ldw < K || ldo < N) return PS_ERR_BAD_ARGUMENT;
    if (K < 256 || K % 4 || lda % 4 || ldw % 4 || (((uintptr_t)A | (uintptr_t)W) & 15)) return PS_ERR_UNSUPPORTED;
    const int parts = parts_of(K), tiles_m = (M + BM - 1) / BM, tiles_n = (N + BN - 1) / BN;
    if (tiles_m > 65535 || (splits != 0 && splits != 1 && 2 * splits != parts && splits != parts)) return PS_ERR_UNSUPPORTED;
    static size_t raised[ps::MAX_DEVICES] = {0};
    if (!ps::ensure_dynamic_smem((const void*)gemm_f32_tc_kernel, SMEM, raised)) return PS_ERR_LAUNCH;
    if (splits == 0) {
        const long long tiles = (long long)tiles_m * tiles_n;
        float least = 0.f;
        for (int s : {1, parts / 2, parts}) {
            const int at_once = resident_clusters(s);
            const float time = (float)((tiles + at_once - 1) / at_once) * (FIXED + PER_SPLIT * s + PER_STAGE * ((K + BK - 1) / BK) / s);
            if (least == 0.f || time < least) { least = time; splits = s; }
        }
    }
    CUtensorMap map_a, map_w;
    if (!make_map(&map_a, A, M, K, lda) || !make_map(&map_w, W, N, K, ldw)) return PS_ERR_LAUNCH;
    return ps::launch_pdl_clusters(gemm_f32_tc_kernel, dim3(tiles_n * splits, tiles_m), dim3(THREADS), SMEM, (cudaStream_t)stream,
                                   dim3(splits), map_a, map_w, A, lda, W, ldw, bias, out, ldo, M, N, K, act, accumulate, parts, splits, status);
}
