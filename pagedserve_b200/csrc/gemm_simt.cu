// CUDA-core GEMM: out = epilogue(A[M,K] * W[N,K]^T + bias).
//
// This is the matrix product of the true 32-bit path (float32 multiply-adds only; no tensor-core
// mode of reduced precision) and the exact reference of the tensor-core GEMM in
// the kernel tests (bf16 inputs, float32 accumulation).  The K loop of each kernel runs in one
// fixed order, so a row's result does not depend on which other rows share its
// tile or on M, on the kernel that it runs on.  Float32 products of at most 16 rows (Ops.linear) run on the few-rows kernel, whose
// order is another one: a row among at most 16 and the same row among more differ by the rounding of float32 sums.  (The tiles' order
// on few rows, 8 x 8 to 16 x 64 outputs a CTA, was measured: 5 rows of 768 x 768 2.4 -> 4.8 us, 768 x 3,072 5.8 -> 13.9.)
//   y = x W^T + b            (reference: nn.Linear at src/model/paged_decoder.py:49-50, 178-179, 295-299)
//   epilogues: bias, GELU(tanh|erf) (reference: src/model/paged_decoder.py:273-280),
//              residual accumulate into a float32 stream (reference: :184, :188)
//
// gemm_f32_tile_kernel   float32, any shape: tiles in shared memory, stages of asynchronous copies.
// gemm_f32_rows_kernel   float32, at most 16 rows: streams the weights once, K over lanes and warps.
// gemm_simt_kernel       bfloat16 operands (shapes that the tensor-core kernels refuse; the tests' reference).
#include "common.cuh"

namespace ps {

constexpr int BM = 64, BN = 64, BK = 16;

template <typename TIn, typename TOut>
__global__ void __launch_bounds__(256)
gemm_simt_kernel(const TIn* __restrict__ A, int lda, const TIn* __restrict__ W, int ldw,
                 const float* __restrict__ bias, TOut* __restrict__ out, int ldo,
                 int M, int N, int K, int act, int accumulate) {
    __shared__ float As[BK][BM + 4];
    __shared__ float Ws[BK][BN + 4];
    pdl_prologue();
    A = pdl_fresh(A);
    int tid = threadIdx.x;
    int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    int tx = tid & 15, ty = tid >> 4;  // 16 x 16 threads, 4x4 outputs each
    int lr = tid >> 2, lk = (tid & 3) * 4;  // loader: row 0..63, k offset 0,4,8,12
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

    for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            int k = k0 + lk + j;
            int m = m0 + lr, n = n0 + lr;
            As[lk + j][lr] = (m < M && k < K) ? to_float(A[(size_t)m * lda + k]) : 0.f;
            Ws[lk + j][lr] = (n < N && k < K) ? to_float(W[(size_t)n * ldw + k]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            float a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = As[kk][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = Ws[kk][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        int m = m0 + ty * 4 + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            int n = n0 + tx * 4 + j;
            if (n >= N) continue;
            float v = acc[i][j];
            if (bias) v = (accumulate & PS_COLUMN_FACTOR) ? v * bias[n] : v + bias[n];
            v = apply_act(v, act);
            size_t o = (size_t)m * ldo + n;
            if (accumulate & PS_ACCUMULATE) v += to_float(out[o]);
            out[o] = from_float<TOut>(v);
        }
    }
}

template <typename TIn, typename TOut>
int launch_gemm_simt(const void* A, int lda, const void* W, int ldw, const float* bias, void* out, int ldo,
                     int M, int N, int K, int act, int accumulate, cudaStream_t s) {
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    return launch_pdl(gemm_simt_kernel<TIn, TOut>, grid, dim3(256), 0, s, (const TIn*)A, lda, (const TIn*)W, ldw, bias,
                      (TOut*)out, ldo, M, N, K, act, accumulate);
}

// ------------------------------------------------------------------------------------------ float32, tiles
namespace f32 {

constexpr int BK = 32;                       // k's of a stage: a row of 128 bytes
constexpr int ROW = BK + 4;                  // its pitch in shared memory: eight neighbouring rows start on eight different
                                             // groups of four banks, so the reads below meet no conflicts

// VEC: floats of one copy (4 where rows start on 16-byte boundaries, else 1); ok false writes zeros
template <int VEC>
__device__ __forceinline__ void copy_async(float* dst, const float* src, bool ok) {
    const uint32_t to = (uint32_t)__cvta_generic_to_shared(dst);
    const int bytes = ok ? 4 * VEC : 0;
    if constexpr (VEC == 4) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(src), "r"(bytes) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(to), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT> __device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory"); }

// A CTA computes BM x BN outputs, a warp 8 TM x 4 TN of them, a thread TM x TN (rows ty + 8 i, columns 8 (j / 2) + 2 tx + j % 2
// of the warp's part).  Rows of A and W lie in shared memory as they lie in memory, 32 k's of each; a thread reads four k's
// of a row at a time.  Every tile shape adds an output's terms one k after the other.
template <int BM, int BN, int TM, int TN, int STAGES, int VEC>
__global__ void __launch_bounds__((BM / (8 * TM)) * (BN / (4 * TN)) * 32)
gemm_f32_tile_kernel(const float* __restrict__ A, int lda, const float* __restrict__ W, int ldw,
                     const float* __restrict__ bias, float* __restrict__ out, int ldo, int M, int N, int K, int act,
                     int accumulate) {
    constexpr int WARPS_M = BM / (8 * TM), WARPS_N = BN / (4 * TN), THREADS = WARPS_M * WARPS_N * 32;
    constexpr int STAGE = (BM + BN) * ROW;                       // floats of a stage: BM rows of A, BN rows of W
    constexpr int PIECES = BK / VEC, STEP = THREADS / PIECES;    // a thread copies the same piece of every STEP-th row
    static_assert(THREADS % PIECES == 0 && BM % STEP == 0 && BN % STEP == 0, "rows are shared out evenly");
    extern __shared__ __align__(16) float stage_s[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ty = lane >> 2, tx = lane & 3;
    const int row0 = (warp / WARPS_N) * 8 * TM + ty, col0 = (warp % WARPS_N) * 4 * TN + 2 * tx;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int blocks = (K + BK - 1) / BK;
    const int my_row = tid / PIECES, my_k = (tid % PIECES) * VEC;
    float* const to = stage_s + my_row * ROW + my_k;
    const float* a_from = A + (size_t)min(m0 + my_row, M - 1) * lda + my_k;
    const float* const w_from = W + (size_t)min(n0 + my_row, N - 1) * ldw + my_k;

    auto load_weights = [&](int kb) {                            // (K is a multiple of VEC)
        const bool inside = kb * BK + my_k < K;
#pragma unroll
        for (int r = 0; r < BN; r += STEP) {
            const bool ok = inside && n0 + my_row + r < N;
            copy_async<VEC>(to + (kb % STAGES) * STAGE + (BM + r) * ROW, ok ? w_from + (size_t)r * ldw + kb * BK : W, ok);
        }
    };
    auto load_rows = [&](int kb) {
        const bool inside = kb * BK + my_k < K;
#pragma unroll
        for (int r = 0; r < BM; r += STEP) {
            const bool ok = inside && m0 + my_row + r < M;
            copy_async<VEC>(to + (kb % STAGES) * STAGE + r * ROW, ok ? a_from + (size_t)r * lda + kb * BK : A, ok);
        }
    };
    // weights that do not depend on the kernel before this one: those of the first stages go ahead of the wait
    const bool ready = accumulate & PS_WEIGHTS_READY;
    if (ready) {
#pragma unroll
        for (int s = 0; s < STAGES - 1; ++s)
            if (s < blocks) load_weights(s);
    }
    pdl_prologue();
    a_from = pdl_fresh(a_from);
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < blocks) {
            if (!ready) load_weights(s);
            load_rows(s);
        }
        copy_commit();
    }
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

    for (int kb = 0; kb < blocks; ++kb) {
        copy_wait<STAGES - 2>();
        __syncthreads();                                         // stage kb is there, and everyone is done with stage kb - 1
        if (kb + STAGES - 1 < blocks) {
            load_weights(kb + STAGES - 1);
            load_rows(kb + STAGES - 1);
        }
        copy_commit();
        const float* a_s = stage_s + (kb % STAGES) * STAGE + row0 * ROW;
        const float* w_s = stage_s + (kb % STAGES) * STAGE + (BM + col0) * ROW;
#pragma unroll
        for (int k = 0; k < BK; k += 4) {
            float4 a[TM];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const float4*>(a_s + 8 * i * ROW + k);
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const float4 w = *reinterpret_cast<const float4*>(w_s + (8 * (j >> 1) + (j & 1)) * ROW + k);
#pragma unroll
                for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[i].x, w.x, acc[i][j]);
#pragma unroll
                for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[i].y, w.y, acc[i][j]);
#pragma unroll
                for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[i].z, w.z, acc[i][j]);
#pragma unroll
                for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[i].w, w.w, acc[i][j]);
            }
        }
    }
    copy_wait<0>();
#pragma unroll
    for (int j = 0; j < TN; ++j) {
        const int n = n0 + col0 + 8 * (j >> 1) + (j & 1);
        if (n >= N) continue;
        const float b = bias ? bias[n] : 0.f;
#pragma unroll
        for (int i = 0; i < TM; ++i) {
            const int m = m0 + row0 + 8 * i;
            if (m >= M) continue;
            float v = acc[i][j];
            if (bias) v = (accumulate & PS_COLUMN_FACTOR) ? v * b : v + b;
            v = apply_act(v, act);
            float* at = out + (size_t)m * ldo + n;
            *at = (accumulate & PS_ACCUMULATE) ? *at + v : v;
        }
    }
}

template <int BM, int BN, int TM, int TN, int STAGES, int VEC>
int launch_tile(const float* A, int lda, const float* W, int ldw, const float* bias, float* out, int ldo, int M, int N, int K,
                int act, int accumulate, cudaStream_t s) {
    auto kernel = gemm_f32_tile_kernel<BM, BN, TM, TN, STAGES, VEC>;
    constexpr size_t smem = (size_t)STAGES * (BM + BN) * ROW * sizeof(float);
    static size_t raised[MAX_DEVICES] = {0};
    if (!ensure_dynamic_smem((const void*)kernel, smem, raised)) return PS_ERR_LAUNCH;
    return launch_pdl(kernel, dim3((N + BN - 1) / BN, (M + BM - 1) / BM), dim3((BM / (8 * TM)) * (BN / (4 * TN)) * 32), smem, s, A,
                      lda, W, ldw, bias, out, ldo, M, N, K, act, accumulate);
}

// The same product for large shapes (M and N at least 128, K a multiple of 16): a CTA of four warps computes 128 x 128 outputs, a
// thread 8 x 16, from tiles that are turned on their way into shared memory ([k][row], through registers), so that a thread
// reads its 8 rows and 16 columns of one k with six 16-byte accesses for 128 multiply-adds, which are issued as pairs of
// neighbouring columns (fma.rn.f32x2: each half rounds as fmaf does, and the sums are those of the other kernel).  What
// bounds it: the multiply-adds (128 per clock and SM), and how well the registers of the main loop are laid out: the last
// tiles of a row or column are moved back inside the matrix instead of being guarded (what they compute again is not
// stored), and the results pass through shared memory to a rolled loop, because a guarded load or an activation in the
// unrolled registers made the main loop 10 to 25 % slower.  2,048 x 2,304 x 768: 151 us, 48 TFLOP/s; the form above with 64 x 64
// tiles 188, the kernel with scalar loads that was here before 303.
constexpr int WIDE = 128, WIDE_K = 16, WIDE_ROW = WIDE + 4, WIDE_THREADS = 128;

__global__ void __launch_bounds__(WIDE_THREADS, 2)
gemm_f32_wide_kernel(const float* __restrict__ A, int lda, const float* __restrict__ W, int ldw, const float* __restrict__ bias,
                     float* __restrict__ out, int ldo, int M, int N, int K, int act, int accumulate) {
    __shared__ __align__(16) float tiles[4][WIDE_K][WIDE_ROW];                       // two of A, two of W
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, ty = lane >> 2, tx = lane & 3;
    const int m0 = min((int)blockIdx.y * WIDE, M - WIDE), n0 = min((int)blockIdx.x * WIDE, N - WIDE);
    const int row0 = (warp >> 1) * 64, col0 = (warp & 1) * 64;   // the warp's part; a thread: rows 4 ty + {0..3, 32..35}, columns
                                                                 // 4 tx + 16 j + {0..3}
    constexpr int COPIES = WIDE * WIDE_K / 4 / WIDE_THREADS, STEP = WIDE_THREADS / (WIDE_K / 4);
    const int my_row = tid / (WIDE_K / 4), my_k = (tid % (WIDE_K / 4)) * 4;
    const int blocks = K / WIDE_K;
    const float* a_from = A + (size_t)(m0 + my_row) * lda + my_k;
    const float* w_from = W + (size_t)(n0 + my_row) * ldw + my_k;
    float4 a_in[COPIES], w_in[COPIES];
    auto fetch_weights = [&](int kb) {
#pragma unroll
        for (int c = 0; c < COPIES; ++c) w_in[c] = *reinterpret_cast<const float4*>(w_from + (size_t)c * STEP * ldw + kb * WIDE_K);
    };
    auto fetch_rows = [&](int kb) {
#pragma unroll
        for (int c = 0; c < COPIES; ++c) a_in[c] = *reinterpret_cast<const float4*>(a_from + (size_t)c * STEP * lda + kb * WIDE_K);
    };
    auto put = [&](int buf) {
#pragma unroll
        for (int c = 0; c < COPIES; ++c) {
            float (*a_s)[WIDE_ROW] = tiles[buf], (*w_s)[WIDE_ROW] = tiles[2 + buf];
            const int r = my_row + c * STEP;
            a_s[my_k][r] = a_in[c].x; a_s[my_k + 1][r] = a_in[c].y; a_s[my_k + 2][r] = a_in[c].z; a_s[my_k + 3][r] = a_in[c].w;
            w_s[my_k][r] = w_in[c].x; w_s[my_k + 1][r] = w_in[c].y; w_s[my_k + 2][r] = w_in[c].z; w_s[my_k + 3][r] = w_in[c].w;
        }
    };
    pdl_prologue();
    a_from = pdl_fresh(a_from);
    w_from = pdl_fresh(w_from);                                  // (the kernel in front may have made W too)
    fetch_rows(0);
    fetch_weights(0);
    put(0);
    __syncthreads();
    unsigned long long acc[8][8];                                // row i, columns 2 j and 2 j + 1
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0ull;
    for (int kb = 0; kb < blocks; ++kb) {
        const int buf = kb & 1;
        if (kb + 1 < blocks) { fetch_rows(kb + 1); fetch_weights(kb + 1); }
#pragma unroll
        for (int k = 0; k < WIDE_K; ++k) {
            const float4 lo = *reinterpret_cast<const float4*>(&tiles[buf][k][row0 + 4 * ty]);
            const float4 hi = *reinterpret_cast<const float4*>(&tiles[buf][k][row0 + 4 * ty + 32]);
            const float a[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
            ulonglong2 w[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) w[j] = *reinterpret_cast<const ulonglong2*>(&tiles[2 + buf][k][col0 + 4 * tx + 16 * j]);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const unsigned long long twice = pair_of(a[i], a[i]);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    acc[i][2 * j] = pair_fma(twice, w[j].x, acc[i][2 * j]);
                    acc[i][2 * j + 1] = pair_fma(twice, w[j].y, acc[i][2 * j + 1]);
                }
            }
        }
        if (kb + 1 < blocks) put(buf ^ 1);
        __syncthreads();
    }
    // 16 rows x 64 columns of the warp's part at a time through its share of the tiles' memory
    float* own = &tiles[warp][0][0];
    constexpr int OWN_ROW = 68, OWN_ROWS = 16;
    static_assert(OWN_ROWS * OWN_ROW <= WIDE_K * WIDE_ROW, "a warp's rows fit its share");
    const int n = n0 + col0 + 2 * lane, first_m = blockIdx.y * WIDE, first_n = blockIdx.x * WIDE;
    const float b0 = bias ? bias[n] : 0.f, b1 = bias ? bias[n + 1] : 0.f;
#pragma unroll
    for (int part = 0; part < 4; ++part) {                       // rows i = 2 part, 2 part + 1 of every ty
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j)
                *reinterpret_cast<ulonglong2*>(own + (2 * ty + i) * OWN_ROW + 4 * tx + 16 * j) =
                    make_ulonglong2(acc[2 * part + i][2 * j], acc[2 * part + i][2 * j + 1]);
        __syncwarp();
#pragma unroll 1
        for (int r = 0; r < OWN_ROWS; ++r) {
            const int m = m0 + row0 + 4 * (r >> 1) + 32 * (part >> 1) + 2 * (part & 1) + (r & 1);
            if (m < first_m || n + 1 < first_n) continue;        // what a tile before this one stores
            const float2 two = *reinterpret_cast<const float2*>(own + r * OWN_ROW + 2 * lane);
            float v0 = two.x, v1 = two.y;
            if (bias) {
                v0 = (accumulate & PS_COLUMN_FACTOR) ? v0 * b0 : v0 + b0;
                v1 = (accumulate & PS_COLUMN_FACTOR) ? v1 * b1 : v1 + b1;
            }
            if (act != PS_ACT_NONE) { v0 = apply_act(v0, act); v1 = apply_act(v1, act); }
            float* at = out + (size_t)m * ldo + n;
            if (n >= first_n) at[0] = (accumulate & PS_ACCUMULATE) ? at[0] + v0 : v0;
            at[1] = (accumulate & PS_ACCUMULATE) ? at[1] + v1 : v1;
        }
    }
}

template <int VEC>
int run_tile(int tile, const float* A, int lda, const float* W, int ldw, const float* bias, float* out, int ldo, int M, int N, int K,
             int act, int accumulate, cudaStream_t s) {
    if (tile == 2) return launch_tile<64, 64, 4, 8, 4, VEC>(A, lda, W, ldw, bias, out, ldo, M, N, K, act, accumulate, s);
    if (tile == 3) return launch_tile<32, 64, 4, 4, 5, VEC>(A, lda, W, ldw, bias, out, ldo, M, N, K, act, accumulate, s);
    if (tile == 4) return launch_tile<32, 32, 2, 4, 6, VEC>(A, lda, W, ldw, bias, out, ldo, M, N, K, act, accumulate, s);
    return launch_tile<32, 16, 2, 2, 8, VEC>(A, lda, W, ldw, bias, out, ldo, M, N, K, act, accumulate, s);
}

// The tile shape by the tiles that the busiest SM gets: a fixed cost and a cost per tile of each shape, fitted on B200 at K = 768 (us):
// large tiles need fewer reads per multiply-add, small ones leave fewer SMs idle.  The best shape hardly depends on K, which the rule
// leaves out: over 17 to 2,048 rows, 768 to 6,400 columns and K of 768 to 6,400 it is 2.1 % behind the best shape on average, at most
// 14 % but for 200 x 1,600 x 6,400 (22 %).  Us with 128 x 128 / 64 x 64 / 32 x 64 / 32 x 32 / 32 x 16 tiles: 384 x 2,304 x 768
// 97 / 54 / 41 / 56 / 68, 128 x 768 x 768 92 / 36 / 24 / 14 / 15, 2,048 x 768 x 768 95 / 74 / 80 / 98 / 118, 128 x 768 x 3,072
// 377 / 118 / 82 / 50 / 55, 2,048 x 768 x 3,072 357 / 258 / 296 / 377 / 457, 651 x 1,024 x 4,096 476 / 257 / 197 / 241 / 294, 2,048 x 1,024 x
// 4,096 473 / 476 / 538 / 636 / 790.
// (wide: whether the 128 x 128 tiles take the shape.)
inline int choose_tile(int M, int N, bool wide) {
    constexpr int rows[5] = {128, 64, 32, 32, 32}, columns[5] = {128, 64, 64, 32, 16};
    constexpr float fixed[5] = {24.f, 15.f, 10.f, 3.f, 4.f}, each[5] = {64.f, 21.5f, 13.3f, 11.4f, 6.3f};
    int tile = 0;
    float least = 0.f;
    for (int t = wide ? 0 : 1; t < 5; ++t) {
        const long long ctas = (long long)((M + rows[t] - 1) / rows[t]) * ((N + columns[t] - 1) / columns[t]);
        const float cost = fixed[t] + each[t] * (float)((ctas + 147) / 148);
        if (least == 0.f || cost < least) { least = cost; tile = t + 1; }
    }
    return tile;
}
inline bool takes_wide(int M, int N, int K, bool aligned) { return aligned && M >= WIDE && N >= WIDE && K % WIDE_K == 0; }

int pick_tile(const float* A, int lda, const float* W, int ldw, const float* bias, float* out, int ldo, int M, int N, int K,
              int act, int accumulate, int tile, cudaStream_t s) {
    const bool aligned = (((uintptr_t)A | (uintptr_t)W) & 15) == 0 && lda % 4 == 0 && ldw % 4 == 0 && K % 4 == 0;
    const bool wide = takes_wide(M, N, K, aligned);
    if (tile < 0 || tile > 5 || (tile == 1 && !wide)) return PS_ERR_UNSUPPORTED;
    if (tile == 0) tile = choose_tile(M, N, wide);
    if (tile == 1)
        return launch_pdl(gemm_f32_wide_kernel, dim3((N + WIDE - 1) / WIDE, (M + WIDE - 1) / WIDE), dim3(WIDE_THREADS), 0, s, A, lda,
                          W, ldw, bias, out, ldo, M, N, K, act, accumulate);
    if (aligned) return run_tile<4>(tile, A, lda, W, ldw, bias, out, ldo, M, N, K, act, accumulate, s);
    return run_tile<1>(tile, A, lda, W, ldw, bias, out, ldo, M, N, K, act, accumulate, s);
}

// ------------------------------------------------------------------------------------------ float32, few rows
// At most 16 rows: the product is bound by the bytes of W and by the latency of getting them.  A CTA owns COLS weight rows
// (output columns); a warp takes 128 k's of them at a time (a lane four), the warps of the CTA share K, and a warp has the
// loads of UNROLL such steps on their way before it waits for the kernel that makes A.  A lane keeps a pair of sums (even
// and odd k's) per output; they are added over the lanes by halving exchanges (after which a lane holds the sum of one
// output), then over the warps in shared memory, in a fixed order.
constexpr int ROWS_WARPS = 8;

template <int TOKENS, int COLS, int UNROLL>
__global__ void __launch_bounds__(ROWS_WARPS * 32)
gemm_f32_rows_kernel(const float* __restrict__ A, int lda, const float* __restrict__ W, int ldw,
                     const float* __restrict__ bias, float* __restrict__ out, int ldo, int M, int N, int K, int act,
                     int accumulate) {
    constexpr int OUTS = COLS * TOKENS;                          // output (m, c) is number m * COLS + c
    static_assert(OUTS <= 32, "a lane ends with the sum of one output");
    constexpr int SHARE = 32 / OUTS;                             // lanes that end with the same sum
    __shared__ float red[ROWS_WARPS][OUTS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n0 = blockIdx.x * COLS;
    const int steps = (K + 127) >> 7;
    const float* w_row[COLS];
#pragma unroll
    for (int c = 0; c < COLS; ++c) w_row[c] = W + (size_t)min(n0 + c, N - 1) * ldw + 4 * lane;
    const int mine = threadIdx.x;                                // the output that this thread stores, if any
    const int my_n = n0 + mine % COLS, my_m = mine / COLS;
    const bool stores = mine < OUTS && my_n < N && my_m < M;
    const float my_bias = (bias && stores) ? bias[my_n] : 0.f;
    float before = 0.f;
    auto after_wait = [&]() {
        pdl_prologue();
        A = pdl_fresh(A);
        if (stores && (accumulate & PS_ACCUMULATE)) before = out[(size_t)my_m * ldo + my_n];
    };
    unsigned long long acc[TOKENS][COLS];
#pragma unroll
    for (int m = 0; m < TOKENS; ++m)
#pragma unroll
        for (int c = 0; c < COLS; ++c) acc[m][c] = 0ull;
    bool waited = false;
    for (int s0 = warp; s0 < steps; s0 += ROWS_WARPS * UNROLL) {
        uint4 w[UNROLL][COLS];
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
            const int k = (s0 + u * ROWS_WARPS) * 128;
            const bool ok = k + 4 * lane < K;                    // (K is a multiple of 4)
#pragma unroll
            for (int c = 0; c < COLS; ++c) {
                w[u][c] = make_uint4(0, 0, 0, 0);
                if (ok) asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                                     : "=r"(w[u][c].x), "=r"(w[u][c].y), "=r"(w[u][c].z), "=r"(w[u][c].w) : "l"(w_row[c] + k));
            }
        }
        if (!waited) { after_wait(); waited = true; }
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
            const int k = (s0 + u * ROWS_WARPS) * 128 + 4 * lane;
            if (k >= K) continue;
            unsigned long long lo[COLS], hi[COLS];
#pragma unroll
            for (int c = 0; c < COLS; ++c) {
                lo[c] = pair_of(__uint_as_float(w[u][c].x), __uint_as_float(w[u][c].y));
                hi[c] = pair_of(__uint_as_float(w[u][c].z), __uint_as_float(w[u][c].w));
            }
#pragma unroll
            for (int m = 0; m < TOKENS; ++m) {
                // (rows past M read the last one again: their sums are not stored)
                const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(A + (size_t)min(m, M - 1) * lda + k);
#pragma unroll
                for (int c = 0; c < COLS; ++c) acc[m][c] = pair_fma(a.x, lo[c], acc[m][c]);
#pragma unroll
                for (int c = 0; c < COLS; ++c) acc[m][c] = pair_fma(a.y, hi[c], acc[m][c]);
            }
        }
    }
    if (!waited) after_wait();
    float v[OUTS];
#pragma unroll
    for (int i = 0; i < OUTS; ++i) {
        float even, odd;
        pair_split(acc[i / COLS][i % COLS], even, odd);
        v[i] = even + odd;
    }
    // each exchange halves the outputs of a lane: it keeps the upper or the lower half by one bit of its number
    int held = OUTS;
#pragma unroll
    for (int offset = 16; offset > 0; offset >>= 1) {
        if (held > 1) {
            held >>= 1;
            const bool upper = lane & offset;
#pragma unroll
            for (int i = 0; i < OUTS / 2; ++i) {
                if (i < held) {
                    const float give = upper ? v[i] : v[i + held], keep = upper ? v[i + held] : v[i];
                    v[i] = keep + __shfl_xor_sync(0xffffffffu, give, offset);
                }
            }
        } else {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], offset);
        }
    }
    if (lane % SHARE == 0) red[warp][lane / SHARE] = v[0];
    __syncthreads();
    if (!stores) return;
    float sum = 0.f;
#pragma unroll
    for (int w = 0; w < ROWS_WARPS; ++w) sum += red[w][mine];
    if (bias) sum = (accumulate & PS_COLUMN_FACTOR) ? sum * my_bias : sum + my_bias;
    out[(size_t)my_m * ldo + my_n] = before + apply_act(sum, act);
}

// The same for K up to 128 WARPS, where a warp has one step: it keeps its part of the rows of A in registers, walks over several
// groups of COLS columns and has the next group's weights on their way while it adds up the present one.  The sums are those of
// the kernel above.  8 rows x 50,257 x 768: 82 -> 41 us, 1 row 35 -> 24 (with a CTA per group each of 42 rounds of CTAs waited for its weights).
template <int TOKENS, int COLS, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, 2)
gemm_f32_rows_walk_kernel(const float* __restrict__ A, int lda, const float* __restrict__ W, int ldw,
                          const float* __restrict__ bias, float* __restrict__ out, int ldo, int M, int N, int K, int act,
                          int accumulate) {
    constexpr int OUTS = COLS * TOKENS, SHARE = 32 / OUTS;
    static_assert(OUTS <= 32, "a lane ends with the sum of one output");
    __shared__ float red[2][WARPS][OUTS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, k = 128 * warp + 4 * lane;
    const bool inside = k < K;                                   // (K is a multiple of 4)
    uint4 w[COLS];
    auto fetch = [&](int n0) {
#pragma unroll
        for (int c = 0; c < COLS; ++c) {
            w[c] = make_uint4(0, 0, 0, 0);
            if (inside) asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                                     : "=r"(w[c].x), "=r"(w[c].y), "=r"(w[c].z), "=r"(w[c].w) : "l"(W + (size_t)min(n0 + c, N - 1) * ldw + k));
        }
    };
    fetch(blockIdx.x * COLS);
    pdl_prologue();
    A = pdl_fresh(A);
    ulonglong2 a[TOKENS];
#pragma unroll
    for (int m = 0; m < TOKENS; ++m)
        a[m] = inside ? *reinterpret_cast<const ulonglong2*>(A + (size_t)min(m, M - 1) * lda + k) : make_ulonglong2(0ull, 0ull);
    int turn = 0;
    for (int n0 = blockIdx.x * COLS; n0 < N; n0 += gridDim.x * COLS, turn ^= 1) {
        float v[OUTS];
#pragma unroll
        for (int c = 0; c < COLS; ++c) {
            const unsigned long long lo = pair_of(__uint_as_float(w[c].x), __uint_as_float(w[c].y));
            const unsigned long long hi = pair_of(__uint_as_float(w[c].z), __uint_as_float(w[c].w));
#pragma unroll
            for (int m = 0; m < TOKENS; ++m) {
                float even, odd;
                pair_split(pair_fma(a[m].y, hi, pair_fma(a[m].x, lo, 0ull)), even, odd);
                v[m * COLS + c] = even + odd;
            }
        }
        if (n0 + (int)gridDim.x * COLS < N) fetch(n0 + gridDim.x * COLS);
        int held = OUTS;
#pragma unroll
        for (int offset = 16; offset > 0; offset >>= 1) {
            if (held > 1) {
                held >>= 1;
                const bool upper = lane & offset;
#pragma unroll
                for (int i = 0; i < OUTS / 2; ++i) {
                    if (i < held) {
                        const float give = upper ? v[i] : v[i + held], keep = upper ? v[i + held] : v[i];
                        v[i] = keep + __shfl_xor_sync(0xffffffffu, give, offset);
                    }
                }
            } else {
                v[0] += __shfl_xor_sync(0xffffffffu, v[0], offset);
            }
        }
        if (lane % SHARE == 0) red[turn][warp][lane / SHARE] = v[0];
        __syncthreads();                                         // (two buffers: the next group's sums go into the other one)
        const int mine = threadIdx.x, n = n0 + mine % COLS, m = mine / COLS;
        if (mine < OUTS && n < N && m < M) {
            float sum = 0.f;
#pragma unroll
            for (int i = 0; i < WARPS; ++i) sum += red[turn][i][mine];
            if (bias) sum = (accumulate & PS_COLUMN_FACTOR) ? sum * bias[n] : sum + bias[n];
            float* to = out + (size_t)m * ldo + n;
            sum = apply_act(sum, act);
            *to = (accumulate & PS_ACCUMULATE) ? *to + sum : sum;
        }
    }
}

// CTAs of the walking form on an SM at once, by their registers
constexpr int walkers_per_sm(int tokens, int warps) { return tokens == 2 ? (warps == 6 ? 4 : 3) : tokens == 4 ? (warps == 6 ? 3 : 2) : 2; }

// K up to 1,024: CTAs that stay and walk over the groups where there are more of them than are resident at once (2 to 4 on an SM), each of
// which would wait for its weights again; few rows leave room for enough (registers) to be as fast without.  Us, one CTA a group / walking: 8
// rows 2,304 x 768 4.9 / 3.7, 3,072 x 768 6.6 / 4.7, 4,096 x 1,024 9.0 / 6.4, 768 x 768 (one wave) 2.3 / 2.5; 16 rows 768 x 768 5.8 / 3.3,
// 2,304 x 768 10.7 / 5.3; 4 rows 3,072 x 768 5.0 / 3.6; 2 rows 2,304 x 768 2.2 / 2.8, 4,096 x 1,024 4.5 / 4.8.  As many walkers as are resident: 4 rows x
// 50,257 x 768, 444 / 592 of them 29 / 37, 2 rows x 50,257 x 1,024 33 / 40.
// Beyond: the steps whose weights a warp has on their way together, against the registers they take (with 8 rows and one step two CTAs are on
// an SM, with three one).  Us, 1 / 2 / 3 steps: 2 rows 768 x 3,072 3.7 / 3.4 / 2.7, 4,800 x 1,600 8.1 / 7.3 / 9.1, 1,600 x 6,400 10.2 / 8.8 / 11.5; 4 rows
// 4,800 x 1,600 12.0 / 9.5 / 9.9, 768 x 3,072 3.9 / 3.6 / 2.8; 8 rows 768 x 3,072 5.3 / 9.2 / 5.9, 1,024 x 4,096 7.0 / 12.7 / 8.7, 1,600 x 6,400 19.7 / 27 / 18.2,
// but where each CTA has an SM to itself one step leaves it waiting: 592 x 3,072 (148 CTAs) 4.3 with one, 3.0 with three, 600 x 3,072 4.2 / 5.0;
// 16 rows 768 x 3,072 13.8 / 10.0 / 12.4, 1,600 x 6,400 44 / 31 / 45.
template <int TOKENS, int COLS>
int launch_rows(const float* A, int lda, const float* W, int ldw, const float* bias, float* out, int ldo, int M, int N, int K,
                int act, int accumulate, cudaStream_t s) {
    const int groups = (N + COLS - 1) / COLS;
    const dim3 grid(groups), block(ROWS_WARPS * 32);
#define PS_ROWS(KERNEL, GRID, BLOCK) return launch_pdl(KERNEL, GRID, BLOCK, 0, s, A, lda, W, ldw, bias, out, ldo, M, N, K, act, accumulate)
    if (K <= 128 * ROWS_WARPS) {
        if (groups > (TOKENS == 2 ? 1184 : 296)) {
            const bool narrow = K <= 128 * 6;
            const dim3 walkers(min(groups, 148 * walkers_per_sm(TOKENS, narrow ? 6 : 8)));
            if (narrow) PS_ROWS((gemm_f32_rows_walk_kernel<TOKENS, COLS, 6>), walkers, dim3(6 * 32));
            PS_ROWS((gemm_f32_rows_walk_kernel<TOKENS, COLS, 8>), walkers, block);
        }
        PS_ROWS((gemm_f32_rows_kernel<TOKENS, COLS, 1>), grid, block);
    }
    if constexpr (TOKENS == 16) {
        PS_ROWS((gemm_f32_rows_kernel<TOKENS, COLS, 2>), grid, block);
    } else if constexpr (TOKENS == 8) {
        if (K <= 4096 && groups > 148) PS_ROWS((gemm_f32_rows_kernel<TOKENS, COLS, 1>), grid, block);
    } else {
        if (K <= 2048 || (TOKENS == 2 && K > 4096)) PS_ROWS((gemm_f32_rows_kernel<TOKENS, COLS, 2>), grid, block);
    }
    if constexpr (TOKENS < 16) PS_ROWS((gemm_f32_rows_kernel<TOKENS, COLS, 3>), grid, block);
#undef PS_ROWS
}

}  // namespace f32

}  // namespace ps

// in_dtype: dtype of A and W. out_dtype: dtype of out. accumulate: PS_ACCUMULATE: out += result (out must be f32);
// PS_COLUMN_FACTOR: the numbers of `bias` multiply the columns; PS_WEIGHTS_READY: float32 weights may be read before the kernel in
// front has ended.  tile: 0 = choose; float32: 1 to 5 = tiles of 128 x 128 (M and N at least 128, K a multiple of 16, 16-byte rows),
// 64 x 64, 32 x 64, 32 x 32, 32 x 16.
PS_EXPORT int ps_gemm_simt(const void* A, int lda, const void* W, int ldw, const float* bias, void* out,
                           int ldo, int M, int N, int K, int in_dtype, int out_dtype, int act,
                           int accumulate, int tile, void* stream) {
    if (M <= 0 || N <= 0) return PS_OK;
    if (K <= 0 || lda < K || ldw < K || ldo < N) return PS_ERR_BAD_ARGUMENT;
    if ((accumulate & PS_ACCUMULATE) && out_dtype != PS_F32) return PS_ERR_BAD_ARGUMENT;
    cudaStream_t s = (cudaStream_t)stream;
    using bf = __nv_bfloat16;
    if (in_dtype == PS_F32 && out_dtype == PS_F32)
        return ps::f32::pick_tile((const float*)A, lda, (const float*)W, ldw, bias, (float*)out, ldo, M, N, K, act, accumulate, tile, s);
    if (tile) return PS_ERR_UNSUPPORTED;
    if (in_dtype == PS_BF16 && out_dtype == PS_F32)
        return ps::launch_gemm_simt<bf, float>(A, lda, W, ldw, bias, out, ldo, M, N, K, act, accumulate, s);
    if (in_dtype == PS_BF16 && out_dtype == PS_BF16)
        return ps::launch_gemm_simt<bf, bf>(A, lda, W, ldw, bias, out, ldo, M, N, K, act, accumulate, s);
    return PS_ERR_UNSUPPORTED;
}

// The tile that ps_gemm_simt chooses for a float32 product; aligned: K and leading dimensions multiples of 4, 16-byte addresses.
PS_EXPORT int ps_gemm_f32_tile(int M, int N, int K, int aligned) {
    return ps::f32::choose_tile(M, N, ps::f32::takes_wide(M, N, K, aligned && K % 4 == 0));
}

// float32 products of at most 16 rows: K and both leading dimensions multiples of 4, A and W on 16-byte boundaries.  W is read
// before the kernel in front has ended, whatever PS_WEIGHTS_READY says.
PS_EXPORT int ps_gemm_f32_rows(const float* A, int lda, const float* W, int ldw, const float* bias, float* out, int ldo, int M,
                               int N, int K, int act, int accumulate, void* stream) {
    if (M <= 0 || N <= 0) return PS_OK;
    if (K <= 0 || lda < K || ldw < K || ldo < N) return PS_ERR_BAD_ARGUMENT;
    if (M > 16 || K % 4 || lda % 4 || ldw % 4 || (((uintptr_t)A | (uintptr_t)W) & 15)) return PS_ERR_UNSUPPORTED;
    cudaStream_t s = (cudaStream_t)stream;
    if (M <= 2) return ps::f32::launch_rows<2, 4>(A, lda, W, ldw, bias, out, ldo, M, N, K, act, accumulate, s);
    if (M <= 4) return ps::f32::launch_rows<4, 4>(A, lda, W, ldw, bias, out, ldo, M, N, K, act, accumulate, s);
    if (M <= 8) return ps::f32::launch_rows<8, 4>(A, lda, W, ldw, bias, out, ldo, M, N, K, act, accumulate, s);
    return ps::f32::launch_rows<16, 2>(A, lda, W, ldw, bias, out, ldo, M, N, K, act, accumulate, s);
}
