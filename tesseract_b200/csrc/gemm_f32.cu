// True 32-bit matrix product for the float32 path: C[M,N] = A[M,K] * W[N,K]^T.
//
// Fused multiply-adds on the ordinary pipe (no tensor cores, so no reduced-precision matrix mode can slip in).
// Every output element is summed in one order that K alone decides, whatever M, N, the tile position or the batch, so
// logits do not depend on how a prompt is cut or what shares the step.  The order: K is cut into blocks of 256, a block
// into four chains, and chain c of block b is the chain of fused multiply-adds over
//     k = 256 b + 32 i + 8 c + e,   i = 0..7 outside, e = 0..7 inside,
// started at zero; the element is the sum of its chains, ascending by (b, c).  Four lanes that hold the four chains of
// a block read whole 128-byte lines of a weight row, which is what the streaming kernel for few rows is made of; the tile
// kernel for many rows walks the same order.  Chains of 64 are also more exact than one of K: products of unit normals are
// 1.8e-7 (K = 2,048) and 2.5e-7 (K = 8,192) off the 64-bit product in the 2-norm, one chain of K 8.1e-7 and 1.6e-6.
// The reference runs this product through a library in bfloat16 only (src/cuda/cublas.rs:49-92); a 32-bit path has no
// counterpart there.
#include "common.cuh"

namespace {

constexpr int KBLOCK = 256, CHAINS = 4, GROUPS = 8;     // a chain is GROUPS runs of 8 numbers

// ---- many rows: tiles in shared memory ------------------------------------------------------------------------------

constexpr int BK = 16;          // numbers of K a stage: two runs of eight of one chain

// Two multiply-adds an instruction: the pipe is as fast as with single ones, but half the issue slots are left for the
// loads from shared memory (the bits are those of fmaf).
__device__ __forceinline__ void fma2(uint64_t& d, uint64_t a, uint64_t b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ void add2(uint64_t& d, uint64_t a) { asm("add.rn.f32x2 %0, %0, %1;" : "+l"(d) : "l"(a)); }
__device__ __forceinline__ uint64_t twice(float a) {
    uint64_t d;
    asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(a));
    return d;
}

// Stage t = 16 b + 4 c + p covers the runs i = 2p, 2p + 1 of chain c of block b; its first number of K:
__host__ __device__ __forceinline__ int stage_start(int t) { return (t >> 4) * KBLOCK + (t & 3) * 64 + ((t >> 2) & 3) * 8; }
// The next stage that reaches into K (the others of the last block would add zeros alone).
__device__ __forceinline__ int next_stage(int t, int stages, int K) {
    do { ++t; } while (t < stages && stage_start(t) >= K);
    return t;
}

// A thread's totals: rows (i / 4) (BM / 2) + 4 ty + i % 4, columns h (BN / 2) + 4 tx .. of its tile.
template <int BM, int BN, int TN>
__device__ __forceinline__ void store_tile(const uint64_t (&total)[8][TN / 2], float* C, int64_t ldc, int m0, int n0, int tx, int ty,
                                           int M, int N) {
    constexpr int QN = TN / 4;
    const bool packets = ldc % 4 == 0 && (uintptr_t)C % 16 == 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int m = m0 + (i / 4) * (BM / 2) + ty * 4 + i % 4;
        if (m >= M) continue;
#pragma unroll
        for (int h = 0; h < QN; ++h) {
            const int n = n0 + h * (BN / 2) + tx * 4;
            float* row = C + (int64_t)m * ldc + n;
            const float2 lo = *reinterpret_cast<const float2*>(&total[i][h * 2]);
            const float2 hi = *reinterpret_cast<const float2*>(&total[i][h * 2 + 1]);
            if (packets && n + 4 <= N) {
                *reinterpret_cast<float4*>(row) = make_float4(lo.x, lo.y, hi.x, hi.y);
            } else {
                if (n < N) row[0] = lo.x;
                if (n + 1 < N) row[1] = lo.y;
                if (n + 2 < N) row[2] = hi.x;
                if (n + 3 < N) row[3] = hi.y;
            }
        }
    }
}

// A thread keeps 8 x TN sums of the current chain and as many totals in registers.  Bound by the loads from shared memory
// (the path is 76 % busy, the multiply-add pipe 61 %) where the tiles fill the chip, by the latency of a stage where they
// do not.  500 rows of 16,384 x 2,048 take 799 us (42 TFLOP/s; single-number instructions 12 % more, 64 x 64 tiles of one
// chain of K, as before, 1,009), 2,048 rows 3.14 ms (3.92).
// Blocks that are placed while the kernel in front still runs go to where room is left, two or four to a multiprocessor while
// others stay empty.  So blocks that would fit beyond an even share are kept off by the shared memory they ask for (spread() below:
// 39 rows of 16,384 x 2,048 in a layer of the 1B sizes 117 us less), and the next kernel is let in when the sums are done (200 rows
// of 2,048 x 128 one after another 7.5 us, 14.9 with the next one let in at the start).
// (A is not declared __restrict__: loads that the compiler takes for constant may be moved in front of the wait.)
template <bool VEC, int BM, int BN, int TN>
__global__ void __launch_bounds__((BM / 8) * (BN / TN))
gemm_f32_tile_kernel(const float* A, int64_t lda, const float* W, int64_t ldw, float* C, int64_t ldc, int M, int N,
                     int K) {
    constexpr int THREADS = (BM / 8) * (BN / TN), COLS = BN / TN, QN = TN / 4;
    constexpr int LA = BM * 4 / THREADS, LW = BN * 4 / THREADS;        // 16-byte packets a thread loads a stage
    __shared__ __align__(16) float As[2][BK][BM + 4];
    __shared__ __align__(16) float Ws[2][BK][BN + 4];
    const int tid = threadIdx.x;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int tx = tid % COLS, ty = tid / COLS;
    const int stages = (K + KBLOCK - 1) / KBLOCK * 16;

    uint64_t acc[8][TN / 2], total[8][TN / 2];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) acc[i][j] = total[i][j] = 0;

    float a[LA][4], w[LW][4];
    auto fetch_one = [&](const float* base, int64_t ld, int row, int rows, int kk, float* v) {
        v[0] = v[1] = v[2] = v[3] = 0.0f;
        if (row >= rows) return;
        if (VEC) {
            if (kk < K) {
                const float4 t = *reinterpret_cast<const float4*>(base + (int64_t)row * ld + kk);
                v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
            }
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (kk + e < K) v[e] = base[(int64_t)row * ld + kk + e];
        }
    };
    auto fetch = [&](int t) {
        const int q = tid % 4, kk = stage_start(t) + (q >> 1) * 32 + (q & 1) * 4;
#pragma unroll
        for (int l = 0; l < LA; ++l) fetch_one(A, lda, m0 + l * (THREADS / 4) + tid / 4, M, kk, a[l]);
#pragma unroll
        for (int l = 0; l < LW; ++l) fetch_one(W, ldw, n0 + l * (THREADS / 4) + tid / 4, N, kk, w[l]);
    };
    auto put = [&](int buffer) {
        const int q = tid % 4;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
#pragma unroll
            for (int l = 0; l < LA; ++l) As[buffer][q * 4 + e][l * (THREADS / 4) + tid / 4] = a[l][e];
#pragma unroll
            for (int l = 0; l < LW; ++l) Ws[buffer][q * 4 + e][l * (THREADS / 4) + tid / 4] = w[l][e];
        }
    };

    pdl_wait();
    int t = 0, buffer = 0;
    fetch(t);
    put(0);
    __syncthreads();
    while (t < stages) {
        const int ahead = next_stage(t, stages, K);
        if (ahead < stages) fetch(ahead);
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            float ar[8];
            uint64_t wr[TN / 2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float4 v = *reinterpret_cast<const float4*>(&As[buffer][k][h * (BM / 2) + ty * 4]);
                ar[h * 4] = v.x; ar[h * 4 + 1] = v.y; ar[h * 4 + 2] = v.z; ar[h * 4 + 3] = v.w;
            }
#pragma unroll
            for (int h = 0; h < QN; ++h) {
                const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(&Ws[buffer][k][h * (BN / 2) + tx * 4]);
                wr[h * 2] = v.x; wr[h * 2 + 1] = v.y;
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint64_t both = twice(ar[i]);
#pragma unroll
                for (int j = 0; j < TN / 2; ++j) fma2(acc[i][j], both, wr[j]);
            }
        }
        if ((ahead >> 2) != (t >> 2)) {         // the chain ends here
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < TN / 2; ++j) {
                    add2(total[i][j], acc[i][j]);
                    acc[i][j] = 0;
                }
        }
        buffer ^= 1;
        if (ahead < stages) put(buffer);
        __syncthreads();
        t = ahead;
    }
    pdl_trigger();
    store_tile<BM, BN, TN>(total, C, ldc, m0, n0, tx, ty, M, N);
}

// Tiles that walk K as it lies, 32 numbers a stage, with the sums of all four chains of a block side by side (a thread 4 x 4
// outputs): a short K fills its stages, where a chain after another leaves half or three quarters of one empty.  SHORT (K <= 32):
// a chain is eight numbers, so one sum at a time is enough and twice the threads fit.  Bound by the latency of a stage: 200 rows of
// 2,048 x 32 take 2.9 us (the chains one after another, 7.5), 64 rows of 2,048 x 96 6.3 (7.2), 100 rows of 100 x 33 3.8 (5.0); with
// more than two tiles a multiprocessor the registers cost more than the stages give (300 rows of 5,120 x 96: 17.5 against 14.3).
constexpr int EK = 32;
template <bool VEC, bool SHORT>
__global__ void __launch_bounds__(256, SHORT ? 4 : 2)
gemm_f32_even_kernel(const float* A, int64_t lda, const float* W, int64_t ldw, float* C, int64_t ldc, int M, int N, int K) {
    constexpr int P = 64 + 4;
    __shared__ __align__(16) float As[2][EK][P];
    __shared__ __align__(16) float Ws[2][EK][P];
    const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
    const int m0 = blockIdx.y * 64, n0 = blockIdx.x * 64;
    const int stages = (K + EK - 1) / EK;
    // a thread's packets of a stage: row (u >> 1) & 63, numbers 4 q .. 4 q + 3 (neighbouring lanes take a row's 32 bytes, and
    // write to different banks)
    const int row_of = (tid >> 1) & 63, q0 = (tid & 1) + 2 * (tid >> 7);

    float a[2][4], w[2][4];
    auto fetch_one = [&](const float* base, int64_t ld, int row, int rows, int kk, float* v) {
        v[0] = v[1] = v[2] = v[3] = 0.0f;
        if (row >= rows) return;
        if (VEC) {
            if (kk < K) {
                const float4 t = *reinterpret_cast<const float4*>(base + (int64_t)row * ld + kk);
                v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
            }
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (kk + e < K) v[e] = base[(int64_t)row * ld + kk + e];
        }
    };
    auto fetch = [&](int stage) {
#pragma unroll
        for (int l = 0; l < 2; ++l) {
            const int kk = stage * EK + (q0 + 4 * l) * 4;
            fetch_one(A, lda, m0 + row_of, M, kk, a[l]);
            fetch_one(W, ldw, n0 + row_of, N, kk, w[l]);
        }
    };
    auto put = [&](int buffer) {
#pragma unroll
        for (int l = 0; l < 2; ++l)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                As[buffer][(q0 + 4 * l) * 4 + e][row_of] = a[l][e];
                Ws[buffer][(q0 + 4 * l) * 4 + e][row_of] = w[l][e];
            }
    };

    constexpr int LIVE = SHORT ? 1 : CHAINS;       // sums of chains that are under way at a time
    float acc[LIVE][4][4], total[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            total[i][j] = 0.0f;
#pragma unroll
            for (int c = 0; c < LIVE; ++c) acc[c][i][j] = 0.0f;
        }
    auto add_up = [&](float (&sum)[4][4]) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                total[i][j] += sum[i][j];
                sum[i][j] = 0.0f;
            }
    };
    pdl_wait();
    fetch(0);
    put(0);
    __syncthreads();
    for (int stage = 0; stage < stages; ++stage) {
        const int buffer = stage & 1;
        const bool more = stage + 1 < stages;
        if (more) fetch(stage + 1);
#pragma unroll
        for (int c = 0; c < CHAINS; ++c) {
            if (stage * EK + c * 8 >= K) break;
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const float4 x = *reinterpret_cast<const float4*>(&As[buffer][c * 8 + e][ty * 4]);
                const float4 y = *reinterpret_cast<const float4*>(&Ws[buffer][c * 8 + e][tx * 4]);
                const float xs[4] = {x.x, x.y, x.z, x.w}, ys[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[SHORT ? 0 : c][i][j] = fmaf(xs[i], ys[j], acc[SHORT ? 0 : c][i][j]);
            }
            if (SHORT) add_up(acc[0]);
        }
        if (!SHORT && (stage % GROUPS == GROUPS - 1 || !more)) {       // the block ends here: its chains in order
#pragma unroll
            for (int c = 0; c < LIVE; ++c) add_up(acc[c]);
        }
        if (more) {
            put(buffer ^ 1);
            __syncthreads();
        }
    }
    pdl_trigger();
    const bool packets = ldc % 4 == 0 && (uintptr_t)C % 16 == 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = m0 + ty * 4 + i, n = n0 + tx * 4;
        if (m >= M) continue;
        float* row = C + (int64_t)m * ldc + n;
        if (packets && n + 4 <= N) {
            *reinterpret_cast<float4*>(row) = make_float4(total[i][0], total[i][1], total[i][2], total[i][3]);
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (n + j < N) row[j] = total[i][j];
        }
    }
}

// The tiles where they are too few to give a multiprocessor more than one: G groups of threads take a tile's chains in turn (K a
// multiple of 256, packets), and the first group adds the sums in the order of the chains, the others' through
// shared memory, so that the bits are those of the kernel above.  Bound by the latency of a group's stages, which the groups hide
// from one another.   128 x 64
// tiles of two groups and 64 x 64 tiles of four take 121 and 72 us for K = 2,048 (one group, where a multiprocessor has one tile:
// 141 and 95).
// (A is not declared __restrict__: loads that the compiler takes for constant may be moved in front of the wait.)
template <int BM, int BN, int TN, int G>
__global__ void __launch_bounds__((BM / 8) * (BN / TN) * G, 1)
gemm_f32_groups_kernel(const float* A, int64_t lda, const float* W, int64_t ldw, float* C, int64_t ldc, int M, int N, int K) {
    constexpr int THREADS = (BM / 8) * (BN / TN), COLS = BN / TN, QN = TN / 4, SUMS = 8 * TN / 4;
    constexpr int LA = BM * 4 / THREADS, LW = BN * 4 / THREADS;
    constexpr int AP = BM + 4, WP = BN + 4, STAGE = BK * (AP + WP);
    extern __shared__ __align__(16) float shared[];
    const int group = threadIdx.x / THREADS, tid = threadIdx.x % THREADS;
    float* stages_at = shared + group * 2 * STAGE;                                    // [2][As | Ws] of this group
    float4* given = reinterpret_cast<float4*>(shared + G * 2 * STAGE);                // [G - 1][SUMS][THREADS]
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int tx = tid % COLS, ty = tid / COLS;
    const int stages = K / KBLOCK * 16;
    auto group_barrier = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "n"(THREADS) : "memory"); };

    uint64_t acc[8][TN / 2], total[8][TN / 2];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) acc[i][j] = total[i][j] = 0;
    float a[LA][4], w[LW][4];
    auto fetch_one = [&](const float* base, int64_t ld, int row, int rows, int kk, float* v) {
        const float4 t = row < rows ? *reinterpret_cast<const float4*>(base + (int64_t)row * ld + kk) : make_float4(0.f, 0.f, 0.f, 0.f);
        v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    };
    const int q = tid % 4, row_of = tid / 4;
    auto fetch = [&](int t) {
        const int kk = stage_start(t) + (q >> 1) * 32 + (q & 1) * 4;
#pragma unroll
        for (int l = 0; l < LA; ++l) fetch_one(A, lda, m0 + l * (THREADS / 4) + row_of, M, kk, a[l]);
#pragma unroll
        for (int l = 0; l < LW; ++l) fetch_one(W, ldw, n0 + l * (THREADS / 4) + row_of, N, kk, w[l]);
    };
    auto put = [&](int buffer) {
        float *As = stages_at + buffer * STAGE, *Ws = As + BK * AP;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
#pragma unroll
            for (int l = 0; l < LA; ++l) As[(q * 4 + e) * AP + l * (THREADS / 4) + row_of] = a[l][e];
#pragma unroll
            for (int l = 0; l < LW; ++l) Ws[(q * 4 + e) * WP + l * (THREADS / 4) + row_of] = w[l][e];
        }
    };
    pdl_wait();
    int t = group * 4, buffer = 0;                     // (K / 64 chains, a multiple of four: every group takes as many)
    fetch(t);
    put(0);
    group_barrier();
    while (t < stages) {
        const bool ends = (t & 3) == 3;                // the chain's last stage; the group's next chain is G further
        const int ahead = ends ? t + 1 + 4 * (G - 1) : t + 1;
        if (ahead < stages) fetch(ahead);
        const float *As = stages_at + buffer * STAGE, *Ws = As + BK * AP;
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            float ar[8];
            uint64_t wr[TN / 2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float4 v = *reinterpret_cast<const float4*>(As + k * AP + h * (BM / 2) + ty * 4);
                ar[h * 4] = v.x; ar[h * 4 + 1] = v.y; ar[h * 4 + 2] = v.z; ar[h * 4 + 3] = v.w;
            }
#pragma unroll
            for (int h = 0; h < QN; ++h) {
                const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(Ws + k * WP + h * (BN / 2) + tx * 4);
                wr[h * 2] = v.x; wr[h * 2 + 1] = v.y;
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint64_t both = twice(ar[i]);
#pragma unroll
                for (int j = 0; j < TN / 2; ++j) fma2(acc[i][j], both, wr[j]);
            }
        }
        if (ends) {
            if (group > 0) {
                if (t >= 4 * G) asm volatile("bar.sync %0, %1;" ::"r"(G + 1), "n"(THREADS * G) : "memory");      // the last sums are taken
#pragma unroll
                for (int i = 0; i < SUMS; ++i) {
                    const uint64_t* from = &acc[i * 2 / (TN / 2)][i * 2 % (TN / 2)];
                    const float2 lo = *reinterpret_cast<const float2*>(from), hi = *reinterpret_cast<const float2*>(from + 1);
                    given[((group - 1) * SUMS + i) * THREADS + tid] = make_float4(lo.x, lo.y, hi.x, hi.y);
                }
                asm volatile("bar.arrive %0, %1;" ::"r"(G + 2), "n"(THREADS * G) : "memory");
            } else {
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int j = 0; j < TN / 2; ++j) add2(total[i][j], acc[i][j]);
                asm volatile("bar.sync %0, %1;" ::"r"(G + 2), "n"(THREADS * G) : "memory");                     // the others' sums are there
#pragma unroll
                for (int other = 0; other < G - 1; ++other)
#pragma unroll
                    for (int i = 0; i < SUMS; ++i) {
                        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(&given[(other * SUMS + i) * THREADS + tid]);
                        add2(total[i * 2 / (TN / 2)][i * 2 % (TN / 2)], v.x);
                        add2(total[i * 2 / (TN / 2)][i * 2 % (TN / 2) + 1], v.y);
                    }
                if (ahead < stages) asm volatile("bar.arrive %0, %1;" ::"r"(G + 1), "n"(THREADS * G) : "memory");
            }
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0;
        }
        buffer ^= 1;
        if (ahead < stages) put(buffer);
        group_barrier();
        t = ahead;
    }
    pdl_trigger();
    if (group > 0) return;
    store_tile<BM, BN, TN>(total, C, ldc, m0, n0, tx, ty, M, N);
}

// ---- few rows: the weights stream through registers -----------------------------------------------------------------

constexpr int WARPS = 8, FEATURES = 16;                // a block: 16 weight rows, eight blocks of K at a time
constexpr int STEP = WARPS * KBLOCK;
constexpr int AHEAD = 4;                               // groups of weights in flight a thread
constexpr int kMostStreamed = 1024;                    // rows (a grid's second dimension is far from its limit)

__device__ __forceinline__ void load8(const float* p, bool in, float* v) {
    if (in) {
        asm volatile("ld.global.L1::no_allocate.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
                     : "l"(p));
    } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = 0.0f;
    }
}

// Bound by the stream of the weights up to four rows (N x K = 16,384 x 2,048: 22 us at one row, 23 at four, 5.9 TB/s; the
// 64 x 64 tiles 189): registers hold four groups of weights in flight a thread, 128 KiB a multiprocessor of two blocks.  Blocks of
// eight rows take 160 KiB of shared memory, so that one fits a multiprocessor and half as much is in flight: 33 us, and as
// much again for every eight rows.  2,048 x 8,192 takes 13 to 19 us up to eight rows (the tiles 581), the head of
// 128,256 x 2,048 at one row 151 (961).
// Lane (f, c) runs chain c of its warp's block for the weight rows f and f + 8 and ROWS rows of A.  The rows' part that
// a warp needs lies in shared memory that only this warp writes and reads.
template <int ROWS>
__global__ void __launch_bounds__(WARPS * 32, 2)                     // (of eight rows one block fits, by its shared memory)
gemm_f32_rows_kernel(const float* A, int64_t lda, const float* W, int64_t ldw, float* C, int64_t ldc, int M, int N,
                     int K) {
    extern __shared__ __align__(16) float shared[];
    constexpr int OUTS = ROWS * FEATURES, PART = WARPS * CHAINS * OUTS;
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, f = lane / 4, c = lane % 4;
    float* part = shared;                                            // [2][chain][OUTS]
    float* rows = shared + 2 * PART + warp * 2 * ROWS * KBLOCK;      // [2][ROWS][KBLOCK]
    const int m0 = blockIdx.y * ROWS, tiles = (N + FEATURES - 1) / FEATURES, steps = (K + STEP - 1) / STEP;
    const int units = ((tiles - 1 - blockIdx.x) / gridDim.x + 1) * steps;      // a unit: one tile's 2,048 numbers of K

    const float* w0 = W;
    const float* w1 = W;
    int k_at = 0;
    auto aim = [&](int unit) {                                       // the weights of a unit
        const int n = (blockIdx.x + unit / steps * gridDim.x) * FEATURES + f;
        k_at = unit % steps * STEP + warp * KBLOCK + c * 8;
        w0 = W + (int64_t)min(n, N - 1) * ldw + k_at;
        w1 = W + (int64_t)min(n + 8, N - 1) * ldw + k_at;
    };
    float w[AHEAD][2][8];
    auto fetch = [&](int slot, int group) {
        const bool in = k_at + group * 32 < K;
        load8(w0 + group * 32, in, w[slot][0]);
        load8(w1 + group * 32, in, w[slot][1]);
    };
    auto fetch_rows = [&](int step, int buffer) {
        float* to = rows + buffer * ROWS * KBLOCK;
#pragma unroll
        for (int r = 0; r < ROWS; ++r)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int k = step * STEP + warp * KBLOCK + h * 128 + lane * 4;
                const bool in = m0 + r < M && k < K;
                const float* from = in ? A + (int64_t)(m0 + r) * lda + k : A;
                const uint32_t at = (uint32_t)__cvta_generic_to_shared(to + r * KBLOCK + h * 128 + lane * 4);
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(at), "l"(from), "r"(in ? 16 : 0));
            }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    pdl_trigger();
    aim(0);
    // the first unit's weights go on their way to L2 while the kernel in front still runs (into L2 only: nothing is read
    // before the wait, so the kernel in front may even be the one that writes them)
#pragma unroll
    for (int g = 0; g < GROUPS; ++g)
        if (c == 0 && k_at + g * 32 < K) {
            asm volatile("prefetch.global.L2 [%0];" ::"l"(w0 + g * 32));
            asm volatile("prefetch.global.L2 [%0];" ::"l"(w1 + g * 32));
        }
    pdl_wait();
    fetch_rows(0, 0);
#pragma unroll
    for (int g = 0; g < AHEAD; ++g) fetch(g, g);
    float total = 0.0f;
    for (int unit = 0; unit < units; ++unit) {
        const int buffer = steps > 1 ? unit & 1 : 0;
        const bool more = unit + 1 < units;
        if (steps > 1 && more) {
            __syncwarp();                                            // the other buffer's readers are done
            fetch_rows((unit + 1) % steps, buffer ^ 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncwarp();
        const float* x = rows + buffer * ROWS * KBLOCK + c * 8;
        float acc[2][ROWS];
#pragma unroll
        for (int r = 0; r < ROWS; ++r) acc[0][r] = acc[1][r] = 0.0f;
#pragma unroll
        for (int g = 0; g < GROUPS; ++g) {
            const int slot = g % AHEAD;
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int r = 0; r < ROWS; ++r) {
                    const float4 v = *reinterpret_cast<const float4*>(x + r * KBLOCK + g * 32 + h * 4);
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const float* wv = &w[slot][j][h * 4];
                        acc[j][r] = fmaf(v.x, wv[0], acc[j][r]);
                        acc[j][r] = fmaf(v.y, wv[1], acc[j][r]);
                        acc[j][r] = fmaf(v.z, wv[2], acc[j][r]);
                        acc[j][r] = fmaf(v.w, wv[3], acc[j][r]);
                    }
                }
            if (g == GROUPS - AHEAD && more) aim(unit + 1);
            if (g < GROUPS - AHEAD || more) fetch(slot, (g + AHEAD) % GROUPS);
        }
        float* sums = part + (unit & 1) * PART + (warp * CHAINS + c) * OUTS;
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            sums[r * FEATURES + f] = acc[0][r];
            sums[r * FEATURES + f + 8] = acc[1][r];
        }
        __syncthreads();        // one barrier a unit: the part of two units ago has been summed by now
        if (threadIdx.x < OUTS) {
            const float* from = part + (unit & 1) * PART + threadIdx.x;
#pragma unroll
            for (int s = 0; s < WARPS * CHAINS; ++s) total += from[s * OUTS];
            if ((unit + 1) % steps == 0) {
                const int m = m0 + threadIdx.x / FEATURES;
                const int n = (blockIdx.x + unit / steps * gridDim.x) * FEATURES + threadIdx.x % FEATURES;
                if (m < M && n < N) C[(int64_t)m * ldc + n] = total;
                total = 0.0f;
            }
        }
    }
}

template <int ROWS>
cudaError_t launch_rows(const float* A, int64_t lda, const float* W, int64_t ldw, float* C, int64_t ldc, int M, int N,
                        int K, cudaStream_t stream) {
    constexpr int bytes = (2 * WARPS * CHAINS * ROWS * FEATURES + WARPS * 2 * ROWS * KBLOCK) * 4;
    // (asked for on every call: the attribute is the current device's)
    const cudaError_t set = cudaFuncSetAttribute(gemm_f32_rows_kernel<ROWS>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (set != cudaSuccess) return set;
    const int tiles = (N + FEATURES - 1) / FEATURES, groups = (M + ROWS - 1) / ROWS;
    const dim3 grid(tiles < 296 ? tiles : 296, groups);              // two blocks on each of the 148 multiprocessors (of eight rows: one, in turn)
    return tb_launch_pdl(gemm_f32_rows_kernel<ROWS>, grid, dim3(WARPS * 32), bytes, stream, A, lda, W, ldw, C, ldc, M, N, K);
}

// Shared memory to ask for beyond a block's `own`, so that no multiprocessor takes more than its share of the tiles (`side`: the blocks
// that fit without).  The kernel is allowed the most that any product asks for, whatever this one does: another thread's may be
// on its way.
template <typename Kernel>
cudaError_t spread(Kernel kernel, int64_t tiles, int side, int own, size_t& extra) {
    auto beyond = [&](int64_t share) { return (int)(228 * 1024 / (share + 1) + 1024 - own); };
    const int64_t share = (tiles + 147) / 148;
    extra = share < side ? beyond(share) : 0;
    return extra == 0 ? cudaSuccess : cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, beyond(1));
}

template <bool VEC, int BM, int BN, int TN>
cudaError_t launch_tile(const float* A, int64_t lda, const float* W, int64_t ldw, float* C, int64_t ldc, int M, int N,
                        int K, cudaStream_t stream) {
    const dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    auto kernel = gemm_f32_tile_kernel<VEC, BM, BN, TN>;
    size_t extra;
    const cudaError_t set = spread(kernel, (int64_t)grid.x * grid.y, BM == 64 ? 4 : 2, 2 * BK * (BM + BN + 8) * 4, extra);
    if (set != cudaSuccess) return set;
    return tb_launch_pdl(kernel, grid, dim3((BM / 8) * (BN / TN)), extra, stream, A, lda, W, ldw, C, ldc, M, N, K);
}

template <bool VEC>
cudaError_t launch_even(const float* A, int64_t lda, const float* W, int64_t ldw, float* C, int64_t ldc, int M, int N,
                        int K, cudaStream_t stream) {
    const dim3 grid((N + 63) / 64, (M + 63) / 64);
    auto kernel = K <= EK ? gemm_f32_even_kernel<VEC, true> : gemm_f32_even_kernel<VEC, false>;
    size_t extra;
    const cudaError_t set = spread(kernel, (int64_t)grid.x * grid.y, K <= EK ? 4 : 2, 4 * EK * (64 + 4) * 4, extra);
    if (set != cudaSuccess) return set;
    return tb_launch_pdl(kernel, grid, dim3(256), extra, stream, A, lda, W, ldw, C, ldc, M, N, K);
}

template <int BM, int BN, int TN, int G>
cudaError_t launch_groups(const float* A, int64_t lda, const float* W, int64_t ldw, float* C, int64_t ldc, int M, int N,
                          int K, cudaStream_t stream) {
    constexpr int threads = (BM / 8) * (BN / TN);
    constexpr int bytes = (G * 2 * BK * (BM + BN + 8) + (G - 1) * BM * BN) * 4;
    const cudaError_t set = cudaFuncSetAttribute(gemm_f32_groups_kernel<BM, BN, TN, G>,
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (set != cudaSuccess) return set;
    const dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    return tb_launch_pdl(gemm_f32_groups_kernel<BM, BN, TN, G>, grid, dim3(threads * G), bytes, stream, A, lda, W, ldw, C, ldc, M,
                         N, K);
}

// ---- which form a product takes -------------------------------------------------------------------------------------
//
// The one whose estimated time is least.  The estimates are fits to 3,374 products (K 1 to 8,192, N 64 to 128,256, 1 to 2,048
// rows; operands on and off the packets' alignment), each form timed at each: 2 to 6 % off in the middle, 10 to 20 % at nine in
// ten, and the form they pick takes 1.004 of the best one's time on average, 1.25 at worst.  Against 64 x 64 tiles of one chain
// of K, which all products took before, a picked form is slower at some K of 33 to 127 alone, whose last stages are partly empty
// (K = 96: up to 1.18 times; K = 48: up to 1.2 times 3.6 us), and at K of 16 or less with 128,256 features (1.11).

enum Form : int { ROWS = 0, EVEN, SQUARE, TALL, SQUARE_GROUPS, TALL_GROUPS };

// Microseconds: to start, a tile of a multiprocessor, and a stage where a multiprocessor has one tile / for each of several;
// tiles that fit a multiprocessor side by side.
struct TileCost {
    float start, tile, one, many;
    int side;
};

float tiles_take(const TileCost& c, int64_t tiles, int stages) {
    const int64_t wave = 148 * c.side, whole = tiles / wave, left = (tiles % wave + 147) / 148;
    auto stage = [&](int64_t side_by_side) { return side_by_side == 0 ? 0.0f : fmaxf(c.one, c.many * side_by_side); };
    return c.start + c.tile * ((tiles + 147) / 148) + stages * (whole * stage(c.side) + stage(left));
}

// The streaming kernel: units of 16 features x 2,048 numbers of K, `unit` at an empty K, `full` more at a whole one, a pass over
// the weights for every eight rows at `megabyte` a megabyte.  A unit takes nearly the same whatever part of its K is there, so
// a short K is read as slowly as a long one: 48 rows of 2,048 x 128 take 23.1 us, as tiles 7.2.
float rows_take(int M, int N, int K) {
    const int which = M == 1 ? 0 : M == 2 ? 1 : M <= 4 ? 2 : 3, rows = 1 << which;
    static const float start[4] = {0.56f, 0.32f, 0.31f, 0.2f}, wave[4] = {0.0f, 0.0f, 0.0f, 1.02f};
    static const float unit[4] = {1.24f, 1.81f, 3.04f, 2.80f}, full[4] = {0.29f, 0.17f, 0.0f, 0.77f};
    static const float megabyte[4] = {0.141f, 0.167f, 0.207f, 0.226f};
    const int64_t tiles = (N + FEATURES - 1) / FEATURES, passes = (M + rows - 1) / rows;
    const int64_t slots = which == 3 ? 148 : 296, steps = (K + STEP - 1) / STEP;      // (blocks of eight rows fill a multiprocessor)
    const int64_t waves = ((tiles < 296 ? tiles : 296) * passes + slots - 1) / slots, units = (tiles * passes + slots - 1) / slots * steps;
    const float mb = 4e-6f * (float)N * (float)K * passes;
    return start[which] + fmaxf(waves * wave[which] + units * (unit[which] + full[which] * (K < STEP ? K : STEP) / STEP), megabyte[which] * mb);
}

// packets: rows of both operands start on 16 bytes and K is a multiple of four; streams: the weights' rows start on 32 bytes and K
// is a multiple of eight as well.
Form form_for(int M, int N, int K, bool packets, bool streams) {
    const int64_t across = (N + 63) / 64, square = (M + 63) / 64 * across, tall = (M + 127) / 128 * across;
    int stages = 0;                                // of 16 numbers of K, chain after chain
    for (int t = 0; t < 16; ++t) stages += stage_start(t) < K % KBLOCK;
    stages += K / KBLOCK * 16;
    Form best = K <= EK ? EVEN : SQUARE;
    float least = 0.0f;
    if (K <= EK)
        least = packets ? 0.56f + 0.06f * K + fmaxf(0.55f, 0.0055f * square) : 1.4f + 0.12f * K + fmaxf(0.2f, 0.00435f * square);
    else
        least = tiles_take(packets ? TileCost{1.65f, 0.04f, 0.66f, 0.504f, 4} : TileCost{1.2f, 0.49f, 0.85f, 0.71f, 4}, square, stages);
    auto consider = [&](Form form, float takes) {
        if (takes < least) {
            least = takes;
            best = form;
        }
    };
    if (K > EK) {
        if ((K < KBLOCK || !packets) && square <= 296)
            consider(EVEN, tiles_take(packets ? TileCost{0.85f, 0.14f, 1.49f, 1.26f, 2} : TileCost{0.17f, 0.0f, 1.69f, 1.46f, 2}, square, (K + EK - 1) / EK));
        consider(TALL, tiles_take(packets ? TileCost{2.0f, 0.51f, 0.964f, 0.835f, 2} : TileCost{2.06f, 0.0f, 1.256f, 1.105f, 2}, tall, stages));
        if (packets && K % KBLOCK == 0) {
            consider(SQUARE_GROUPS, tiles_take(TileCost{0.0f, 1.72f, 0.487f, 0.526f, 1}, square, stages));
            consider(TALL_GROUPS, tiles_take(TileCost{0.0f, 1.48f, 0.905f, 0.905f, 1}, tall, stages));
        }
    }
    if (streams && M <= kMostStreamed) consider(ROWS, rows_take(M, N, K));
    return best;
}

}  // namespace

// The form that tb_gemm_f32_nt takes: 0 streamed rows, 1 even tiles, 2 square tiles, 3 tall tiles, 4 and 5 those whose chains
// groups of threads share.
TB_EXPORT int tb_gemm_f32_form(int M, int N, int K, int packets, int streams) {
    return M < 1 || N < 1 || K < 1 ? -1 : (int)form_for(M, N, K, packets != 0, streams != 0);
}

// Zero padding inside a chain adds exact zeros, which leaves every partial sum unchanged, so the guarded and the packet
// paths and all kernels give the same bits.
TB_EXPORT int tb_gemm_f32_nt(const float* A, int64_t lda, const float* W, int64_t ldw, float* C, int64_t ldc,
                             int M, int N, int K, cudaStream_t stream) {
    if (M == 0 || N == 0) return 0;
    if (K <= 0) return TB_ERR_BAD_SIZE;
    if ((M + 63) / 64 > 65535) return TB_ERR_BAD_SIZE;
    const bool vec = (K % 4 == 0) && (lda % 4 == 0) && (ldw % 4 == 0) && ((uintptr_t)A % 16 == 0) &&
                     ((uintptr_t)W % 16 == 0);
    const bool streams = vec && K % 8 == 0 && ldw % 8 == 0 && (uintptr_t)W % 32 == 0;
    switch (form_for(M, N, K, vec, streams)) {
        case ROWS:
            if (M == 1) return (int)launch_rows<1>(A, lda, W, ldw, C, ldc, M, N, K, stream);
            if (M == 2) return (int)launch_rows<2>(A, lda, W, ldw, C, ldc, M, N, K, stream);
            if (M <= 4) return (int)launch_rows<4>(A, lda, W, ldw, C, ldc, M, N, K, stream);
            return (int)launch_rows<8>(A, lda, W, ldw, C, ldc, M, N, K, stream);
        case EVEN:
            return (int)(vec ? launch_even<true>(A, lda, W, ldw, C, ldc, M, N, K, stream)
                             : launch_even<false>(A, lda, W, ldw, C, ldc, M, N, K, stream));
        case SQUARE:
            return (int)(vec ? launch_tile<true, 64, 64, 4>(A, lda, W, ldw, C, ldc, M, N, K, stream)
                             : launch_tile<false, 64, 64, 4>(A, lda, W, ldw, C, ldc, M, N, K, stream));
        case TALL:
            return (int)(vec ? launch_tile<true, 128, 64, 8>(A, lda, W, ldw, C, ldc, M, N, K, stream)
                             : launch_tile<false, 128, 64, 8>(A, lda, W, ldw, C, ldc, M, N, K, stream));
        case SQUARE_GROUPS:
            return (int)launch_groups<64, 64, 8, 4>(A, lda, W, ldw, C, ldc, M, N, K, stream);
        default:
            return (int)launch_groups<128, 64, 8, 2>(A, lda, W, ldw, C, ldc, M, N, K, stream);
    }
}
