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
__device__ __forceinline__ int stage_start(int t) { return (t >> 4) * KBLOCK + (t & 3) * 64 + ((t >> 2) & 3) * 8; }
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

    pdl_trigger();
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
    store_tile<BM, BN, TN>(total, C, ldc, m0, n0, tx, ty, M, N);
}

// The tiles where they are too few to give a multiprocessor more than one: G groups of threads take a tile's chains in turn (K a
// multiple of 256, packets), and the first group adds the sums in the order of the chains, the others' through
// shared memory, so that the bits are those of the kernel above.  Bound by the latency of a group's stages, which the groups hide
// from one another.   128 x 64
// tiles of two groups and 64 x 64 tiles of four take 121 and 72 us for K = 2,048 (one group, where a multiprocessor has one tile:
// 141 and 95).
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
    pdl_trigger();
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
    if (group > 0) return;
    store_tile<BM, BN, TN>(total, C, ldc, m0, n0, tx, ty, M, N);
}

// ---- few rows: the weights stream through registers -----------------------------------------------------------------

constexpr int WARPS = 8, FEATURES = 16;                // a block: 16 weight rows, eight blocks of K at a time
constexpr int STEP = WARPS * KBLOCK;
constexpr int AHEAD = 4;                               // groups of weights in flight a thread

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
// 64 x 64 tiles 189), by multiply-adds and loads of the rows from shared memory above (33 us at eight, a further 31 for
// every eight).  2,048 x 8,192 takes 13 to 19 us up to eight rows (the tiles 581), the head of 128,256 x 2,048 at one row
// 151 (961).  Registers hold four groups of weights in flight a thread, 128 KiB a multiprocessor.
// Lane (f, c) runs chain c of its warp's block for the weight rows f and f + 8 and ROWS rows of A.  The rows' part that
// a warp needs lies in shared memory that only this warp writes and reads.
template <int ROWS>
__global__ void __launch_bounds__(WARPS * 32, 2)
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
    const dim3 grid(tiles < 296 ? tiles : 296, groups);              // two blocks on each of the 148 multiprocessors
    return tb_launch_pdl(gemm_f32_rows_kernel<ROWS>, grid, dim3(WARPS * 32), bytes, stream, A, lda, W, ldw, C, ldc, M, N, K);
}

template <bool VEC, int BM, int BN, int TN>
cudaError_t launch_tile(const float* A, int64_t lda, const float* W, int64_t ldw, float* C, int64_t ldc, int M, int N,
                        int K, cudaStream_t stream) {
    const dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    return tb_launch_pdl(gemm_f32_tile_kernel<VEC, BM, BN, TN>, grid, dim3((BM / 8) * (BN / TN)), 0, stream, A, lda, W, ldw,
                         C, ldc, M, N, K);
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

}  // namespace

// Zero padding inside a chain adds exact zeros, which leaves every partial sum unchanged, so the guarded and the packet
// paths and both kernels give the same bits.
TB_EXPORT int tb_gemm_f32_nt(const float* A, int64_t lda, const float* W, int64_t ldw, float* C, int64_t ldc,
                             int M, int N, int K, cudaStream_t stream) {
    if (M == 0 || N == 0) return 0;
    if (K <= 0) return TB_ERR_BAD_SIZE;
    if ((M + 63) / 64 > 65535) return TB_ERR_BAD_SIZE;
    const bool vec = (K % 4 == 0) && (lda % 4 == 0) && (ldw % 4 == 0) && ((uintptr_t)A % 16 == 0) &&
                     ((uintptr_t)W % 16 == 0);
    const int64_t tall = (int64_t)((M + 127) / 128) * ((N + 63) / 64), square = (int64_t)((M + 63) / 64) * ((N + 63) / 64);
    // Streaming passes over the weights once for every eight rows, a tile takes 0.7 us for sixteen numbers of K whatever
    // else runs.  At N x K = 16,384 x 2,048 the two meet near 50 rows (32: 126 against 198 us, 64: 248 against 229); with
    // few tiles later (3,072 x 2,048, 64 rows: 54 against 100; 2,048 x 8,192, 64 rows: 109 against 398; 2,048 x 2,048,
    // 200 rows, 128 tiles: 112 against 94).  A short K leaves most of a streaming block's warps without work.
    const bool stream_weights = M <= 48 || (square <= 80 && K >= STEP);
    if (stream_weights && vec && K % 8 == 0 && ldw % 8 == 0 && (uintptr_t)W % 32 == 0) {
        if (M == 1) return (int)launch_rows<1>(A, lda, W, ldw, C, ldc, M, N, K, stream);
        if (M == 2) return (int)launch_rows<2>(A, lda, W, ldw, C, ldc, M, N, K, stream);
        if (M <= 4) return (int)launch_rows<4>(A, lda, W, ldw, C, ldc, M, N, K, stream);
        return (int)launch_rows<8>(A, lda, W, ldw, C, ldc, M, N, K, stream);
    }
    if (!vec) return (int)launch_tile<false, 64, 64, 4>(A, lda, W, ldw, C, ldc, M, N, K, stream);
    // One tile a multiprocessor: groups of threads share its chains.  200 rows of 2,048 x 2,048 (128 square tiles) 94 -> 72 us,
    // 160 of 3,072 x 2,048 171 -> 72, 64 rows of 16,384 x 2,048 (tall tiles would be half empty) 220 -> 158; 380 rows of
    // 3,072 x 2,048 (144 tall tiles) 188 -> 130, 500 of 2,048 x 2,048 203 -> 121.  With more tiles two of one group share a
    // multiprocessor, which is faster (380 rows of 16,384 x 2,048: 684 against 787).
    if (K % KBLOCK == 0 && (square <= 148 || M <= 64)) return (int)launch_groups<64, 64, 8, 4>(A, lda, W, ldw, C, ldc, M, N, K, stream);
    if (K % KBLOCK == 0 && tall <= 148) return (int)launch_groups<128, 64, 8, 2>(A, lda, W, ldw, C, ldc, M, N, K, stream);
    // Tall tiles load less from shared memory for a product but leave the chip emptier: 200 rows of 2,048 x 2,048 (64 of
    // them) take 139 us, as square tiles 94; 380 rows (96) 141 against 145, and 547 against 566 at K = 8,192.
    if (tall >= 96) return (int)launch_tile<true, 128, 64, 8>(A, lda, W, ldw, C, ldc, M, N, K, stream);
    return (int)launch_tile<true, 64, 64, 4>(A, lda, W, ldw, C, ldc, M, N, K, stream);
}
