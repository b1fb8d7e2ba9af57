// Plain paged attention: one warp (in steps of few rows a block) per (query row, query head), keys walked in ascending
// blocks of 32 through the request's block table.  It serves the 32-bit path of every
// model and any size the fast bfloat16 kernels refuse.
//
// For row r at absolute position p of request q, head h (kv head h / group):
//   keys j in [max(0, p - window + 1), p]   (window <= 0: all keys; causal by construction)
//   s_j = (q_r . k_j) * scale ; masked lanes -1e30
//   streaming softmax per block: m' = max(m, max s); p_j = exp(s_j - m');
//   l = l*exp(m - m') + sum p ; acc = acc*exp(m - m') + sum round(p_j) * v_j
//   out = round(acc / max(l, 1e-8))
// as the reference's ragged attention does with blocks of 16 (src/cuda/kernels.rs:447-562).
// Scores, softmax state and the accumulator are 32-bit.  The order of every reduction depends
// only on (p, window, head_dim): not on the batch, the cut of the prompt, or the page ids.
#include "common.cuh"

namespace {

constexpr int kWarpsPerBlock = 4;
constexpr int kKeyBlock = 32;
constexpr int kFewBlocks = 592;      // up to four blocks a multiprocessor

template <typename T>
struct Vec16;
template <>
struct Vec16<float> {
    static constexpr int N = 4;
    static __device__ __forceinline__ void load(const float* p, float* out) {
        const float4 v = *reinterpret_cast<const float4*>(p);
        out[0] = v.x; out[1] = v.y; out[2] = v.z; out[3] = v.w;
    }
};
template <>
struct Vec16<__nv_bfloat16> {
    static constexpr int N = 8;
    static __device__ __forceinline__ void load(const __nv_bfloat16* p, float* out) {
        const uint4 v = *reinterpret_cast<const uint4*>(p);
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            out[2 * i] = __uint_as_float(w[i] << 16);
            out[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
        }
    }
};

// UNDER: loads under way at a time (packets of a key, values of a block); 0: as they are needed, and none for a key without weight.
template <typename T, int NC, int UNDER>
__global__ void __launch_bounds__(kWarpsPerBlock * 32)
attention_rows_kernel(const T* __restrict__ q, int64_t q_stride, T* __restrict__ out, int64_t out_stride,
                      const T* __restrict__ cache, const int* __restrict__ positions,
                      const int* __restrict__ seq_of_row, const int* __restrict__ block_table, int bt_stride,
                      int num_heads, int num_kv_heads, int head_dim, int page_size, int window, float scale) {
    extern __shared__ float q_smem[];  // kWarpsPerBlock * head_dim
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row = blockIdx.x;
    const int head = blockIdx.y * kWarpsPerBlock + warp;
    if (head >= num_heads) return;  // whole warp leaves together; no block-wide barrier below
    const int kv_head = head / (num_heads / num_kv_heads);
    const int pos = positions[row];
    const int seq = seq_of_row[row];
    const int first_key = (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;

    float* qs = q_smem + warp * head_dim;
    const T* qrow = q + (int64_t)row * q_stride + (int64_t)head * head_dim;
    for (int i = lane; i < head_dim; i += 32) qs[i] = Elem<T>::load(qrow + i);
    __syncwarp();

    const int64_t head_block = (int64_t)page_size * head_dim;
    const int64_t page_block = 2 * (int64_t)num_kv_heads * head_block;
    const T* kbase = cache + (int64_t)kv_head * head_block;
    const T* vbase = kbase + (int64_t)num_kv_heads * head_block;
    const int* table = block_table + (int64_t)seq * bt_stride;

    float m = -1.0e30f, l = 0.0f;
    float acc[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) acc[c] = 0.0f;

    for (int kb = first_key / kKeyBlock; kb * kKeyBlock <= pos; ++kb) {
        const int key = kb * kKeyBlock + lane;
        const bool valid = key >= first_key && key <= pos;
        int64_t key_offset = 0;
        float s = -1.0e30f;
        if (valid) {
            const int page = table[key / page_size];
            key_offset = (int64_t)page * page_block + (int64_t)(key % page_size) * head_dim;
            const T* kp = kbase + key_offset;
            float dot = 0.0f;
            if constexpr (UNDER == 0) {
                float kv[Vec16<T>::N];
                for (int i = 0; i < head_dim; i += Vec16<T>::N) {
                    Vec16<T>::load(kp + i, kv);
#pragma unroll
                    for (int e = 0; e < Vec16<T>::N; ++e) dot = fmaf(qs[i + e], kv[e], dot);
                }
            } else {
                // (UNDER packets asked for at a time; the sum runs on in order)
                for (int i0 = 0; i0 < head_dim; i0 += UNDER * Vec16<T>::N) {
                    float kv[UNDER][Vec16<T>::N];
#pragma unroll
                    for (int u = 0; u < UNDER; ++u)
                        if (i0 + u * Vec16<T>::N < head_dim) Vec16<T>::load(kp + i0 + u * Vec16<T>::N, kv[u]);
#pragma unroll
                    for (int u = 0; u < UNDER; ++u)
                        if (i0 + u * Vec16<T>::N < head_dim) {
#pragma unroll
                            for (int e = 0; e < Vec16<T>::N; ++e) dot = fmaf(qs[i0 + u * Vec16<T>::N + e], kv[u][e], dot);
                        }
                }
            }
            s = dot * scale;
        }
        const float m_new = fmaxf(m, warp_max(s));
        const float p = valid ? expf(s - m_new) : 0.0f;
        const float corr = expf(m - m_new);
        l = l * corr + warp_sum(p);
#pragma unroll
        for (int c = 0; c < NC; ++c) acc[c] *= corr;
        const float p_mma = Elem<T>::round(p);
        const int keys_here = min(kKeyBlock, pos - kb * kKeyBlock + 1);
        if constexpr (UNDER == 0) {
            for (int j = 0; j < keys_here; ++j) {
                const float pj = __shfl_sync(0xffffffffu, p_mma, j);
                const int64_t off = __shfl_sync(0xffffffffu, key_offset, j);
                if (pj != 0.0f) {  // uniform across the warp; masked keys contribute nothing
                    const T* vp = vbase + off;
#pragma unroll
                    for (int c = 0; c < NC; ++c) {
                        const int col = c * 32 + lane;
                        if (col < head_dim) acc[c] = fmaf(pj, Elem<T>::load(vp + col), acc[c]);
                    }
                }
            }
        } else {
            for (int j0 = 0; j0 < keys_here; j0 += UNDER) {
                float v[UNDER][NC];
#pragma unroll
                for (int u = 0; u < UNDER; ++u) {
                    const T* vp = vbase + __shfl_sync(0xffffffffu, key_offset, j0 + u);    // (a lane without a key: offset 0, not used)
#pragma unroll
                    for (int c = 0; c < NC; ++c)
                        if (j0 + u < keys_here && c * 32 + lane < head_dim) v[u][c] = Elem<T>::load(vp + c * 32 + lane);
                }
#pragma unroll
                for (int u = 0; u < UNDER; ++u) {
                    const float pj = __shfl_sync(0xffffffffu, p_mma, j0 + u);
                    if (j0 + u < keys_here && pj != 0.0f) {  // uniform across the warp; masked keys contribute nothing
#pragma unroll
                        for (int c = 0; c < NC; ++c)
                            if (c * 32 + lane < head_dim) acc[c] = fmaf(pj, v[u][c], acc[c]);
                    }
                }
            }
        }
        m = m_new;
    }
    const float denom = fmaxf(l, 1.0e-8f);
    T* orow = out + (int64_t)row * out_stride + (int64_t)head * head_dim;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        const int col = c * 32 + lane;
        if (col < head_dim) Elem<T>::store(orow + col, acc[c] / denom);
    }
}

// The same work, to the bit, by a block a (row, head): eight warps take the scores of its key blocks side by side and leave them in
// shared memory; since a running maximum is the same maximum however it is found, the weights of all blocks follow side by side as
// well; what is left to go in order, block by block and key by key, is the sum over the weights and that over the values, a warp 32
// columns of it, the next block's values on their way.  Runs of kRun blocks, so that any context fits.
constexpr int kSharedWarps = 8, kRun = 64;

template <typename T, int NC>
__global__ void __launch_bounds__(kSharedWarps * 32, 2)
attention_rows_shared_kernel(const T* q, int64_t q_stride, T* out, int64_t out_stride, const T* cache,
                             const int* __restrict__ positions, const int* __restrict__ seq_of_row,
                             const int* __restrict__ block_table, int bt_stride, int num_heads, int num_kv_heads, int head_dim,
                             int page_size, int window, float scale) {
    constexpr int UNDER = sizeof(T) == 4 ? 8 : 1;    // packets of a key under way (bfloat16: four at a time spilled, and took 4 to 14 % longer)
    __shared__ float score[kRun * kKeyBlock];        // then the weights
    __shared__ int64_t offset[kRun * kKeyBlock];     // of a key in its half of the cache
    __shared__ float block_max[kRun], block_sum_of[kRun], max_so_far[kRun], qs[NC * 32];
    pdl_trigger();
    pdl_wait();                                      // rows, keys and the step's metadata come from kernels in front
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row = blockIdx.x, head = blockIdx.y, kv_head = head / (num_heads / num_kv_heads);
    const int pos = positions[row];
    const int first_key = (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;
    const int* table = block_table + (int64_t)seq_of_row[row] * bt_stride;
    const T* qrow = q + (int64_t)row * q_stride + (int64_t)head * head_dim;
    for (int i = threadIdx.x; i < head_dim; i += kSharedWarps * 32) qs[i] = Elem<T>::load(qrow + i);
    __syncthreads();
    const int64_t head_block = (int64_t)page_size * head_dim;
    const int64_t page_block = 2 * (int64_t)num_kv_heads * head_block;
    const T* kbase = cache + (int64_t)kv_head * head_block;
    const T* vbase = kbase + (int64_t)num_kv_heads * head_block;
    const int col = warp * 32 + lane;
    const bool has_columns = warp < NC;

    float m = -1.0e30f, l = 0.0f, acc = 0.0f;
    const int last_block = pos / kKeyBlock;
    for (int kb0 = first_key / kKeyBlock; kb0 <= last_block; kb0 += kRun) {
        const int blocks = min(kRun, last_block - kb0 + 1);
        for (int b = warp; b < blocks; b += kSharedWarps) {
            const int key = (kb0 + b) * kKeyBlock + lane;
            const bool valid = key >= first_key && key <= pos;
            int64_t at = 0;
            float s = -1.0e30f;
            if (valid) {
                at = (int64_t)table[key / page_size] * page_block + (int64_t)(key % page_size) * head_dim;
                const T* kp = kbase + at;
                float dot = 0.0f;
                for (int i0 = 0; i0 < head_dim; i0 += UNDER * Vec16<T>::N) {
                    float kv[UNDER][Vec16<T>::N];
#pragma unroll
                    for (int u = 0; u < UNDER; ++u)
                        if (i0 + u * Vec16<T>::N < head_dim) Vec16<T>::load(kp + i0 + u * Vec16<T>::N, kv[u]);
#pragma unroll
                    for (int u = 0; u < UNDER; ++u)
                        if (i0 + u * Vec16<T>::N < head_dim) {
#pragma unroll
                            for (int e = 0; e < Vec16<T>::N; ++e) dot = fmaf(qs[i0 + u * Vec16<T>::N + e], kv[u][e], dot);
                        }
                }
                s = dot * scale;
            }
            score[b * kKeyBlock + lane] = s;
            offset[b * kKeyBlock + lane] = at;
            s = warp_max(s);
            if (lane == 0) block_max[b] = s;
        }
        __syncthreads();
        float v[2][kKeyBlock];
        auto ask = [&](int b, float (&to)[kKeyBlock]) {
            if (!has_columns || b >= blocks) return;
            const int keys = min(kKeyBlock, pos - (kb0 + b) * kKeyBlock + 1);
#pragma unroll
            for (int j = 0; j < kKeyBlock; ++j)
                to[j] = j < keys && col < head_dim ? Elem<T>::load(vbase + offset[b * kKeyBlock + j] + col) : 0.0f;
        };
        ask(0, v[0]);
        for (int b = warp; b < blocks; b += kSharedWarps) {
            float before = -1.0e30f;
            for (int i = lane; i < b; i += 32) before = fmaxf(before, block_max[i]);
            const float m_new = fmaxf(fmaxf(m, warp_max(before)), block_max[b]);
            const int key = (kb0 + b) * kKeyBlock + lane;
            const float p = key >= first_key && key <= pos ? expf(score[b * kKeyBlock + lane] - m_new) : 0.0f;
            const float sum = warp_sum(p);
            score[b * kKeyBlock + lane] = Elem<T>::round(p);
            if (lane == 0) {
                block_sum_of[b] = sum;
                max_so_far[b] = m_new;
            }
        }
        __syncthreads();
        if (has_columns) {
            auto take = [&](int b, const float (&values)[kKeyBlock]) {
                const float m_new = max_so_far[b], corr = expf(m - m_new);
                l = l * corr + block_sum_of[b];
                acc *= corr;
                const int keys = min(kKeyBlock, pos - (kb0 + b) * kKeyBlock + 1);
#pragma unroll
                for (int j = 0; j < kKeyBlock; ++j) {
                    const float pj = score[b * kKeyBlock + j];
                    if (j < keys && pj != 0.0f) acc = fmaf(pj, values[j], acc);
                }
                m = m_new;
            };
            for (int b = 0; b < blocks; b += 2) {
                ask(b + 1, v[1]);
                take(b, v[0]);
                if (b + 1 >= blocks) break;
                ask(b + 2, v[0]);
                take(b + 1, v[1]);
            }
        }
        m = max_so_far[blocks - 1];
        __syncthreads();                             // (the next run writes over this one's scores)
    }
    if (has_columns && col < head_dim)
        Elem<T>::store(out + (int64_t)row * out_stride + (int64_t)head * head_dim + col, acc / fmaxf(l, 1.0e-8f));
}

template <typename T>
int launch(const void* q, int64_t q_stride, void* out, int64_t out_stride, const void* cache,
           const int* positions, const int* seq_of_row, const int* block_table, int bt_stride, int rows,
           int num_heads, int num_kv_heads, int head_dim, int page_size, int reach, int window, float scale,
           cudaStream_t stream) {
    // Few rows by a block, us against a warp a (row, head).  32-bit, up to 296 blocks (two fit a multiprocessor): 32 heads of 64
    // behind 130 keys, 4 / 8 / 16 rows 9.4 / 9.6 / 18.5 against 16.4 / 16.4 / 16.5, 4 rows behind 5,000 251 against 614.  Above 64
    // numbers also where the blocks take two turns, unless the keys are few: 32 rows of 16 heads of 128 behind 130 / 48 / 30 / 16 keys
    // 24.0 / 11.9 / 9.2 / 8.6 against 28.4 / 12.4 / 8.4 / 6.4.  bfloat16, up to 296 blocks: 4 rows of 32 heads of 64 behind 130 keys
    // 18.5 against 23.2, behind 12 6.2 against 4.7; 4 of 16 heads of 256 behind 16 8.5 against 11.1; heads of 32 and less behind any
    // keys longer (17.6 against 14.2).
    const int most = sizeof(T) == 4 ? (head_dim > 64 && reach > 32 ? 592 : 296) : head_dim > (reach > 16 ? 32 : 64) ? 296 : 0;
    if ((int64_t)rows * num_heads <= most) {
        auto kernel = head_dim <= 32 ? attention_rows_shared_kernel<T, 1> : head_dim <= 64 ? attention_rows_shared_kernel<T, 2>
                    : head_dim <= 128 ? attention_rows_shared_kernel<T, 4> : attention_rows_shared_kernel<T, 8>;
        const cudaError_t launched = tb_launch_pdl(kernel, dim3(rows, num_heads), dim3(kSharedWarps * 32), (size_t)0, stream, (const T*)q,
                                                   q_stride, (T*)out, out_stride, (const T*)cache, positions, seq_of_row, block_table,
                                                   bt_stride, num_heads, num_kv_heads, head_dim, page_size, window, scale);
        return launched == cudaSuccess ? tb_launch_status() : (int)launched;
    }
    dim3 grid(rows, (num_heads + kWarpsPerBlock - 1) / kWarpsPerBlock);
    const size_t smem = (size_t)kWarpsPerBlock * head_dim * sizeof(float);
#define TB_LAUNCH(NC, UNDER)                                                                                          \
    attention_rows_kernel<T, NC, UNDER><<<grid, kWarpsPerBlock * 32, smem, stream>>>(                                 \
        (const T*)q, q_stride, (T*)out, out_stride, (const T*)cache, positions, seq_of_row, block_table,       \
        bt_stride, num_heads, num_kv_heads, head_dim, page_size, window, scale)
    // Few warps a multiprocessor are bound by the latency of their loads, and more under way shorten it: 4 rows of 32 heads of 64 behind
    // some 100 keys (which the blocks above take by now) 13.4 us in 32-bit with 32 under way, 30.7 as they are needed.  The registers that this
    // takes hold back other warps as soon as there are more: 64 rows of 32 heads of 128 behind 300 keys, 32-bit, 8 / 16 under way or
    // as needed 140 / 288 / 251.  So 592 blocks, four a multiprocessor, take the form that was the fastest or close to it over all
    // of them (32-bit: 0.4 to 0.8 of the time as needed, bfloat16 0.65 to 0.9), and steps that fill the chip take few or none:
    // 600 rows of 8 heads of 32 behind up to 1,500 keys 359 us as needed, 395 with two; of 256 in bfloat16 1,462 and 1,681 with one.
    // The engine takes this kernel in 32-bit; bfloat16 callers have heads that the tensor-core kernels are not built for.
    constexpr bool wide = sizeof(T) == 4;
    const int64_t blocks = (int64_t)rows * grid.y;
    const bool few = blocks <= kFewBlocks, some = blocks <= 2 * kFewBlocks;
    if (head_dim <= 32) {
        if (few) TB_LAUNCH(1, (wide ? 16 : 8));
        else TB_LAUNCH(1, 0);
    } else if (head_dim <= 64) {
        if (few) TB_LAUNCH(2, (wide ? 32 : 4));
        else TB_LAUNCH(2, (wide ? 2 : 1));
    } else if (head_dim <= 128) {
        // (bfloat16: one under way where its blocks, ten a multiprocessor, take no more waves than the twelve without)
        if (wide && few) TB_LAUNCH(4, (wide ? 8 : 1));
        else if (wide ? some : (blocks + 1479) / 1480 <= (blocks + 1775) / 1776) TB_LAUNCH(4, (wide ? 2 : 1));
        else TB_LAUNCH(4, 0);
    } else {
        if (few) TB_LAUNCH(8, (wide ? 8 : 4));
        else if (wide && some) TB_LAUNCH(8, (wide ? 2 : 0));
        else TB_LAUNCH(8, 0);
    }
#undef TB_LAUNCH
    return tb_launch_status();
}

}  // namespace

// q: rows x (num_heads*head_dim) with row stride q_stride (elements); out likewise.
// cache: base of the cache entry, [page][K|V][kv_head][page_size][head_dim].
// head_dim must be a multiple of 8 (16-byte key rows) and at most 256.  reach: the keys that a request's table can hold, at
// most (it picks the form only; both give the same bits).
TB_EXPORT int tb_attention_rows(const void* q, int64_t q_stride, void* out, int64_t out_stride, const void* cache,
                                const int* positions, const int* seq_of_row, const int* block_table,
                                int bt_stride, int rows, int num_heads, int num_kv_heads, int head_dim,
                                int page_size, int reach, int window, float scale, int dtype, cudaStream_t stream) {
    if (rows == 0) return 0;
    if (head_dim <= 0 || head_dim > 256 || head_dim % 8 != 0) return TB_ERR_BAD_SIZE;
    if (num_kv_heads <= 0 || num_heads % num_kv_heads != 0) return TB_ERR_BAD_SIZE;
    if ((uintptr_t)cache % 16 != 0) return TB_ERR_BAD_ALIGN;
    if (dtype == TB_F32)
        return launch<float>(q, q_stride, out, out_stride, cache, positions, seq_of_row, block_table, bt_stride,
                             rows, num_heads, num_kv_heads, head_dim, page_size, reach, window, scale, stream);
    if (dtype == TB_BF16)
        return launch<__nv_bfloat16>(q, q_stride, out, out_stride, cache, positions, seq_of_row, block_table,
                                     bt_stride, rows, num_heads, num_kv_heads, head_dim, page_size, reach, window,
                                     scale, stream);
    return TB_ERR_BAD_DTYPE;
}
