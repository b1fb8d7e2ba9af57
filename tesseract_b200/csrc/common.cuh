// Shared device helpers for the sm_100a kernels of this package.
//
// Every kernel file is compiled on its own into a small shared library with
// plain C entry points (no framework headers), so that a model compiles only the
// kernels it needs and a fresh checkout builds in seconds.  Entry points return
// 0 on success or a negative code for a refused size / a positive cudaError_t.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#define TB_EXPORT extern "C" __attribute__((visibility("default")))

// Refusal codes (negative so that they never collide with cudaError_t values).
#define TB_ERR_BAD_DTYPE (-2)
#define TB_ERR_BAD_SIZE (-3)
#define TB_ERR_BAD_ALIGN (-4)

enum TbDtype : int { TB_F32 = 0, TB_BF16 = 1 };

// Programmatic dependent launch.  A kernel started with tb_launch_pdl may begin while the kernel before it in
// the stream is still draining; everything it does before pdl_wait() must not depend on that kernel's results
// (reading weights is fine).  pdl_trigger() in a kernel lets the next such kernel start early.  Both are no-ops
// for kernels launched the ordinary way.  A kernel that reads more than weights before pdl_wait() (where a row lies: positions,
// block tables) is started with tb_launch, early only if its caller vouches that no kernel in front may still be writing that.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... KernelArgs, typename... Args>
static inline cudaError_t tb_launch(bool early, void (*kernel)(KernelArgs...), dim3 grid, dim3 block, size_t smem,
                                    cudaStream_t stream, Args... args) {
    cudaLaunchConfig_t config = {};
    config.gridDim = grid;
    config.blockDim = block;
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    cudaLaunchAttribute attribute[1];
    attribute[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute[0].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attribute;
    config.numAttrs = early ? 1 : 0;
    return cudaLaunchKernelEx(&config, kernel, KernelArgs(args)...);
}

template <typename... KernelArgs, typename... Args>
static inline cudaError_t tb_launch_pdl(void (*kernel)(KernelArgs...), dim3 grid, dim3 block, size_t smem,
                                        cudaStream_t stream, Args... args) {
    return tb_launch(true, kernel, grid, block, smem, stream, args...);
}

// Where a key lies in pages of `size` tokens, without a division or a branch (a thread of the attention kernels looks up four to eight keys
// a tile, and a branch to a division or a shift at each made portions of 20 tokens a tenth slower).  With 2^l the smallest power of two that is not below size,
// N = 32 + max(l - 1, 0) and m = (2^N - 1) / size rounded down (m < 2^32), (key + 1) * m / 2^N rounded down is key / size for every
// key and size below 2^31: m * size = 2^N - 1 - r with r < size, so the quotient falls short of (key + 1) / size by
// (key + 1) * (r + 1) / (size * 2^N), which is more than nothing and, as (key + 1) * (r + 1) <= 2^31 * 2^l, no more than 1 / size.
struct Paging {
    uint32_t inverse;
    int shift, size;
    __device__ __forceinline__ int page_of(int key) const { return (int)(__umulhi((uint32_t)key + 1u, inverse) >> shift); }
    __device__ __forceinline__ int within(int key) const { return key - page_of(key) * size; }
};
static inline Paging tb_paging(int page_size) {
    Paging p = {0, 0, page_size};
    while (((int64_t)2 << p.shift) < page_size) ++p.shift;
    p.inverse = (uint32_t)((((uint64_t)1 << (32 + p.shift)) - 1) / (uint64_t)page_size);
    return p;
}

static inline int tb_launch_status() {
    cudaError_t err = cudaGetLastError();
    return err == cudaSuccess ? 0 : (int)err;
}

template <typename T>
struct Elem;

template <>
struct Elem<float> {
    static __device__ __forceinline__ float load(const float* p) { return *p; }
    static __device__ __forceinline__ void store(float* p, float v) { *p = v; }
    // Value an element takes when written and read back (identity in 32-bit).
    static __device__ __forceinline__ float round(float v) { return v; }
};

template <>
struct Elem<__nv_bfloat16> {
    static __device__ __forceinline__ float load(const __nv_bfloat16* p) { return __bfloat162float(*p); }
    static __device__ __forceinline__ void store(__nv_bfloat16* p, float v) { *p = __float2bfloat16_rn(v); }
    static __device__ __forceinline__ float round(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }
};

// 16-byte packets: 8 bfloat16 or 4 floats.
template <typename T>
struct Packet;
template <>
struct Packet<float> {
    static constexpr int N = 4;
    static __device__ __forceinline__ void load(const float* p, float* v) {
        const float4 t = *reinterpret_cast<const float4*>(p);
        v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    }
    static __device__ __forceinline__ void store(float* p, const float* v) {
        *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
    }
    // a packet kept as it was loaded (16 bytes) and taken apart later
    static __device__ __forceinline__ void unpack(const uint4& t, float* v) {
        v[0] = __uint_as_float(t.x); v[1] = __uint_as_float(t.y); v[2] = __uint_as_float(t.z); v[3] = __uint_as_float(t.w);
    }
};
template <>
struct Packet<__nv_bfloat16> {
    static constexpr int N = 8;
    static __device__ __forceinline__ void load(const __nv_bfloat16* p, float* v) {
        const uint4 t = *reinterpret_cast<const uint4*>(p);
        const uint32_t w[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            v[2 * i] = __uint_as_float(w[i] << 16);
            v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
        }
    }
    static __device__ __forceinline__ void unpack(const uint4& t, float* v) {
        const uint32_t w[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            v[2 * i] = __uint_as_float(w[i] << 16);
            v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
        }
    }
    static __device__ __forceinline__ void store(__nv_bfloat16* p, const float* v) {
        uint32_t w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
            w[i] = *reinterpret_cast<uint32_t*>(&h);
        }
        *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
    }
};

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Block-wide sum with a fixed reduction tree (depends only on blockDim), so that
// a row's statistic does not depend on what else is in the batch.
// `scratch` must hold 32 floats.  Every thread receives the result.
__device__ __forceinline__ float block_sum(float v, float* scratch) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int warps = (blockDim.x + 31) >> 5;
    v = warp_sum(v);
    __syncthreads();
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    float t = (lane < warps) ? scratch[lane] : 0.0f;
    t = warp_sum(t);
    return t;
}

__device__ __forceinline__ float block_max(float v, float* scratch) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int warps = (blockDim.x + 31) >> 5;
    v = warp_max(v);
    __syncthreads();
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    float t = (lane < warps) ? scratch[lane] : -INFINITY;
    t = warp_max(t);
    return t;
}
