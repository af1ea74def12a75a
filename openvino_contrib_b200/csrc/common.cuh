// Shared device helpers of the attention kernels (sm_100a only).
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

#include "b2a.h"

namespace b2a {

template <typename T>
__device__ __forceinline__ float to_f32(T x);
template <>
__device__ __forceinline__ float to_f32<float>(float x) { return x; }
template <>
__device__ __forceinline__ float to_f32<__half>(__half x) { return __half2float(x); }
template <>
__device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 x) { return __bfloat162float(x); }

template <typename T>
__device__ __forceinline__ T from_f32(float x);
template <>
__device__ __forceinline__ float from_f32<float>(float x) { return x; }
template <>
__device__ __forceinline__ __half from_f32<__half>(float x) { return __float2half_rn(x); }
template <>
__device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float x) { return __float2bfloat16_rn(x); }

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ void report(int32_t* status, uint32_t bits) {
    if (status != nullptr) atomicOr(reinterpret_cast<unsigned int*>(status), bits);
}

// The four int32 tables of a paged step plus the pool geometry.
struct PagedTables {
    const int32_t* past_lens;
    const int32_t* subsequence_begins;
    const int32_t* block_indices;
    const int32_t* block_indices_begins;
    int32_t num_seqs, num_tokens, num_blocks_total, block_size;
};

// Layout of one u8 chunk [block_size*D values | block_size f16 scales | block_size f16 zero-points].
__host__ __device__ __forceinline__ size_t u8_chunk_bytes(int block_size, int d) {
    return static_cast<size_t>(block_size) * (d + 4);
}

constexpr float kLog2e = 1.4426950408889634f;

// Two probabilities as packed pieces of T, for a second product on the tensor core that keeps float32's precision.
//   f16: p = hi + lo 2^-11, eleven bits each, and lo in an accumulator of its own: with one scale for both, the
//     probabilities of many keys beside one that stands far above them fall below f16's smallest value (32768 equal keys 17.4
//     below one with a zero value row: 3 % off).  The caller scales p by a power of two, to 2^15 at most, which its row sum
//     carries too; what counts then reaches down to 2^-35 of the value one.
//   bf16: p = hi + mid + lo, eight bits each.
// Every piece but the last is cut from a value a little below what is left, so that all are above zero wherever p is (f16:
// above 2^-23): an infinity in V then stays one in the sum of the products, where a piece of zero or below would make it NaN.
template <typename T>
struct ProbPieces;
template <>
struct ProbPieces<__half> {
    static constexpr int kCount = 2, kAccs = 2;  // pieces; accumulators (piece e goes to the e-th or the last of them)
    static constexpr float kLowScale = 1.f / 2048.f;
    static __device__ __forceinline__ void split(float p0, float p1, uint32_t (&w)[2]) {
        // (two lanes an instruction; the remainder (p - hi) 2^11 is exact in this order of operations too)
        uint64_t p, below, rest;
        float b0, b1;
        asm("mov.b64 %0, {%1, %2};" : "=l"(p) : "f"(p0), "f"(p1));
        asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(below) : "l"(p), "l"(0x3f7ff8003f7ff800ull));  // 1 - 2^-13
        asm("mov.b64 {%0, %1}, %2;" : "=f"(b0), "=f"(b1) : "l"(below));
        asm("cvt.rz.f16x2.f32 %0, %1, %2;" : "=r"(w[0]) : "f"(b1), "f"(b0));
        const float2 h = __half22float2(*reinterpret_cast<const __half2*>(&w[0]));
        uint64_t hi;
        asm("mov.b64 %0, {%1, %2};" : "=l"(hi) : "f"(h.x), "f"(h.y));
        asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(rest) : "l"(p), "l"(0x4500000045000000ull));             // 2^11
        asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(rest) : "l"(hi), "l"(0xc5000000c5000000ull), "l"(rest));
        asm("mov.b64 {%0, %1}, %2;" : "=f"(b0), "=f"(b1) : "l"(rest));
        const __half2 l = __floats2half2_rn(b0, b1);
        w[1] = *reinterpret_cast<const uint32_t*>(&l);
    }
};
template <>
struct ProbPieces<__nv_bfloat16> {
    static constexpr int kCount = 3, kAccs = 1;
    static __device__ __forceinline__ void split(float p0, float p1, uint32_t (&w)[3]) {
        uint64_t p;
        asm("mov.b64 %0, {%1, %2};" : "=l"(p) : "f"(p0), "f"(p1));
#pragma unroll
        for (int e = 0; e < 2; ++e) {  // (two lanes an instruction; the subtraction is exact)
            uint64_t below, cut;
            uint32_t b0, b1;
            asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(below) : "l"(p), "l"(0x3f7fc0003f7fc000ull));  // 1 - 2^-10
            asm("mov.b64 {%0, %1}, %2;" : "=r"(b0), "=r"(b1) : "l"(below));
            w[e] = __byte_perm(b0, b1, 0x7632);
            asm("mov.b64 %0, {%1, %2};" : "=l"(cut) : "r"(b0 & 0xffff0000u), "r"(b1 & 0xffff0000u));
            asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(p) : "l"(cut), "l"(0xbf800000bf800000ull), "l"(p));
        }
        asm("mov.b64 {%0, %1}, %2;" : "=f"(p0), "=f"(p1) : "l"(p));
        const __nv_bfloat162 l = __floats2bfloat162_rn(p0, p1);
        w[2] = *reinterpret_cast<const uint32_t*>(&l);
    }
};

// Programmatic dependent launch: a kernel launched with launch_overlapped may be scheduled while the kernel before
// it on the stream is still running (as soon as that one has executed grid_launch_dependents in every CTA, or has
// finished), so that its launch latency and set-up hide behind the predecessor's tail.  It must call
// grid_dependency_wait before it reads or writes anything an earlier kernel on the stream touches: the wait
// returns when the predecessor grid has completed and its memory operations are visible.  EVERY kernel launched
// this way calls the wait (a kernel that skipped it could finish before its predecessor and let ITS successor
// overtake that one).  Both calls are no-ops in a kernel launched the ordinary way.
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// `bytes` from `src` (both in whole 16-byte pieces) on their way to L2
__device__ __forceinline__ void prefetch_l2(const void* src, int bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(src), "r"(bytes) : "memory");
}

template <typename... KernelArgs, typename... Args>
inline cudaError_t launch_overlapped(void (*kernel)(KernelArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                     Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, KernelArgs(args)...);
}

// The same with thread-block clusters of `cluster_x` CTAs along the grid's x dimension.
template <typename... KernelArgs, typename... Args>
inline cudaError_t launch_overlapped_cluster(void (*kernel)(KernelArgs...), dim3 grid, dim3 block, int cluster_x, size_t smem,
                                             cudaStream_t stream, Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = static_cast<unsigned>(cluster_x);
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, kernel, KernelArgs(args)...);
}

// Raises a kernel's limit of dynamic shared memory, once per device (an attribute of the function, not a stream operation: legal
// while a stream is being captured).  Several host threads may get here at once; setting it twice is harmless.
using OncePerDevice = std::atomic<bool>[64];
template <typename Kern>
inline int configure_once(Kern kern, OncePerDevice& done, int smem) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return B2A_ERR_CUDA;
    if (dev < 0 || dev >= 64 || !done[dev].load(std::memory_order_acquire)) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return B2A_ERR_CUDA;
        if (dev >= 0 && dev < 64) done[dev].store(true, std::memory_order_release);
    }
    return B2A_OK;
}

}  // namespace b2a
