// Shared device helpers for the SpMV kernels.
#pragma once

#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>

namespace csp {
namespace dev {

constexpr int kWarp = 32;

// Matrix values are stored as FP32 or BF16; arithmetic is always FP32.
template <class V> struct Val;

template <> struct Val<float> {
    __device__ __forceinline__ static float ld(const float* p) { return __ldg(p); }
    // Four consecutive values; p must be 16-byte aligned.
    __device__ __forceinline__ static float4 ld4(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }
    // The same from shared memory.
    __device__ __forceinline__ static float4 lds4(const float* p) { return *reinterpret_cast<const float4*>(p); }
};

template <> struct Val<__nv_bfloat16> {
    __device__ __forceinline__ static float ld(const __nv_bfloat16* p)
    {
        unsigned short u = __ldg(reinterpret_cast<const unsigned short*>(p));
        return __uint_as_float(((unsigned)u) << 16);
    }
    // Four consecutive values; p must be 8-byte aligned.
    __device__ __forceinline__ static float4 ld4(const __nv_bfloat16* p)
    {
        return widen(__ldg(reinterpret_cast<const uint2*>(p)));
    }
    __device__ __forceinline__ static float4 lds4(const __nv_bfloat16* p) { return widen(*reinterpret_cast<const uint2*>(p)); }
    __device__ __forceinline__ static float4 widen(uint2 u)
    {
        float4 f;
        f.x = __uint_as_float(u.x << 16);
        f.y = __uint_as_float(u.x & 0xffff0000u);
        f.z = __uint_as_float(u.y << 16);
        f.w = __uint_as_float(u.y & 0xffff0000u);
        return f;
    }
};

// The point of a kernel after which it may touch what the kernel before it in the stream
// reads or writes: x and y.  In a chain of launches with programmatic stream serialization
// (csp_iterate) the part before it -- loads of the matrix -- overlaps the previous kernel;
// in any other launch it returns at once.  The next kernel is let in only here, after the
// previous one has completed, so at most two of the chain run at a time and no SM holds
// lines of x from two steps ago.  x is read by plain loads in such kernels (it is written
// within the life of a waiting kernel, which the read-only path does not allow).
__device__ __forceinline__ void grid_dependency()
{
    asm volatile("griddepcontrol.wait;\ngriddepcontrol.launch_dependents;\n" ::: "memory");
}

// The same for kernels of many CTAs that live about a microsecond each.  Letting the next kernel
// in costs the chip 1.1 to 1.2 ns per CTA, one after the other, which then bounds such a kernel; so
// from two waves of 148 x 8 CTAs up it lets the next one in by leaving.
__device__ __forceinline__ void grid_dependency_short()
{
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    if (gridDim.x <= 2 * 148 * 8) asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
}

__device__ __forceinline__ void cp_async4(void* dst, const void* src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// Requests the whole 16-byte units of [p, p + bytes) for L2, by one instruction; no result is
// waited for.
__device__ __forceinline__ void prefetch_l2(const void* p, int bytes)
{
    const uintptr_t a = (reinterpret_cast<uintptr_t>(p) + 15) & ~(uintptr_t)15;
    const int n = (int)((reinterpret_cast<uintptr_t>(p) + bytes - a) & ~(uintptr_t)15);
    if (n > 0 && bytes > 0) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(a), "r"(n));
}

__device__ __forceinline__ int4 ld_int4(const int* p) { return __ldg(reinterpret_cast<const int4*>(p)); }
__device__ __forceinline__ float ldx(const float* x, int i) { return __ldg(x + i); }
__device__ __forceinline__ float4 ldx4(const float* x, int i) { return __ldg(reinterpret_cast<const float4*>(x + i)); }

// Sum over the G lanes of an aligned lane group (G a power of two, <= 32).
template <int G>
__device__ __forceinline__ float group_sum(float v)
{
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o, G);
    return v;
}

// Block-wide sum; every thread gets the total.  `scratch` holds >= blockDim.x / 32 floats.
__device__ __forceinline__ float block_sum(float v, float* scratch)
{
    v = group_sum<kWarp>(v);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    __syncthreads();
    if (lane == 0) scratch[wid] = v;
    __syncthreads();
    float t = 0.0f;
    for (int i = 0; i < nw; i++) t += scratch[i];
    return t;
}

}  // namespace dev
}  // namespace csp
