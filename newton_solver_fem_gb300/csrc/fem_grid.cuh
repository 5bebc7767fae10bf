// Device helpers shared by the persistent PCG kernels: the bounded grid barrier, warp reductions,
// 3x3 block products and packed float3 access.
#pragma once
#include "fem_internal.cuh"
#include "fem_math.cuh"

namespace fem {

__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ int ld_relaxed_int(const int* p) {
    int v;
    asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Grid barrier over a monotone counter (zero before the launch), entered by
// one thread per CTA after a CTA or warp barrier has ordered the CTA's writes
// before it.  The arrival is a release reduction, so those writes are visible
// at GPU scope before it; the wait is an acquire load, so the other CTAs'
// writes are visible after it.  The wait is bounded: it gives up after
// limit_ns nanoseconds, or as soon as another CTA has given up, and returns 0.
__device__ __forceinline__ int arrive_and_wait(unsigned* counter, unsigned nblocks, unsigned& epoch, int* status,
                                               long long limit_ns) {
    epoch += 1;
    const unsigned target = epoch * nblocks;
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(counter) : "memory");
    const unsigned long long t0 = global_ns();
    unsigned spins = 0;
    while ((int)(ld_acquire(counter) - target) < 0) {  // wrap-safe: the counter only grows
        if ((++spins & 63u) == 1u) {  // first spin, then every 64th
            if ((ld_relaxed_int(status) & kStatusTimeout) != 0 || (long long)(global_ns() - t0) >= limit_ns) {
                atomicOr(status, kStatusTimeout);
                return 0;
            }
        }
    }
    return 1;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, off));
    return v;
}
__device__ __forceinline__ float3 bmul(float4 a, float4 b, float c, float3 p) {
    return f3(a.x * p.x + a.y * p.y + a.z * p.z, a.w * p.x + b.x * p.y + b.y * p.z, b.z * p.x + b.w * p.y + c * p.z);
}

__device__ __forceinline__ float3 load3(const float* p, int i) { return f3(p[3 * i], p[3 * i + 1], p[3 * i + 2]); }
__device__ __forceinline__ void store3(float* p, int i, float3 v) {
    p[3 * i] = v.x;
    p[3 * i + 1] = v.y;
    p[3 * i + 2] = v.z;
}

__device__ __forceinline__ float rhs_scale(float maximum) {
    // kernels.py:1785-1793
    float scale = 1.0f;
    if (maximum > 0.0f && maximum < 1.0e-12f) scale = fminf(1.0f / maximum, 1.0e30f);
    return scale;
}

}  // namespace fem
