// ed_grid.cuh — grid-wide barrier and exact grid reductions of the persistent
// (cooperative) Lanczos kernels.
#pragma once

#include <cuda_runtime.h>

#include "ed_device.cuh"
#include "ed_lanczos.hpp"

namespace ed {
namespace dev {

constexpr uint64_t kLimb = (1ULL << 42) - 1;

__device__ __forceinline__ unsigned int ld_relaxed_gpu(const unsigned int* p) {
    unsigned int v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void red_release_gpu_add(unsigned int* p, unsigned int v) {
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ void fence_acq_rel_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Thread 0: add a CTA's sum and max to an accumulator set.
__device__ __forceinline__ void red_push(LzRedSet* r, i128 v, uint64_t m) {
    const u128 uv = (u128)v;
    atomicAdd(&r->l0, (unsigned long long)(uv & kLimb));
    atomicAdd(&r->l1, (unsigned long long)((uv >> 42) & kLimb));
    atomicAdd(&r->l2, (unsigned long long)(int64_t)(v >> 84));
    atomicMax(&r->mx, (unsigned long long)m);
}

// Thread 0, after the barrier: the grid totals.
__device__ __forceinline__ void red_pull(const LzRedSet* r, i128& v, uint64_t& m) {
    const unsigned long long l0 = __ldcg(&r->l0), l1 = __ldcg(&r->l1), l2 = __ldcg(&r->l2);
    m = __ldcg(&r->mx);
    v = (i128)((u128)l0 + ((u128)l1 << 42) + ((u128)(i128)(int64_t)l2 << 84));
}

// A warp's (v, m) into per-instance shared limb sums (all 32 lanes call it).
__device__ __forceinline__ void batch_flush(i128 v, uint64_t m, unsigned long long* accl, unsigned long long* accm) {
    v = warp_sum_i128(v);
    m = warp_max_u64(m);
    if ((threadIdx.x & 31) == 0) {
        const u128 uv = (u128)v;
        atomicAdd(&accl[0], (unsigned long long)(uv & kLimb));
        atomicAdd(&accl[1], (unsigned long long)((uv >> 42) & kLimb));
        atomicAdd(&accl[2], (unsigned long long)(int64_t)(v >> 84));
        atomicMax(accm, (unsigned long long)m);
    }
}

__device__ __forceinline__ i128 batch_total(const unsigned long long* accl) {
    return (i128)((u128)accl[0] + ((u128)accl[1] << 42) + ((u128)(i128)(int64_t)accl[2] << 84));
}

// Grid-wide barrier on a monotone arrival counter: the k-th barrier of the
// launch completes when k * gridDim.x CTAs have arrived.  Writes and atomics
// before it (by any thread of any CTA) are visible after it.  False when the
// wait gave up; *give_up is then set for the whole CTA.
__device__ __forceinline__ bool grid_sync(unsigned int* gbar, unsigned int& target, int* give_up, int* err,
                                          const GridWait& lim) {
    __syncthreads();
    if (threadIdx.x == 0) {
        target += gridDim.x;
        // release: this CTA's writes and atomics (ordered before this thread
        // by the CTA barrier above) before the arrival
        red_release_gpu_add(gbar, 1u);
        const unsigned long long t0 = global_ns();
        const unsigned int want = target + lim.extra;
        long long it = 0;
        while (ld_relaxed_gpu(gbar) < want) {
            if (++it > lim.spin || global_ns() - t0 > lim.ns) {
                atomicExch(err, 1);
                *give_up = 1;
                break;
            }
        }
        fence_acq_rel_gpu();  // acquire: everything released before the last arrival
    }
    __syncthreads();
    return *give_up == 0;
}

}  // namespace dev
}  // namespace ed
