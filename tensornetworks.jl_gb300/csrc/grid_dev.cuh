// Barriers of a cluster or a cooperative grid and a few short-cuts around FP64,
// shared by the eigensolver's multi-block kernels.
#pragma once

#include "common.cuh"

namespace tn {
namespace griddev {

constexpr uint64_t HWAIT_NS = 2000000000ull;  // 2 s bound on any wait

__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned cluster_size() {
    unsigned r;
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint64_t hclock() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// x 2^s by the exponent field; x zero, or of a magnitude that keeps it normal
__device__ __forceinline__ double scale2(double x, int s) {
    const int h = __double2hiint(x);
    return (h & 0x7ff00000) ? __hiloint2double(h + (s << 20), __double2loint(x)) : 0.0;
}
// 1 / x for x in [2^-20, 2^20]: FP32 seed, two Newton steps (five FP64
// instructions where the division takes ten)
__device__ __forceinline__ double recip(double x) {
    double r = (double)__frcp_rn((float)x);
    r = fma(r, fma(-x, r, 1.0), r);
    return fma(r, fma(-x, r, 1.0), r);
}

// Barrier of all blocks of a cooperative launch on a counter that only grows, by one
// thread of each block; the wait is bounded by the global timer, false when it ran
// out here or in another block (looked at every 32 polls: a look is a second trip
// to L2).
__device__ __forceinline__ void grid_arrive(unsigned* count) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
}
__device__ __forceinline__ bool grid_wait(unsigned* count, int* err, unsigned target) {
    uint64_t t0 = 0;
    for (int polls = 1;; ++polls) {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
        if (v >= target) return true;
        if (polls % 32) continue;
        if (*(volatile int*)err) return false;
        const uint64_t t = hclock();
        if (t0 == 0) t0 = t;
        else if (t - t0 > HWAIT_NS) {
            atomicExch(err, 1);
            return false;
        }
    }
}
// the same for all threads of the block
__device__ __forceinline__ bool grid_sync(unsigned* count, int* err, unsigned target) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        grid_arrive(count);
        s_ok = grid_wait(count, err, target);
    }
    __syncthreads();
    return s_ok != 0;
}

}  // namespace griddev
}  // namespace tn
