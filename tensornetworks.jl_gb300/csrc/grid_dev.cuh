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

// Barrier of all blocks of a cooperative launch on a counter that only grows;
// bounded by the global timer, false (in every thread of the block) when the
// wait ran out here or in another block.
__device__ __forceinline__ bool grid_sync(unsigned* count, int* err, unsigned target) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        int ok = 1;
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
        if (v < target) {
            const uint64_t t0 = hclock();
            do {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
                if (*(volatile int*)err) ok = 0;
                else if (hclock() - t0 > HWAIT_NS) {
                    atomicExch(err, 1);
                    ok = 0;
                }
            } while (ok && v < target);
        }
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

}  // namespace griddev
}  // namespace tn
