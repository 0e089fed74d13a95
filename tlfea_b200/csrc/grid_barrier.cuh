// grid_barrier.cuh -- the barrier of the resident (cooperative) solvers.
#pragma once

#include "common.cuh"

namespace tlfea {

// Grid barrier of a cooperative launch in two halves, so that work that waits for nobody can
// run between them.  Every block adds one to *count (its threads' writes are visible before)
// and waits until `target` blocks have; wait returns false (in every thread) once its
// bounded polling has run out.
constexpr int LIN_WAIT_LIMIT = 1 << 23;
__device__ __forceinline__ void lin_grid_arrive(unsigned int* count) {
    __syncthreads();
    if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
}
// The first warp waits, then folds the blocks' shares in block order; the total in `sum_sh`.
__device__ __forceinline__ bool lin_grid_wait_sum(const unsigned int* count, unsigned int target, const double* part,
                                                  int n, int* ok_sh, double* sum_sh) {
    if (threadIdx.x < 32) {
        if (threadIdx.x == 0) {
            int ok = 0;
            for (int k = 0; k < LIN_WAIT_LIMIT; ++k) {
                unsigned int v;
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
                if ((int)(v - target) >= 0) {
                    ok = 1;
                    break;
                }
            }
            *ok_sh = ok;
        }
        __syncwarp();
        double w = 0.0;
        for (int b = threadIdx.x; b < n; b += 32) w += __ldcg(part + b);
        w = warp_sum(w);
        if (threadIdx.x == 0) *sum_sh = w;
    }
    __syncthreads();
    return *ok_sh != 0;
}

}  // namespace tlfea
