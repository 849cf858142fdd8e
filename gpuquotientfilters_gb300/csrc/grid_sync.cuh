// Bounded barrier across a co-resident grid (a cooperative launch).
#pragma once

#include "sqf_build.cuh"

namespace gqf {

// Grid-wide barrier for a co-resident grid: thread 0 of each CTA arrives,
// the last one opens the next generation.  The wait is bounded; a CTA that
// gives up records DEV_ERR_TIMEOUT and the abort word, and every CTA leaves
// at the next barrier.  Returns false when the pipeline must stop.
__device__ __forceinline__ bool grid_sync(uint32_t *bar, uint32_t *err)
{
    __shared__ uint32_t s_go;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t go = 1;
        volatile uint32_t *vbar = bar;
        const uint32_t gen = vbar[1];
        __threadfence();  // this CTA's phase writes before its arrival
        if (atomicAdd(bar, 1u) == gridDim.x - 1) {
            vbar[0] = 0u;
            __threadfence();
            atomicAdd(bar + 1, 1u);
        } else {
            uint32_t i = 0;
            while (vbar[1] == gen) {
                if (++i > SPIN_LIMIT) {
                    atomicOr(err, DEV_ERR_TIMEOUT);
                    atomicExch(bar + 2, 1u);
                    break;
                }
            }
        }
        __threadfence();
        if (vbar[2]) go = 0;
        s_go = go;
    }
    __syncthreads();
    return s_go != 0;
}

}  // namespace gqf
