// Barrier over the blocks of one cooperative launch.
#pragma once
#include "abm_kernels.cuh"

namespace abm {

// Polls before a barrier gives up (about a second): a launch whose blocks cannot all
// arrive ends with ST_BARRIER instead of spinning on.  The record then holds arrivals of a
// launch that has ended, so no later launch may wait on it (HALT_LOST).
const unsigned GRID_BAR_POLLS = 1u << 21;

// Barrier over `nb` blocks, each of which calls it with all its threads (sense reversal:
// the last block to arrive resets the count and advances the generation, so launches of
// any size can share the record).  Writes made before it are visible after it: the
// arrival releases and the poll acquires at GPU scope.  False: the wait ran out.
__device__ __forceinline__ bool grid_barrier(GridBar* bar, unsigned nb, Ctrl* ctrl)
{
    __shared__ int sh_ok;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        int ok = 1;
        unsigned gen, old;
        asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(gen) : "l"(&bar->gen) : "memory");
        asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(old) : "l"(&bar->count) : "memory");
        if (old == nb - 1)
        {
            asm volatile("st.relaxed.gpu.global.u32 [%0], 0;" :: "l"(&bar->count) : "memory");
            asm volatile("st.release.gpu.global.u32 [%0], %1;" :: "l"(&bar->gen), "r"(gen + 1) : "memory");
        }
        else
        {
            unsigned polls = 0, now = gen;
            do {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(now) : "l"(&bar->gen) : "memory");
            } while (now == gen && ++polls < GRID_BAR_POLLS);
            if (now == gen)
            {
                ok = 0;
                atomicOr(&ctrl->status, (int)ST_BARRIER);
                atomicOr(&ctrl->halted, (int)HALT_LOST);
            }
        }
        sh_ok = ok;
    }
    __syncthreads();
    return sh_ok != 0;
}

// Barrier over the blocks of one cluster, each calling it with all its threads.  The
// hardware's release and acquire order global memory within the cluster; the fence keeps
// the order at GPU scope as the grid barrier does.
__device__ __forceinline__ void cluster_barrier()
{
    __threadfence();
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    __threadfence();
}

}   // namespace abm
