// Bounded grid-wide barrier for persistent cooperative kernels (sm_103a).
#pragma once

#include <cuda_runtime.h>

// Grid-wide barrier of a persistent (cooperatively launched) kernel.  Every wait is bounded: a
// block that waits longer than `limit` polls sets the error flag and every
// block leaves the kernel at its next barrier, so a lost block cannot hang
// the GPU.  The outcome is read once per block (by the thread that waited)
// and handed to the whole block through shared memory, so all threads of a
// block leave together even when another block raises the flag meanwhile.
struct GridSync {
    unsigned *count;   // zero when the kernel starts
    int *err;
    long long limit;
    unsigned long long *tally;   // optional (may be null): barriers passed, counted once per barrier by block 0
};

// Default wait limit: some seconds of polling at an L2 round trip per poll.
#define GB_GRID_WAIT_LIMIT_DEFAULT (1LL << 24)

// Arrival and wait of one thread per block.  The count grows from one barrier
// to the next (it is zero at the launch), so that nothing is reset and nobody
// has to announce the last arrival: the blocks poll the count itself, a release
// and its trip through L2 less than with a generation that the last one
// publishes.
__device__ __forceinline__ void grid_barrier(const GridSync &gs)
{
    unsigned arrived;
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(arrived) : "l"(gs.count) : "memory");
    const unsigned all = arrived - arrived % gridDim.x + gridDim.x;
    if (arrived + 1u == all) return;
    for (long long it = 0;;) {
        unsigned now;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(now) : "l"(gs.count) : "memory");
        if ((int)(now - all) >= 0) break;
        if (++it > gs.limit || ((it & 15) == 0 && *(volatile int *)gs.err)) {
            atomicExch(gs.err, 1);
            break;
        }
    }
}

// The barrier for the whole grid; false when it gave up.  meanwhile(): what
// the threads outside the first warp do while its first thread waits (it may
// touch shared memory and constants only).
template <class F> __device__ __forceinline__ bool grid_sync(const GridSync &gs, F meanwhile)
{
    __shared__ int s_grid_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        grid_barrier(gs);
        s_grid_ok = *(volatile int *)gs.err == 0;
        if (gs.tally && blockIdx.x == 0) atomicAdd(gs.tally, 1ull);
    } else if (threadIdx.x >= 32) {
        meanwhile();
    }
    __syncthreads();
    return s_grid_ok != 0;
}
__device__ __forceinline__ bool grid_sync(const GridSync &gs)
{
    return grid_sync(gs, [] {});
}
