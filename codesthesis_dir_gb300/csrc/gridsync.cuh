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
    unsigned long long *count;   // zero when the kernel starts
    int *err;
    long long limit;
    unsigned long long *tally;   // optional (may be null): barriers passed, counted once per barrier by block 0
};

// Default wait limit: about 3 s (187 ns a poll, an L2 round trip).
#define GB_GRID_WAIT_LIMIT_DEFAULT (1LL << 24)

// The count at which the barrier of an arrival that found it at `arrived` is
// complete; `last`: at which the block's barrier before was (the first finds
// less than the blocks).  64 bits: a 32-bit count wraps after 2^32 / blocks
// barriers (14 million with 304, some 20 seconds of a solve that does not
// converge), and beyond the wrap blocks would leave early.  From the barrier
// before, because the remainder by the blocks is a 64-bit division on the last
// arrival's way (1.29 -> 1.33 us with 152 blocks).
__host__ __device__ __forceinline__ unsigned long long grid_barrier_end(unsigned long long arrived, unsigned blocks, unsigned long long last)
{
    return arrived < blocks ? blocks : last + blocks;
}

// Arrival and wait of one thread per block.  The count grows from one barrier
// to the next (it is zero at the launch), so that nothing is reset and nobody
// has to announce the last arrival: the blocks poll the count itself, a release
// and its trip through L2 less than with a generation that the last one
// publishes.
__device__ __forceinline__ void grid_barrier(const GridSync &gs)
{
    __shared__ unsigned long long s_grid_end;   // of the arriving thread alone
    unsigned long long arrived;
    asm volatile("atom.add.acq_rel.gpu.global.u64 %0, [%1], 1;" : "=l"(arrived) : "l"(gs.count) : "memory");
    const unsigned long long all = grid_barrier_end(arrived, gridDim.x, s_grid_end);
    s_grid_end = all;
    if (arrived + 1 == all) return;
    for (long long it = 0;;) {
        unsigned long long now;
        asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(now) : "l"(gs.count) : "memory");
        if (now >= all) break;
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
