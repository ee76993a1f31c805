// A multigrid solve shared by the CTAs of one thread-block cluster.
//
// The 2D solves are chains of short phases (form a colour's right-hand
// sides, eliminate its lines, residual, transfer).  One SM issues two FP64
// lanes a cycle, so on one SM the phases around the eliminations cost more
// than the eliminations; a cluster spreads them over up to 16 SMs and meets
// at the hardware cluster barrier, 0.2 us where a grid-wide barrier takes
// 1.3 us (129 x 129 uniform annulus, FP64, four steps: one CTA 23.1 ms, 16 CTAs
// 12.7, of which the eliminations' chains are 9).
// Every CTA runs the same control flow: what decides it (residual
// norms, NaN flags) comes from cl_max, which gives every CTA the same bits.
#pragma once

#include <cooperative_groups.h>
#include <cuda_runtime.h>

#define CL_MAX_CTAS 16

struct Cluster {
    int rank, size;
    __device__ __forceinline__ static Cluster self()
    {
        Cluster c;
        c.rank = (int)cooperative_groups::this_cluster().block_rank();
        c.size = (int)cooperative_groups::this_cluster().num_blocks();
        return c;
    }
    __device__ __forceinline__ int tid() const { return rank * (int)blockDim.x + (int)threadIdx.x; }
    __device__ __forceinline__ int nthr() const { return size * (int)blockDim.x; }
    // The two halves of sync: what is issued between them (fetches of the next
    // phase's constants) overlaps the barrier, where a fetch issued before the
    // release would be waited for.  The unaligned forms: a warp may come here
    // diverged, from a loop that its lanes left at different times, and an aligned
    // barrier is defined for converged warps only.
    __device__ __forceinline__ void arrive() const
    {
        if (size > 1) asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    }
    __device__ __forceinline__ void wait() const
    {
        if (size > 1) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
        else __syncthreads();
    }
    // Orders global and distributed shared memory between all threads of the
    // cluster (arrive with release, wait with acquire at cluster scope).
    __device__ __forceinline__ void sync() const
    {
        if (size > 1) cooperative_groups::this_cluster().sync();
        else __syncthreads();
    }
};

// idx / n and idx % n by one high multiplication: magic = (2^32 - 1) / n + 1
// gives a quotient at most one too large for every 0 <= idx < 2^31 (formed by
// a 32-bit division; a 64-bit one costs as much as a short phase).
struct RowSplit {
    int n;
    unsigned magic;
    __device__ __forceinline__ explicit RowSplit(int n_) : n(n_), magic(0xffffffffu / (unsigned)n_ + 1u)
    {
        if (n_ == 1) magic = 0;
    }
    // of a divisor whose magic was formed before
    __device__ __forceinline__ RowSplit(int n_, unsigned magic_) : n(n_), magic(magic_) {}
    __device__ __forceinline__ void operator()(int idx, int &q, int &r) const
    {
        if (n == 1) {
            q = idx;
            r = 0;
            return;
        }
        q = (int)__umulhi((unsigned)idx, magic);
        r = idx - q * n;
        if (r < 0) {
            --q;
            r += n;
        }
    }
};

// Shared state of cl_max: per-warp partials and two published slots, used in
// turn so that one cluster barrier per reduction is enough (a slot is
// rewritten only after the barrier of the reduction in between).
struct ClMaxState {
    double part[32];
    int flagpart[32];
    double pub[2];
    int flagpub[2];
};

// Maximum of m over the cluster (NaNs ignored) and the or of flags; every
// thread gets the same result.  Also a cluster-wide barrier for everything
// written before the call.
__device__ __forceinline__ double cl_max(const Cluster &cl, ClMaxState &s, int &turn, double m, int &flags)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (int)blockDim.x >> 5;
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    flags = (int)__reduce_or_sync(0xffffffffu, (unsigned)flags);
    if (lane == 0) {
        s.part[warp] = m;
        s.flagpart[warp] = flags;
    }
    __syncthreads();
    const int t = turn;
    turn ^= 1;
    if (warp == 0) {
        m = lane < nw ? s.part[lane] : 0.0;
        flags = lane < nw ? s.flagpart[lane] : 0;
        for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
        flags = (int)__reduce_or_sync(0xffffffffu, (unsigned)flags);
        if (lane == 0) {
            s.pub[t] = m;
            s.flagpub[t] = flags;
        }
    }
    cl.sync();
    if (cl.size == 1) {
        flags = s.flagpub[t];
        return s.pub[t];
    }
    cooperative_groups::cluster_group g = cooperative_groups::this_cluster();
    m = 0.0;
    flags = 0;
    if (lane < cl.size) {
        m = *g.map_shared_rank(&s.pub[t], lane);
        flags = *g.map_shared_rank(&s.flagpub[t], lane);
    }
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    flags = (int)__reduce_or_sync(0xffffffffu, (unsigned)flags);
    return m;
}

// Launches kernel on clusters of `ctas` CTAs, nclusters of them (ctas = 1: an
// ordinary launch).  Sizes above 8 need the kernel's
// cudaFuncAttributeNonPortableClusterSizeAllowed (cl_prepare).  A cluster can be
// refused where an ordinary launch is not, and while a stream is captured the
// step would just lack its solve, so no caller may drop the result (the build
// treats that as an error).
template <class... P, class... A>
[[nodiscard]] static inline cudaError_t cl_launch(void (*kernel)(P...), int nclusters, int ctas, int threads, size_t smem, cudaStream_t s,
                                    A... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(nclusters * ctas));
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)ctas;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, P(args)...);
    if (e != cudaSuccess) cudaGetLastError();   // it is the caller's now, not a later call's
    return e;
}

// Allows clusters of up to CL_MAX_CTAS and smem bytes of dynamic shared
// memory for a kernel.
template <class F> static inline cudaError_t cl_prepare(F kernel, size_t smem)
{
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    return e;
}

// Grids of so few points have no work to spread: their phases are latency, and a
// cluster's barriers and remote accesses only add to it.  Mixed streamfunction
// solves, four steps, on 16 CTAs and on one: 8 x 8 0.64 and 0.54 ms, 16 x 16 1.05
// and 0.87, 32 x 32 1.24 and 1.14, 40 x 40 1.52 and 1.64.
static inline bool cl_small_grid(int n1, int n2) { return (long long)n1 * n2 <= 1024; }

// CTAs per cluster for a solve: `want`, halved until the device can hold one
// such cluster with this shared memory.
template <class F> static inline int cl_fit(F kernel, int want, int threads, size_t smem)
{
    for (int c = want; c > 1; c >>= 1) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)c);
        cfg.blockDim = dim3((unsigned)threads);
        cfg.dynamicSmemBytes = smem;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)c;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) == cudaSuccess && n > 0) return c;
        cudaGetLastError();
    }
    return 1;
}
