// Velocity-component multigrid solves of the 2D periodic Rayleigh-Benard
// driver (poisson2/poisson3, relax2/relax3, corser, finer of
// velvor2dperiodicrbconv.f:1724-2859): one launch per solve, one CTA or one
// cluster of CTAs (cluster.cuh) per equation.  The whole outer sweep loop,
// every level and every convergence test run inside it, so a solve costs one
// kernel launch however many sweeps it takes.  The v and u solves of a step
// are two clusters of one launch (the reference runs them as two OpenMP
// sections, PRB:370-380).
//
// Two smoother orderings:
//   LEX   - lines k = 1..n3 in order, the reference schedule: each line needs
//           the one before it, so one CTA (its threads form a line's
//           right-hand side together, one carries the elimination).
//   ZEBRA - odd lines, then even lines, the lines of a colour shared out over
//           the cluster.
// Either way each line is solved with the reference's banded elimination in
// the reference's operation order (-fmad=false), so LEX results are
// bit-identical to the reference algorithm and ZEBRA results to the same
// algorithm under zebra ordering.
//
// The rotating-annulus variant (relax2/relax3/corser of
// velvor2dnewsch3.4.f:2071-2716) uses the same kernel: its line matrices
// depend on the radius of row i but not on the line k, so they are still
// factored once per level; the line right-hand sides and residuals gain the
// polar terms (E.polar), every level visit runs three relaxations (E.nrelax,
// :2134, :2410), and the coarse right-hand side of seam line n3c keeps the
// fine residual stored there because that corser does not clear it
// (E.seam_keep, :2696-2704).  The Taylor-Couette driver
// (velvor2dtaycouheat.f) has the polar operator with PRB's single
// relaxation and seam reset.
//
// Storage differs from the reference only in scratch that no output depends
// on: each level keeps its solution in place (level 1 in psif, the coarser
// ones in their packed slots; the reference copies the level at hand through
// psif), the right-hand sides are read from the packed per-level arrays, and
// residuals are formed where something reads them.  Every value the solution
// depends on is formed by the same arithmetic on the same operands.
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <type_traits>

#include "banded.cuh"
#include "cluster.cuh"
#include "gbcommon.cuh"
#include "mg_op.cuh"
#include "prb_internal.cuh"
#include "warpline.cuh"

// FP64: the eliminations want registers.  FP32 on global memory serves the
// large grids, whose passes want threads (272 x 1200 annulus, a step: 24.2 ms
// with 256, 20.7 with 512).
#define MG_THREADS 256
#define MG_THREADS_MIXED 512
#define MG_SPREAD 8    // the cluster size a caller may ask for (gb_prb_set_solve_spread)

// One level of one equation: its solution in place (level 1: psif, else the
// packed slot), pitch ld.
template <class T> struct MgView {
    int which, n1, n3, ld, polar, xwall;
    T *v;
    const T *f;
    T hhri, hhpi, hri;
    const T *rvi, *rvq, *fac;
    // unknowns of a line and the last line (the tank's v lines stop short of
    // its wall k = n3, velvor2dhorconvtank.f:1170, :1216)
    __device__ __forceinline__ int rows() const { return which == 2 ? n1 : n1 - 1; }
    __device__ __forceinline__ int lines() const { return xwall && which == 2 ? n3 - 1 : n3; }
    // the line after k: periodic, or the tank's last u line's zero k = 0 as
    // its wall (velvor2dhorconvtank.f:1275)
    __device__ __forceinline__ int after(int k) const { return k == n3 ? (xwall ? 0 : 1) : k + 1; }
};
__device__ __forceinline__ MgView<double> mg_view(const MgEq &E, int l, double)
{
    const MgLevel &L = E.lev[l];
    return {E.which, L.n1, L.n3, l == 1 ? E.ld : L.n1 + 1, E.polar, E.xwall, l == 1 ? E.psif : L.v, L.f, L.hhri, L.hhpi, L.hri,
            L.rvi, L.rvq, L.fac};
}
__device__ __forceinline__ MgView<float> mg_view(const MgEq &E, int l, float)
{
    const MgLevel &L = E.lev[l];
    return {E.which, L.n1, L.n3, l == 1 ? E.ld : L.n1 + 1, E.polar, E.xwall, l == 1 ? E.psif32 : L.v32, L.f32, (float)L.hhri,
            (float)L.hhpi, (float)L.hri, L.rvi32, L.rvq32, L.fac32};
}

// Dynamic shared memory of a solve: the level's line factors and the staged
// lines' right-hand sides.
#define MG_SMEM_BYTES (160 * 1024)

// The nl lines first, first + step, ... (relax2 PRB:2113-2191 pentadiagonal,
// relax3 PRB:2414-2460 tridiagonal), which read none of one another: a
// colour, or one line of the reference's order.  Each CTA takes a contiguous
// share, in batches that fit its shared memory: all threads form the
// right-hand sides, the lines are eliminated (FP64: one thread per line in the
// reference's order; FP32: up to 32 lanes per line), the solutions go back.
// fresh: the level's factors are not in shared memory yet (the reference's order
// comes here line by line).
template <class T> __device__ __noinline__ void mg_lines(const MgEq &E, int l, int first, int step, int nl, bool fresh)
{
    extern __shared__ __align__(16) unsigned char s_mg[];
    constexpr bool F64 = sizeof(T) == 8;
    const Cluster cl = Cluster::self();
    const MgView<T> L = mg_view(E, l, T(0));
    const int n = L.rows(), ldf = L.n1 + 1;
    const int flen = (int)(F64 ? (L.which == 2 ? pdma_fac_len(n) : tdma_fac_len(n)) : (L.which == 2 ? pdma32_len(n) : tdma32_len(n)));
    const int lpitch = F64 ? 0 : wl_pitch(n), lg = F64 ? 0 : wl_log2m(n);
    const int share = (nl + cl.size - 1) / cl.size;
    const int t0 = cl.rank * share, t1 = min(nl, t0 + share);
    const int words = (int)(MG_SMEM_BYTES / sizeof(T)) - ((flen + 3) & ~3);
    int B = F64 ? words / n - 1 : words / lpitch;
    const bool staged = B >= 1;   // the factors and a line fit (rows up to 2900 in FP64)
    if (!staged) B = 1;
    B = min(B, min(share, (int)blockDim.x));
    T *sfac = (T *)s_mg, *x = staged ? sfac + ((flen + 3) & ~3) : sfac;
    const RowSplit split(n);
    if (staged && fresh && t0 < t1) async_copy(sfac, L.fac, flen, threadIdx.x, blockDim.x);
    for (int b0 = t0; b0 < t1; b0 += B) {
        const int nb = min(B, t1 - b0), pitch = nb | 1;
        // FP64: [row][line], odd pitch; FP32: [line][row], padded per lane
        auto at = [&](int t, int q) -> T & { return F64 ? x[q * pitch + t] : x[t * lpitch + wl_slot(lg, q)]; };
        for (int idx = threadIdx.x; idx < nb * n; idx += blockDim.x) {
            int t, q;
            split(idx, t, q);
            const int k = first + step * (b0 + t), i = q + 1;
            T r = -(L.v[i + L.ld * L.after(k)] + L.v[i + L.ld * (k - 1)]) * L.hhpi;
            if (L.polar) r = r * L.rvq[i];
            at(t, q) = r + L.f[i + ldf * k];
        }
        if constexpr (!F64) {   // rows past the line's end
            const int pad = wl_rows(n) - n;
            for (int idx = threadIdx.x; idx < nb * pad; idx += blockDim.x) at(idx / pad, n + idx % pad) = T(0);
        }
        async_copy_wait();
        __syncthreads();
        if constexpr (F64) {
            if ((int)threadIdx.x < nb) {
                T *y = x + threadIdx.x;
                if (!staged) {
                    if (L.which == 2) pdma_staged(L.fac, n, y, pitch);
                    else tdma_staged(L.fac, n, y, pitch);
                } else if (L.which == 2) {
                    pdma_staged(sfac, n, y, pitch);
                } else {
                    tdma_staged(sfac, n, y, pitch);
                }
            }
        } else {
            const T *tab = staged ? sfac : L.fac;
            if (L.which == 2) wl_lines<true>(tab, 0, n, x, lpitch, nb);
            else wl_lines<false>(tab, 0, n, x, lpitch, nb);
        }
        __syncthreads();
        for (int idx = threadIdx.x; idx < nb * n; idx += blockDim.x) {
            int t, q;
            split(idx, t, q);
            const int k = first + step * (b0 + t);
            const T v = at(t, q);
            L.v[q + 1 + L.ld * k] = v;
            if (k == L.n3) L.v[q + 1] = L.xwall ? T(0) : v;   // k = 0 repeats k = n3; the tank's wall is zero
        }
        if (b0 + B < t1) __syncthreads();
    }
    cl.sync();
}

// The reference's line order in FP32: the lines of a level's sweeps one after the
// other by one warp, its table and the line before in registers, the line after
// and the right-hand side of the next line on their way while one is solved.  As
// batches of one line (mg_lines) each line paid four block barriers: 8 x 64 layer,
// two steps, 49.7 ms by one thread per sweep before, 91.4 in batches, 32.3 this way.
// Groups of lanes that have no line repeat the first one's and store nothing.
__device__ __noinline__ void mg_lex32(const MgEq &E, int l)
{
    constexpr int M = 8;
    const MgView<float> L = mg_view(E, l, 0.f);
    const int n = L.rows(), ldf = L.n1 + 1, n3 = L.n3, nrelax = E.nrelax;
    auto sweeps = [&](auto penta) {
        constexpr bool PENTA = decltype(penta)::value;
        const int lw = wl_log2w(n), lane = threadIdx.x & ((1 << lw) - 1), i0 = 1 + lane * M;
        const bool mine = threadIdx.x >> lw == 0;
        WlTab<M, PENTA> tab;
        tab.load(L.fac, lw);
        auto fetch = [&](const float *row, float (&y)[M]) {
#pragma unroll
            for (int u = 0; u < M; ++u) y[u] = lane * M + u < n ? row[i0 + u] : 0.f;
        };
#pragma unroll 1
        for (int irel = 0; irel < nrelax; ++irel) {
            float t[M], a[M], f[M];   // the line before, in turn the present one; the line after; the right-hand side
            fetch(L.v, t);
            fetch(L.v + L.ld * L.after(1), a);
            fetch(L.f + ldf, f);
#pragma unroll 1
            for (int k = 1; k <= n3; ++k) {
#pragma unroll
                for (int u = 0; u < M; ++u) {
                    float r = -(a[u] + t[u]) * L.hhpi;
                    if (L.polar) r = r * L.rvq[min(i0 + u, L.n1 + 1)];
                    t[u] = lane * M + u < n ? r + f[u] : 0.f;
                }
                if (k < n3) {
                    fetch(L.v + L.ld * L.after(k + 1), a);
                    fetch(L.f + ldf * (k + 1), f);
                }
                tab.solve(n, t);
                if (mine) {
                    float *v = L.v + L.ld * k;
#pragma unroll
                    for (int u = 0; u < M; ++u)
                        if (lane * M + u < n) {
                            v[i0 + u] = t[u];
                            if (k == n3) L.v[i0 + u] = t[u];   // k = 0 repeats k = n3
                        }
                }
                __syncwarp();
                if (n3 == 2) {   // the line after the last is the one just solved
#pragma unroll
                    for (int u = 0; u < M; ++u) a[u] = t[u];
                }
            }
        }
    };
    if (threadIdx.x < 32) {
        if (L.which == 2) sweeps(std::true_type());
        else sweeps(std::false_type());
    }
    Cluster::self().sync();
}

// relax2 / relax3's line sweeps (one with nrel = 1; three in the annulus), in
// place on the level's solution.
template <class T> __device__ __forceinline__ void mg_sweeps(const MgEq &E, int l)
{
    const int n3 = E.lev[l].n3, klast = E.xwall && E.which == 2 ? n3 - 1 : n3;
    if constexpr (sizeof(T) == 4) {
        if (E.mode == GB_SMOOTHER_LEX && E.lev[l].n1 <= 256) {   // 8 rows a lane
            mg_lex32(E, l);
            return;
        }
    }
    for (int irel = 0; irel < E.nrelax; ++irel) {
        if (E.mode == GB_SMOOTHER_LEX) {
            for (int k = 1; k <= klast; ++k) mg_lines<T>(E, l, k, 1, 1, irel == 0 && k == 1);
        } else {
            mg_lines<T>(E, l, 1, 2, (klast + 1) / 2, true);
            mg_lines<T>(E, l, 2, 2, klast / 2, true);
        }
    }
}

// The residual of level l, PRB:2306-2357 (v) and PRB:2553-2587 (u), into rc
// (pitch ldr; not followed by a barrier): its largest magnitude (NaNs ignored
// as in the reference's comparison) and whether one is a NaN over the calling
// thread's points.
template <class T, class R> __device__ __noinline__ T mg_residual(const MgEq &E, int l, R *rc, int ldr, int *nan_out)
{
    const Cluster cl = Cluster::self();
    const MgView<T> L = mg_view(E, l, T(0));
    const int n = L.rows(), ldf = L.n1 + 1, tot = n * L.lines();
    const RowSplit split(n);
    T m = T(0);
    int nan = 0;
    for (int idx = cl.tid(); idx < tot; idx += cl.nthr()) {
        int k, i;
        split(idx, k, i);
        ++i;
        ++k;
        const T *row = L.v + L.ld * k;
        T r = mg_apply_op<T>([&](int q) { return row[q]; }, L.v[i + L.ld * L.after(k)], L.v[i + L.ld * (k - 1)], i, L.which, L.polar,
                             L.n1, L.hhri, L.hhpi, L.hri, L.rvi, L.rvq);
        r = L.f[i + ldf * k] - r;
        rc[i + ldr * k] = (R)r;
        r = fabs(r);
        if (r != r) nan = 1;
        if (r > m) m = r;
    }
    *nan_out = nan;
    return m;
}

// corser (PRB:2603-2718): full weighting of rc (pitch E.ld on every level:
// row k = 0 is never written and stays zero) onto the coarse right-hand side;
// the coarse solution is cleared.  The annulus keeps the residual stored at
// the seam lines k = 0 and n3c of the coarse level.
template <class T> __device__ __noinline__ void mg_corser(const MgEq &E, int l)
{
    const Cluster cl = Cluster::self();
    const MgView<T> L = mg_view(E, l + 1, T(0));
    const int ld = E.ld, n1c = L.n1, n3c = L.n3, seam = E.seam_keep;
    const T *rf = sizeof(T) == 8 ? (const T *)E.rc : (const T *)E.rc32;
    T *fc = const_cast<T *>(L.f);
    const int tot = (n1c + 1) * (n3c + 1);
    const RowSplit split(n1c + 1);
    for (int idx = cl.tid(); idx < tot; idx += cl.nthr()) {
        int k, i;
        split(idx, k, i);
        T t = T(0);
        if (i >= 1 && i <= n1c - 1 && k >= 1 && k <= n3c - 1) {
            const T *q = rf + (i + i) + ld * (k + k);
            const T c0 = q[0], ip = q[1], im = q[-1], kp = q[ld], km = q[-ld];
            const T pp = q[1 + ld], pm = q[1 - ld], mp = q[-1 + ld], mm = q[-1 - ld];
            t = mg_full_weight(c0, ip, im, kp, km, pp, pm, mp, mm);
        } else if (seam && i >= 1 && i <= n1c - 1) {
            t = rf[i + ld * k];
        }
        fc[idx] = t;
        L.v[idx] = T(0);
    }
    cl.sync();
}

// finer (PRB:2721-2803): bilinear prolongation of the coarse correction added
// to the fine solution.
template <class T> __device__ __noinline__ void mg_finer(const MgEq &E, int l)
{
    const Cluster cl = Cluster::self();
    const MgView<T> Cc = mg_view(E, l, T(0)), L = mg_view(E, l - 1, T(0));
    const int tot = (L.n1 + 1) * (L.n3 + 1);
    const RowSplit split(L.n1 + 1);
    for (int idx = cl.tid(); idx < tot; idx += cl.nthr()) {
        int k, i;
        split(idx, k, i);
        const T *q = Cc.v + (i >> 1) + Cc.ld * (k >> 1);
        const bool io = i & 1, ko = k & 1;
        const T p = mg_prolong(io, ko, q[0], io ? q[1] : T(0), ko ? q[Cc.ld] : T(0), io && ko ? q[1 + Cc.ld] : T(0));
        T *v = L.v + i + L.ld * k;
        *v = p + *v;
    }
    cl.sync();
}

// The FMG-flavoured down and up legs of PRB:1869-1893.  relax(l, restricted):
// a relaxation on level l, with the residual when a restriction follows;
// level 1 always ends a leg or the cycle and needs it.
template <class T, class Relax> __device__ __forceinline__ void mg_legs(const MgEq &E, Relax relax)
{
    const int nlev = E.nlev;
    if (nlev < 2) return;
    for (int l = 1; l <= nlev - 1; ++l) {
        mg_corser<T>(E, l);
        relax(l + 1, l + 1 < nlev);
    }
    for (int ifmg = 0; ifmg <= nlev - 2; ++ifmg) {
        for (int l = nlev; l >= nlev - ifmg; --l) {
            mg_finer<T>(E, l);
            relax(l - 1, l == nlev - ifmg);
        }
        for (int l = nlev - ifmg - 1; l <= nlev - 1; ++l) {
            mg_corser<T>(E, l);
            relax(l + 1, l + 1 < nlev);
        }
    }
    for (int l = nlev; l >= 2; --l) {
        mg_finer<T>(E, l);
        relax(l - 1, false);
    }
}

// The equation's descriptor in shared memory: behind a global pointer every
// field would come from L2 again after each cluster barrier.
__device__ __forceinline__ void mg_descriptor(MgEq &dst, const MgEq &src)
{
    for (int q = threadIdx.x; q < (int)(sizeof(MgEq) / 4); q += blockDim.x) ((unsigned *)&dst)[q] = ((const unsigned *)&src)[q];
    __syncthreads();
}

// poisson2 / poisson3 (PRB:1796-1927 / PRB:1930-2059).
// This form, on global memory, serves the reference's line order and the
// grids whose levels do not fit a cluster's shared memory (prb_resident.cu).
__global__ void __maxnreg__(255) k_mg_solve(const MgEq *eqs, int first_eq)
{
    __shared__ ClMaxState s_max;
    __shared__ MgEq E;
    const Cluster cl = Cluster::self();
    mg_descriptor(E, eqs[first_eq + blockIdx.x / cl.size]);
    if (*E.abort == GB_RUN_DONE) return;   // a gang member past its last step (the same for every CTA)
    int turn = 0;
    const int ld = E.ld, np = E.np, nlev = E.nlev;
    const int imax = (E.which == 2) ? E.nr + 1 : E.nr;
    const int n1 = E.lev[1].n1;
    double *psif = E.psif, *psi = E.psi, *psip = E.psip;
    const int rows = imax + 1, tot = rows * (np + 1);
    const RowSplit split(rows);
    // initial guess 2 psi - psip; level-1 right-hand side packed
    for (int idx = cl.tid(); idx < tot; idx += cl.nthr()) {
        int k, i;
        split(idx, k, i);
        const int c = i + ld * k;
        psif[c] = 2.0 * psi[c] - psip[c];
        if (i <= n1) E.lev[1].f[(size_t)k * (n1 + 1) + i] = E.rhs[c];
    }
    cl.sync();
    int status = GB_MAXSWEEPS, sweeps = 0, nan1 = 0;
    double res1 = 0.0;
    auto relax = [&](int l, bool restricted) {
        mg_sweeps<double>(E, l);
        if (l != 1 && !restricted) return;
        int nan;
        const double m = mg_residual<double>(E, l, E.rc, ld, &nan);
        if (l == 1) {
            res1 = cl_max(cl, s_max, turn, m, nan);
            nan1 = nan;
        } else {
            cl.sync();
        }
    };
    for (int sweep = 1; sweep <= E.maxsweeps; ++sweep) {
        sweeps = sweep;
        if (sweep != 1) {
            for (int idx = cl.tid(); idx < tot; idx += cl.nthr()) {
                int k, i;
                split(idx, k, i);
                const int c = i + ld * k;
                const double pf = psip[c] + E.sor * (psif[c] - psip[c]);
                psif[c] = pf;
                psip[c] = pf;
            }
            cl.sync();
        }
        if (sweep == 1 || nlev == 1) {
            relax(1, true);
            for (int idx = cl.tid(); idx < tot; idx += cl.nthr()) {
                int k, i;
                split(idx, k, i);
                psip[i + ld * k] = psif[i + ld * k];
            }
            cl.sync();
        }
        mg_legs<double>(E, relax);
        // The last relax of a sweep is on level 1; its NaN flag decides.
        if (nan1) {
            status = GB_NAN;
            break;
        }
        if (res1 < E.tolcon) {
            // the tank: v on k = 1..np-1, u on k = 1..np, zero side walls
            // (velvor2dhorconvtank.f:1032-1043, :1129-1140)
            const int kend = (E.which == 2) ? np - 1 : np;
            for (int idx = cl.tid(); idx < tot; idx += cl.nthr()) {
                int k, i;
                split(idx, k, i);
                const int c = i + ld * k;
                psip[c] = psi[c];
                if (i == 0 || i == imax || (E.xwall && (k == 0 || k > kend))) psi[c] = 0.0;
                else psi[c] = psif[c];
            }
            if (E.xwall && E.which == 3)
                for (int i = cl.tid(); i <= imax; i += cl.nthr()) psi[GIX(i, np + 1, ld)] = 0.0;
            status = GB_OK;
            break;
        }
    }
    if (cl.tid() == 0) {
        E.status[0] = status;
        E.status[1] = sweeps;
        *E.resmax = res1;
        if (status == GB_NAN || (status == GB_MAXSWEEPS && E.stop_on_max)) *E.abort = 1;
    }
    cl.sync();   // no CTA leaves while another may still read its reduction slot
}

// ---------------------------------------------------------------------------
// Mixed precision (GB_PRB_MIXED): FP64 defect correction around the
// reference's sweep schedule run in FP32 on the correction equation A e = r.
// A dependent FP32 operation costs a few cycles where an FP64 one costs tens
// (and an FP64 division hundreds) on this part, and the line eliminations are
// linear recurrences that FP32 may split over a warp's lanes (warpline.cuh).
// psif holds the FP64 iterate.
// ---------------------------------------------------------------------------
__global__ void __maxnreg__(128) k_mg_solve_mixed(const MgEq *eqs, int first_eq)
{
    __shared__ ClMaxState s_max;
    __shared__ MgEq E;
    const Cluster cl = Cluster::self();
    mg_descriptor(E, eqs[first_eq + blockIdx.x / cl.size]);
    if (*E.abort == GB_RUN_DONE) return;   // a gang member past its last step (the same for every CTA)
    int turn = 0;
    const int ld = E.ld, np = E.np;
    const int imax = (E.which == 2) ? E.nr + 1 : E.nr;
    const int n1 = E.lev[1].n1, n3 = E.lev[1].n3;
    double *psif = E.psif, *psi = E.psi, *psip = E.psip;
    const int rows = imax + 1, tot = rows * (np + 1);
    const RowSplit split(rows);
    for (int idx = cl.tid(); idx < tot; idx += cl.nthr()) {
        int k, i;
        split(idx, k, i);
        const int c = i + ld * k;
        psif[c] = 2.0 * psi[c] - psip[c];
        if (i <= n1) E.lev[1].f[(size_t)k * (n1 + 1) + i] = E.rhs[c];
    }
    for (int idx = cl.tid(); idx < ld * (n3 + 1); idx += cl.nthr()) E.psif32[idx] = 0.f;
    cl.sync();
    auto relax = [&](int l, bool restricted) {
        mg_sweeps<float>(E, l);
        if (!restricted) return;
        int nan;
        mg_residual<float>(E, l, E.rc32, ld, &nan);
        cl.sync();
    };
    const int nrow = (E.which == 2) ? n1 : n1 - 1;
    const RowSplit inner(nrow);
    int status = GB_MAXSWEEPS, cycles = 0;
    double res = 0.0;
    for (int it = 0;; ++it) {
        // FP64 residual of the iterate; its FP32 copy is the cycle's right-hand side
        int nan;
        const double m = mg_residual<double>(E, 1, E.lev[1].f32, n1 + 1, &nan);
        res = cl_max(cl, s_max, turn, m, nan);
        if (nan) { status = GB_NAN; break; }
        if (res < E.tolcon) { status = GB_OK; break; }
        if (it == E.maxsweeps) break;
        relax(1, E.nlev > 1);
        mg_legs<float>(E, relax);
        // psi += w e, and e = 0 for the next cycle
        const double w = (it == 0) ? 1.0 : E.sor;
        for (int idx = cl.tid(); idx < nrow * (n3 + 1); idx += cl.nthr()) {
            int k, i;
            inner(idx, k, i);
            const int c = i + 1 + ld * k;
            psif[c] += w * (double)E.psif32[c];
            E.psif32[c] = 0.f;
        }
        cl.sync();
        cycles = it + 1;
    }
    if (status == GB_OK) {
        for (int idx = cl.tid(); idx < tot; idx += cl.nthr()) {
            int k, i;
            split(idx, k, i);
            const int c = i + ld * k;
            psip[c] = psi[c];
            psi[c] = (i == 0 || i == imax) ? 0.0 : psif[c];
        }
    }
    if (cl.tid() == 0) {
        E.status[0] = status;
        E.status[1] = cycles;
        *E.resmax = res;
        if (status == GB_NAN || (status == GB_MAXSWEEPS && E.stop_on_max)) *E.abort = 1;
    }
    cl.sync();
}

// FP32 copies of the radii and the line tables, a block per level.
__global__ void k_mg_factors32(MgEq eq)
{
    const MgLevel &L = eq.lev[1 + blockIdx.x];
    for (int i = threadIdx.x; i <= L.n1 + 1; i += blockDim.x) {
        L.rvi32[i] = (float)L.rvi[i];
        L.rvq32[i] = (float)L.rvq[i];
    }
    if (threadIdx.x != 0) return;
    if (eq.which == 2) pdma32_fold(L.fac, L.n1, L.fac32);
    else tdma32_fold(L.fac, L.n1 - 1, L.fac32);
}

// Factored line matrices of every level (one thread), the coefficients of
// relax2 (PRB:2128-2156) and relax3 (PRB:2421-2436); for the annulus those
// of velvor2dnewsch3.4.f:2104-2131 and :2401-2408 with the per-row 1/r and
// 1/r^2 they use.
__global__ void k_mg_factors(MgEq eq, double *work)
{
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    for (int l = 1; l <= eq.nlev; ++l) {
        const MgLevel &L = eq.lev[l];
        const int n1 = L.n1;
        const double hhri = L.hhri, hhpi = L.hhpi, hri = L.hri;
        double *a = work, *b = a + n1 + 2, *c = b + n1 + 2, *d = c + n1 + 2, *e = d + n1 + 2, *w = e + n1 + 2;
        double *fac = (double *)L.fac;
        double *rvi = L.rvi, *rvq = L.rvq;
        for (int i = 0; i <= n1 + 1; ++i) { rvi[i] = 1.0; rvq[i] = 1.0; }
        if (eq.which == 2) {
            for (int i = 1; i <= n1; ++i) {
                const int j = i - 1;
                if (eq.polar) {
                    const double rval = eq.r0 + ((double)i - 0.5) * L.hr;
                    rvi[i] = 1.0 / rval;
                    rvq[i] = rvi[i] * rvi[i];
                    if (i == 1) {
                        a[j] = 0.0; b[j] = 0.0;
                        c[j] = -2.0 * hhri - 2.0 * hhpi * rvq[i] + rvq[i];
                        d[j] = 5.0 / 3.0 * hhri + 4.0 / 3.0 * hri * rvi[i];
                        e[j] = -0.2 * hhri;
                    } else if (i == n1) {
                        a[j] = -0.2 * hhri;
                        b[j] = 5.0 / 3.0 * hhri - 4.0 / 3.0 * hri * rvi[i];
                        c[j] = -2.0 * hhri - 2.0 * hhpi * rvq[i] + rvq[i];
                        d[j] = 0.0; e[j] = 0.0;
                    } else {
                        a[j] = 0.0;
                        b[j] = hhri - 1.5 * hri * rvi[i];
                        c[j] = -(2.0 * hhri + 2.0 * hhpi * rvq[i]) + rvq[i];
                        d[j] = hhri + 1.5 * hri * rvi[i];
                        e[j] = 0.0;
                    }
                } else if (i == 1) {
                    a[j] = 0.0; b[j] = 0.0;
                    c[j] = -2.0 * hhri - 2.0 * hhpi;
                    d[j] = 5.0 / 3.0 * hhri;
                    e[j] = -0.2 * hhri;
                } else if (i == n1) {
                    a[j] = -0.2 * hhri;
                    b[j] = 5.0 / 3.0 * hhri;
                    c[j] = -2.0 * hhri - 2.0 * hhpi;
                    d[j] = 0.0; e[j] = 0.0;
                } else {
                    a[j] = 0.0; b[j] = hhri;
                    c[j] = -(2.0 * hhri + 2.0 * hhpi);
                    d[j] = hhri; e[j] = 0.0;
                }
            }
            factor_pdma(a, b, c, d, e, n1, fac, w);
        } else {
            for (int j = 0; j < n1 - 1; ++j) {
                const int i = j + 1;
                if (eq.polar) {
                    const double rval = (double)i * L.hr + eq.r0;
                    rvi[i] = 1.0 / rval;
                    rvq[i] = rvi[i] * rvi[i];
                    a[j] = hhri - 1.5 * hri * rvi[i];
                    b[j] = -(2.0 * hhri - rvq[i] + 2.0 * hhpi * rvq[i]);
                    c[j] = hhri + 1.5 * hri * rvi[i];
                } else {
                    a[j] = hhri;
                    b[j] = -(2.0 * hhri + 2.0 * hhpi);
                    c[j] = hhri;
                }
            }
            factor_tdma(a, b, c, n1 - 1, fac);
        }
    }
}

// CTAs of a zebra solve: those asked for, or the largest cluster, or one for a
// small grid of no more than 32 lines (8 x 16 .. 16 x 32: 3 to 11 % faster; 8 x 64
// lines FP64 8 % slower, on one).
static int prb_mg_ctas(const gb_prb *h)
{
    if (h->mg_spread) return std::min(h->mg_spread, h->mg_ctas);
    return cl_small_grid(h->p.nr, h->p.np) && h->p.np <= 32 ? 1 : h->mg_ctas;
}

int prb_mg_create(gb_prb *h)
{
    const gb_prb_params &p = h->p;
    const int nr = p.nr, np = p.np, nlev = h->nlev;
    const int ld = h->dev.ld;
    const double dr = h->dev.dr, dp = h->dev.dp;
    if (nr > MG_MAX_NR) {
        gb_set_error("nr=%d exceeds the multigrid kernel's line length", nr);
        return GB_ERR_INVALID;
    }
    if (np % (1 << nlev) != 0) {
        gb_set_error("np=%d must be divisible by 2^nlev=%d so that every multigrid level has an even number of lines", np, 1 << nlev);
        return GB_ERR_INVALID;
    }
    // pool: per equation psif, rc (full) + per level v, f + factors; plus work
    size_t per_eq = 2 * (size_t)ld * (np + 1) + (size_t)ld * (np + 1) + 8;   // psif, rc; psif32 + rc32
    for (int l = 1; l <= nlev; ++l) {
        const int n1 = nr * 2 / (1 << l), n3 = np * 2 / (1 << l);
        per_eq += 2 * (size_t)(n1 + 1) * (n3 + 1) + pdma_fac_len(n1 + 2) + 2 * (size_t)(n1 + 2);
        // FP32: v32, f32, fac32, rvi32, rvq32 (counted in doubles, rounded up)
        per_eq += ((2 * (size_t)(n1 + 1) * (n3 + 1) + pdma32_len(n1) + 2 * (size_t)(n1 + 2)) + 1) / 2 + 8;
    }
    const size_t work = 8 * (size_t)(nr + 2);
    cudaError_t e = cudaMalloc(&h->mg_pool, sizeof(double) * (2 * per_eq + work));
    if (e != cudaSuccess) { gb_set_error("multigrid pool: %s", cudaGetErrorString(e)); return GB_ERR_ALLOC; }
    cudaMemset(h->mg_pool, 0, sizeof(double) * (2 * per_eq + work));
    double *wk = h->mg_pool + 2 * per_eq;
    for (int q = 0; q < 2; ++q) {
        MgEq &E = h->eq_host[q];
        memset(&E, 0, sizeof(E));
        E.which = q == 0 ? 2 : 3;
        E.nr = nr; E.np = np; E.ld = ld; E.nlev = nlev;
        E.mode = p.smoother; E.maxsweeps = p.maxsweeps; E.tolcon = p.tolcon; E.sor = p.sor;
        E.polar = p.variant == GB_PRB_ANNULUS || p.variant == GB_PRB_TAYCOU;
        E.nrelax = p.variant == GB_PRB_ANNULUS ? 3 : 1;
        E.seam_keep = p.variant == GB_PRB_ANNULUS;
        E.xwall = p.variant == GB_PRB_TANK || p.variant == GB_PRB_DVD;
        if (E.xwall && p.precision != GB_PRB_FP64) return GB_ERR_INVALID;
        E.stop_on_max = p.variant != GB_PRB_ANNULUS;
        E.r0 = p.r0;
        double *base = h->mg_pool + q * per_eq;
        E.psif = base; base += (size_t)ld * (np + 1);
        E.rc = base; base += (size_t)ld * (np + 1);
        float *fbase = (float *)base;
        E.psif32 = fbase; fbase += (size_t)ld * (np + 1);
        E.rc32 = fbase; fbase += (size_t)ld * (np + 1);
        base = (double *)(((uintptr_t)fbase + 15) & ~(uintptr_t)15);
        for (int l = 1; l <= nlev; ++l) {
            MgLevel &L = E.lev[l];
            L.n1 = nr * 2 / (1 << l);
            L.n3 = np * 2 / (1 << l);
            const double hr = dr * (double)(1 << l) * 0.5;
            const double hp = dp * (double)(1 << l) * 0.5;
            L.hr = hr;
            L.hhri = 1.0 / (hr * hr);
            L.hhpi = 1.0 / (hp * hp);
            L.hri = 1.0 / hr;
            const size_t sz = (size_t)(L.n1 + 1) * (L.n3 + 1);
            L.v = base; base += sz;
            L.f = base; base += sz;
            L.fac = base; base += pdma_fac_len(L.n1 + 2);   // >= tdma_fac_len(n1 - 1)
            L.rvi = base; base += (size_t)(L.n1 + 2);
            L.rvq = base; base += (size_t)(L.n1 + 2);
            float *fb = (float *)base;
            L.v32 = fb; fb += sz;
            L.f32 = fb; fb += sz;
            fb = (float *)(((uintptr_t)fb + 15) & ~(uintptr_t)15);   // copied 16 bytes at a time
            L.fac32 = fb; fb += pdma32_len(L.n1);                    // >= tdma32_len(n1 - 1)
            L.rvi32 = fb; fb += (size_t)(L.n1 + 2);
            L.rvq32 = fb; fb += (size_t)(L.n1 + 2);
            base = (double *)(((uintptr_t)fb + 15) & ~(uintptr_t)15);
        }
        E.psi = h->dev.f[q == 0 ? GB_F_vel : GB_F_uel];
        E.psip = h->dev.f[q == 0 ? GB_F_velp : GB_F_uelp];
        E.rhs = h->dev.f[q == 0 ? GB_F_vrh : GB_F_urh];
        E.status = h->dev.mg_status + 2 * q;
        E.resmax = h->dev.mg_resmax + q;
        E.abort = h->dev.abort;
        k_mg_factors<<<1, 1>>>(E, wk);
        k_mg_factors32<<<nlev, 128>>>(E);
    }
    e = cl_prepare(k_mg_solve, MG_SMEM_BYTES);
    if (e == cudaSuccess) e = cl_prepare(k_mg_solve_mixed, MG_SMEM_BYTES);
    if (e != cudaSuccess) { gb_set_error("multigrid shared memory: %s", cudaGetErrorString(e)); return GB_ERR_CUDA; }
    h->mg_ctas = cl_fit(k_mg_solve, CL_MAX_CTAS, MG_THREADS, MG_SMEM_BYTES);
    e = prb_resident_prepare();
    if (e != cudaSuccess) { gb_set_error("multigrid shared memory: %s", cudaGetErrorString(e)); return GB_ERR_CUDA; }
    prb_mg_plan(h->eq_host, 2, p.precision == GB_PRB_MIXED, prb_mg_ctas(h));
    e = cudaMalloc(&h->eq_dev, sizeof(MgEq) * 2);
    if (e != cudaSuccess) { gb_set_error("multigrid descriptors: %s", cudaGetErrorString(e)); return GB_ERR_ALLOC; }
    cudaMemcpy(h->eq_dev, h->eq_host, sizeof(MgEq) * 2, cudaMemcpyHostToDevice);
    return GB_OK;
}

void prb_mg_destroy(gb_prb *h)
{
    cudaFree(h->mg_pool);
    cudaFree(h->eq_dev);
    h->mg_pool = nullptr;
    h->eq_dev = nullptr;
}

// Plans n equations for clusters of ctas CTAs: in shared memory
// (prb_resident.cu) those that fit, E.smem their bytes, else 0.  Returns
// whether all of them fit.
bool prb_mg_plan(MgEq *eqs, int n, int mixed, int ctas)
{
    bool all = true;
    for (int q = 0; q < n; ++q) {
        prb_resident_plan(eqs[q], mixed, ctas);
        if (eqs[q].smem && prb_resident_fit(mixed, ctas, eqs[q].smem) != ctas) eqs[q].smem = 0;
        all = all && eqs[q].smem;
    }
    return all;
}

// The solves of neq equation descriptors (any instances') in one launch, one
// cluster of ctas CTAs each; smem: the most any of them takes in shared
// memory, 0: on global memory.
cudaError_t prb_mg_launch_eqs(const MgEq *d_eqs, int first, int neq, int mixed, int ctas, int smem, cudaStream_t s)
{
    if (neq <= 0) return cudaSuccess;
    if (smem) return prb_resident_launch(d_eqs, first, neq, mixed, ctas, smem, s);
    if (mixed) return cl_launch(k_mg_solve_mixed, neq, ctas, MG_THREADS_MIXED, MG_SMEM_BYTES, s, d_eqs, first);
    return cl_launch(k_mg_solve, neq, ctas, MG_THREADS, MG_SMEM_BYTES, s, d_eqs, first);
}

int prb_mg_cluster_ctas() { return MG_SPREAD; }

// Refreshes the solve parameters that a caller may change between calls
// (tolerance, sweep limit, smoother, SOR factor) and launches the solves.
int prb_launch_mg(gb_prb *h, int do_v, int do_u, cudaStream_t s)
{
    bool changed = false;
    for (int q = 0; q < 2; ++q) {
        MgEq &E = h->eq_host[q];
        if (E.mode != h->p.smoother || E.maxsweeps != h->p.maxsweeps || E.tolcon != h->p.tolcon || E.sor != h->p.sor) {
            E.mode = h->p.smoother; E.maxsweeps = h->p.maxsweeps; E.tolcon = h->p.tolcon; E.sor = h->p.sor;
            changed = true;
        }
    }
    if (changed) cudaMemcpyAsync(h->eq_dev, h->eq_host, sizeof(MgEq) * 2, cudaMemcpyHostToDevice, s);
    const int first = do_v ? 0 : 1;
    const int n = (do_v ? 1 : 0) + (do_u ? 1 : 0);
    if (n == 0) return GB_OK;
    const int mixed = h->p.precision == GB_PRB_MIXED;
    if (h->p.smoother == GB_SMOOTHER_LEX) {
        GB_CUDA_TRY(prb_mg_launch_eqs(h->eq_dev, first, n, mixed, 1, 0, s));
    } else {
        // v and u in one launch: in shared memory when both fit
        const int smem = h->eq_host[0].smem && h->eq_host[1].smem ? std::max(h->eq_host[0].smem, h->eq_host[1].smem) : 0;
        GB_CUDA_TRY(prb_mg_launch_eqs(h->eq_dev, first, n, mixed, prb_mg_ctas(h), smem, s));
    }
    h->launches += 1;
    return GB_OK;
}

extern "C" int gb_prb_set_solve_spread(gb_prb *h, int ctas)
{
    if (!h || (ctas != 0 && ctas != 1 && ctas != MG_SPREAD)) {
        gb_set_error("gb_prb_set_solve_spread: ctas must be 1 or %d, or 0 for the default", MG_SPREAD);
        return GB_ERR_INVALID;
    }
    if (h->mg_spread != ctas) {
        GB_CUDA_TRY(cudaStreamSynchronize(h->stream));   // queued steps use the present plan
        h->mg_spread = ctas;
        prb_mg_plan(h->eq_host, 2, h->p.precision == GB_PRB_MIXED, prb_mg_ctas(h));
        GB_CUDA_TRY(cudaMemcpy(h->eq_dev, h->eq_host, sizeof(MgEq) * 2, cudaMemcpyHostToDevice));
        if (h->graph_exec) { cudaGraphExecDestroy(h->graph_exec); h->graph_exec = nullptr; }
        if (h->graph_exec1) { cudaGraphExecDestroy(h->graph_exec1); h->graph_exec1 = nullptr; }
    }
    return GB_OK;
}
