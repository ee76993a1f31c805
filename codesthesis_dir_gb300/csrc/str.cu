// Stretched-grid streamfunction multigrid of rcsc.f on sm_103a, FP64,
// bit-identical to the oracle (-fmad=false, IEEE division, the reference's
// order): psi_rr + psi_r / r - psi / r^2 + psi_zz with grid.f's per-level
// finite-difference weights, pentadiagonal r-line and z-line Gauss-Seidel,
// nine-point restriction, bilinear prolongation, plain V-cycle (rcsc.f:
// 1118-1444).
//
// One cluster of CTAs per solve (cluster.cuh; the AXI solver's structure).  Every
// r-line has its own matrix (the z weights of its row shift the diagonal)
// and every z-line its own (the r weights and -1/r^2 of its column), so the
// matrix halves of all line eliminations are done once at creation
// (factor_pdma, one thread per line) and a sweep only carries right-hand
// sides through them.  Line orders: the reference's (r-lines j = 1..n2-1 in
// order, then z-lines i = 1..n1-1, on one CTA: each line needs the one
// before it) or four colours (index mod 4 = 1, 2, 3, 0: a line reads the
// lines one and two away, never one of its colour), each colour's lines in
// parallel.
#include "gbcommon.cuh"
#include "banded.cuh"
#include "cluster.cuh"
#include "meridian.cuh"
#include "str_internal.cuh"
#include "warpline.cuh"

#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <vector>

#define STR_THREADS 256
#define STR_MAXLEV 8

struct StrLevel {
    int n1, n2;
    double *r, *cr, *crr, *czz;
    double *ir, *irr;         // 1/r and 1/(r*r) per row (IEEE, host): the divisors' reciprocals
    double *v, *f;            // packed (n1+1)*(n2+1)
    double *fac_r, *fac_z;    // per r-line j (pdma_fac_len(n1-1) each), per z-line i (pdma_fac_len(n2-1))
    // mixed precision: FP32 copies (the factors as warpline.cuh's tables)
    float *r32, *cr32, *crr32, *czz32, *v32, *f32, *fac_r32, *fac_z32;
};

struct StrDev {
    int nlev, nrel, maxsweeps, mode;
    double tolcon;
    double *rc;               // the residual of the level it was last formed on, pitch n1 + 1
    float *rc32;              // the same for the FP32 correction cycles
    double *io_psi, *io_rhs;  // level-1 (n1+1) x (n2+1) staging of the caller's arrays
    StrLevel lev[STR_MAXLEV];
    int *status;              // [0] status, [1] sweeps
    int *abort;               // optional (a time loop's flag): the solve is skipped while it is set and
                              // sets it to 1 when the residual is a NaN
};

#define CR(i, k) L.cr[3 * ((i) - 1) + (k) - 1]
#define CRR(i, k) L.crr[4 * ((i) - 1) + (k) - 1]
#define CZZ(j, k) L.czz[4 * ((j) - 1) + (k) - 1]

// Matrix of r-line j (rcsc.f:1228-1252) or z-line i (rcsc.f:1265-1285).
__device__ void str_line_matrix(const StrLevel &L, int dir, int line, double *a, double *b, double *c, double *dd,
                                double *e)
{
    const int n1 = L.n1, n2 = L.n2;
    if (dir == 0) {
        const int j = line;
        for (int i = 1; i <= n1 - 1; ++i) {
            const int q = i - 1;
            const double r = L.r[i];
            if (i <= n1 / 2) {
                a[q] = 0.0;
                b[q] = CRR(i, 1) + CR(i, 1) / r;
                c[q] = CRR(i, 2) + CR(i, 2) / r - 1.0 / (r * r);
                dd[q] = CRR(i, 3) + CR(i, 3) / r;
                e[q] = CRR(i, 4);
            } else {
                a[q] = CRR(i, 1);
                b[q] = CRR(i, 2) + CR(i, 1) / r;
                c[q] = CRR(i, 3) + CR(i, 2) / r - 1.0 / (r * r);
                dd[q] = CRR(i, 4) + CR(i, 3) / r;
                e[q] = 0.0;
            }
            if (j <= n2 / 2) c[q] = c[q] + CZZ(j, 2);
            else c[q] = c[q] + CZZ(j, 3);
        }
    } else {
        const int i = line;
        const double r = L.r[i];
        for (int j = 1; j <= n2 - 1; ++j) {
            const int q = j - 1;
            if (j <= n2 / 2) {
                a[q] = 0.0;
                b[q] = CZZ(j, 1);
                c[q] = CZZ(j, 2) - 1.0 / (r * r);
                dd[q] = CZZ(j, 3);
                e[q] = CZZ(j, 4);
            } else {
                a[q] = CZZ(j, 1);
                b[q] = CZZ(j, 2);
                c[q] = CZZ(j, 3) - 1.0 / (r * r);
                dd[q] = CZZ(j, 4);
                e[q] = 0.0;
            }
            if (i <= n1 / 2) c[q] = c[q] + CRR(i, 2) + CR(i, 2) / r;
            else c[q] = c[q] + CRR(i, 3) + CR(i, 2) / r;
        }
    }
}

struct StrJob {
    int lev, dir, line;
};

__global__ void k_str_factors(const __grid_constant__ StrDev d, const StrJob *jobs, int njobs, double *work, int wstride)
{
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= njobs) return;
    const StrJob J = jobs[q];
    const StrLevel &L = d.lev[J.lev];
    const int n = J.dir == 0 ? L.n1 - 1 : L.n2 - 1;
    double *w = work + (size_t)q * wstride;
    double *a = w, *b = w + n, *c = w + 2 * n, *dd = w + 3 * n, *e = w + 4 * n, *scratch = w + 5 * n;
    str_line_matrix(L, J.dir, J.line, a, b, c, dd, e);
    double *fac = J.dir == 0 ? L.fac_r + (size_t)(J.line - 1) * pdma_fac_len(n) : L.fac_z + (size_t)(J.line - 1) * pdma_fac_len(n);
    factor_pdma(a, b, c, dd, e, n, fac, scratch);
}

// ---------------------------------------------------------------------------
// The solve.  One cluster of CTAs per solve (cluster.cuh); level l's
// correction v and right-hand side f are (0:n1, 0:n2) arrays of pitch n1 + 1,
// the residual rc the same with the pitch of the level it was formed on.
// T is double for the reference's arithmetic and float for the correction
// cycles of the mixed solve.
// ---------------------------------------------------------------------------
template <class T> struct StrView {
    int n1, n2, ld;
    T *v;
    const T *f;
    const T *cr, *crr, *czz;
    const T *r, *ir, *irr;    // double: r, 1/r, 1/(r r); float: r only
    const T *fac[2];          // r-lines, z-lines
};
__device__ __forceinline__ StrView<double> str_view(const StrLevel &L, double)
{
    return {L.n1, L.n2, L.n1 + 1, L.v, L.f, L.cr, L.crr, L.czz, L.r, L.ir, L.irr, {L.fac_r, L.fac_z}};
}
__device__ __forceinline__ StrView<float> str_view(const StrLevel &L, float)
{
    return {L.n1, L.n2, L.n1 + 1, L.v32, L.f32, L.cr32, L.crr32, L.czz32, L.r32, nullptr, nullptr, {L.fac_r32, L.fac_z32}};
}
#define V(i, j) L.v[(i) + L.ld * (j)]
#define F(i, j) L.f[(i) + L.ld * (j)]

// x / r(i): the IEEE quotient, or a product with the rounded reciprocal
__device__ __forceinline__ double str_over_r(const StrView<double> &L, int i, double x) { return div_by_rcp(x, L.r[i], L.ir[i]); }
__device__ __forceinline__ float str_over_r(const StrView<float> &L, int i, float x) { return x * (1.0f / L.r[i]); }
__device__ __forceinline__ double str_over_rr(const StrView<double> &L, int i, double x)
{
    const double r = L.r[i];
    return div_by_rcp(x, r * r, L.irr[i]);
}
__device__ __forceinline__ float str_over_rr(const StrView<float> &L, int i, float x)
{
    const float ir = 1.0f / L.r[i];
    return x * (ir * ir);
}

// Right-hand sides of r-line j at row i (rcsc.f:1246-1252) and of z-line i at
// row j (rcsc.f:1279-1290).
template <class T> __device__ __forceinline__ T str_rhs(const StrView<T> &L, int dir, int i, int j)
{
    const T *crr = L.crr + 4 * (i - 1), *cr = L.cr + 3 * (i - 1), *czz = L.czz + 4 * (j - 1);
    if (dir == 0) {
        if (j <= L.n2 / 2) return -(czz[0] * V(i, j - 1) + czz[2] * V(i, j + 1) + czz[3] * V(i, j + 2)) + F(i, j);
        return -(czz[0] * V(i, j - 2) + czz[1] * V(i, j - 1) + czz[3] * V(i, j + 1)) + F(i, j);
    }
    const T over = str_over_r(L, i, cr[0] * V(i - 1, j) + cr[2] * V(i + 1, j));
    if (i <= L.n1 / 2) return -(crr[0] * V(i - 1, j) + crr[2] * V(i + 1, j) + crr[3] * V(i + 2, j) + over) + F(i, j);
    return -(crr[0] * V(i - 2, j) + crr[1] * V(i - 1, j) + crr[3] * V(i + 1, j) + over) + F(i, j);
}

// f - L v at (i, j) (relax's residual, rcsc.f:1300-1330)
template <class T> __device__ __forceinline__ T str_resid(const StrView<T> &L, int i, int j)
{
    const T *crr = L.crr + 4 * (i - 1), *cr = L.cr + 3 * (i - 1), *czz = L.czz + 4 * (j - 1);
    const T vc = V(i, j), vm = V(i - 1, j), vp = V(i + 1, j), vd = V(i, j - 1), vu = V(i, j + 1);
    const T over = str_over_r(L, i, cr[0] * vm + cr[1] * vc + cr[2] * vp);
    const T overq = str_over_rr(L, i, vc);
    T t;
    if (i <= L.n1 / 2) t = crr[0] * vm + crr[1] * vc + crr[2] * vp + crr[3] * V(i + 2, j) + over - overq;
    else t = crr[0] * V(i - 2, j) + crr[1] * vm + crr[2] * vc + crr[3] * vp + over - overq;
    if (j <= L.n2 / 2) t = t + czz[0] * vd + czz[1] * vc + czz[2] * vu + czz[3] * V(i, j + 2);
    else t = t + czz[0] * V(i, j - 2) + czz[1] * vd + czz[2] * vc + czz[3] * vu;
    return F(i, j) - t;
}

// Dynamic shared memory of a solve: per staged line its n right-hand sides
// and its factors.
#define STR_SMEM_BYTES (160 * 1024)

// The nl lines first, first + step, ... of one direction (DIR 0: r-lines j,
// DIR 1: z-lines i), which read none of one another: the four-colour order's
// colours, or one line of the reference's order.  Each CTA takes a contiguous
// share, in batches that fit its shared memory: the lines' factors are copied
// there asynchronously (read once, coalesced: fetched from L2 inside an
// elimination they cost each row more than its arithmetic) while all threads
// form the right-hand sides, the lines are eliminated (FP64: one thread per
// line in the reference's order; FP32: up to 32 lanes per line), the solutions
// go back.  (Not inlined: one copy per type and direction keeps the
// eliminations' register blocks free of spills.)
template <class T, int DIR>
__device__ __noinline__ void str_lines(const StrLevel &lev, int first, int step, int nl)
{
    extern __shared__ __align__(16) unsigned char s_str[];
    constexpr bool F64 = sizeof(T) == 8;
    T *smem = (T *)s_str;
    const Cluster cl = Cluster::self();
    const StrView<T> L = str_view(lev, T(0));
    const int n = DIR == 0 ? L.n1 - 1 : L.n2 - 1;
    const int flen = (int)(F64 ? pdma_fac_len(n) : pdma32_len(n));
    const int fpitch = F64 ? flen | 1 : flen;
    const int lpitch = F64 ? 0 : wl_pitch(n), lg = F64 ? 0 : wl_log2m(n);
    const int share = (nl + cl.size - 1) / cl.size;
    const int t0 = cl.rank * share, t1 = min(nl, t0 + share);
    const int words = (int)(STR_SMEM_BYTES / sizeof(T));
    int B = F64 ? (words - n) / (n + fpitch) : words / (lpitch + fpitch);
    const bool staged = B >= 1;       // a line with its factors fits (n up to 2900 in FP64)
    if (!staged) B = 1;
    B = min(B, min(share, (int)blockDim.x));
    T *sfac = smem, *x = staged ? smem + B * fpitch : smem;
    for (int b0 = t0; b0 < t1; b0 += B) {
        const int nb = min(B, t1 - b0), pitch = nb | 1;
        // FP64: [row][line], odd pitch; FP32: [line][row], padded per lane
        auto at = [&](int t, int q) -> T & { return F64 ? x[q * pitch + t] : x[t * lpitch + wl_slot(lg, q)]; };
        if (staged)
            for (int t = 0; t < nb; ++t)
                async_copy(sfac + t * fpitch, L.fac[DIR] + (size_t)(first + step * (b0 + t) - 1) * flen, flen, threadIdx.x,
                           blockDim.x);
        if (DIR == 0) {
            const RowSplit split(n);
            for (int idx = threadIdx.x; idx < nb * n; idx += blockDim.x) {
                int t, q;
                split(idx, t, q);
                at(t, q) = str_rhs<T>(L, 0, q + 1, first + step * (b0 + t));
            }
        } else {
            const RowSplit split(nb);
            for (int idx = threadIdx.x; idx < nb * n; idx += blockDim.x) {
                int q, t;
                split(idx, q, t);
                at(t, q) = str_rhs<T>(L, 1, first + step * (b0 + t), q + 1);
            }
        }
        if constexpr (!F64) {   // rows past the line's end
            const int pad = wl_rows(n) - n;
            for (int idx = threadIdx.x; idx < nb * pad; idx += blockDim.x) at(idx / pad, n + idx % pad) = T(0);
        }
        async_copy_wait();
        __syncthreads();
        if constexpr (F64) {
            if ((int)threadIdx.x < nb) {
                const int t = threadIdx.x;
                if (staged) pdma_staged(sfac + t * fpitch, n, x + t, pitch);
                else pdma_staged(L.fac[DIR] + (size_t)(first + step * (b0 + t) - 1) * flen, n, x + t, pitch);
            }
        } else {
            if (staged) wl_lines<true, false, true>(sfac, fpitch, n, x, lpitch, nb);
            else wl_lines<true, false, true>(L.fac[DIR] + (size_t)(first + step * b0 - 1) * flen, (size_t)step * flen, n, x, lpitch, nb);
        }
        __syncthreads();
        if (DIR == 0) {
            const RowSplit split(n);
            for (int idx = threadIdx.x; idx < nb * n; idx += blockDim.x) {
                int t, q;
                split(idx, t, q);
                V(q + 1, first + step * (b0 + t)) = at(t, q);
            }
        } else {
            const RowSplit split(nb);
            for (int idx = threadIdx.x; idx < nb * n; idx += blockDim.x) {
                int q, t;
                split(idx, q, t);
                V(first + step * (b0 + t), q + 1) = at(t, q);
            }
        }
        if (b0 + B < t1) __syncthreads();
    }
    cl.sync();
}

// relax's line sweeps (rcsc.f:1197-1299), nrel of them, in place on v.  The
// reference also forms the residual after every sweep; only the last one is
// ever read, and the caller forms that.
template <class T> __device__ __forceinline__ void str_sweeps(const StrDev &d, int klev)
{
    const StrLevel &L = d.lev[klev];
    const int nj = L.n2 - 1, ni = L.n1 - 1;
    for (int irel = 0; irel < d.nrel; ++irel) {
        if (d.mode == GB_SMOOTHER_LEX) {
            for (int j = 1; j <= nj; ++j) str_lines<T, 0>(L, j, 1, 1);
            for (int i = 1; i <= ni; ++i) str_lines<T, 1>(L, i, 1, 1);
        } else {
            for (int c = 1; c <= 4; ++c)
                if (c <= nj) str_lines<T, 0>(L, c, 4, (nj - c) / 4 + 1);
            for (int c = 1; c <= 4; ++c)
                if (c <= ni) str_lines<T, 1>(L, c, 4, (ni - c) / 4 + 1);
        }
    }
}

// The residual of level klev into rc (not followed by a barrier), its
// largest magnitude and whether one is a NaN over the calling thread's points.
template <class T, class R> __device__ __noinline__ T str_residual(const StrLevel &lev, R *rc, int *nan_out)
{
    const Cluster cl = Cluster::self();
    const StrView<T> L = str_view(lev, T(0));
    const int ni = L.n1 - 1, tot = ni * (L.n2 - 1);
    const RowSplit split(ni);
    T m = T(0);
    int nan = 0;
    for (int idx = cl.tid(); idx < tot; idx += cl.nthr()) {
        int j, i;
        split(idx, j, i);
        ++i;
        ++j;
        const T r = str_resid<T>(L, i, j);
        rc[i + L.ld * j] = (R)r;
        const T a = fabs(r);
        if (a != a) nan = 1;
        if (a > m) m = a;
    }
    *nan_out = nan;
    return m;
}

// corser (rcsc.f:1343-1390): restriction of rc into the coarse right-hand
// side; rows and columns 0 and n1c of the coarse level (n1 for both
// directions) are zero, as are the boundary rows the restriction does not
// reach (never read by the coarse relax); the coarse correction is zero.
template <class T> __device__ __noinline__ void str_corser(const StrLevel &coarse, const T *rc)
{
    const Cluster cl = Cluster::self();
    const StrView<T> L = str_view(coarse, T(0));
    const int ld = 2 * L.n1 + 1;
    const int n1c = L.n1, n2c = L.n2;
    const int tot = (n1c + 1) * (n2c + 1);
    const RowSplit split(n1c + 1);
    T *fc = const_cast<T *>(L.f);
    for (int idx = cl.tid(); idx < tot; idx += cl.nthr()) {
        int j, i;
        split(idx, j, i);
        T temp = T(0);
        if (i >= 1 && i <= n1c - 1 && j >= 1 && j <= n2c - 1 && j != n1c) {
            const T *q = rc + (i + i) + ld * (j + j);
            temp = q[0];
            temp = temp * T(2) + q[1] + q[-1];
            temp = temp + q[ld] + q[-ld];
            temp = temp * T(2) + q[1 + ld] + q[-1 - ld];
            temp = temp + q[1 - ld] + q[-1 + ld];
            temp = temp * T(0.0625);   // / 16, exactly
        }
        fc[idx] = temp;
        L.v[idx] = T(0);
    }
    cl.sync();
}

// finer (rcsc.f:1392-1444): bilinear prolongation added to the fine level.
// The coarse correction is cleared by the next corser.
template <class T> __device__ __noinline__ void str_finer(const StrLevel &coarse, const StrLevel &fine)
{
    const Cluster cl = Cluster::self();
    const StrView<T> Cc = str_view(coarse, T(0)), L = str_view(fine, T(0));
    const int tot = L.ld * (L.n2 + 1);
    const RowSplit split(L.ld);
    for (int idx = cl.tid(); idx < tot; idx += cl.nthr()) {
        int j, i;
        split(idx, j, i);
        const T *q = Cc.v + (i >> 1) + Cc.ld * (j >> 1);
        T p;
        if (!(i & 1)) p = !(j & 1) ? q[0] : (q[0] + q[Cc.ld]) * T(0.5);
        else if (!(j & 1)) p = (q[0] + q[1]) * T(0.5);
        else p = (q[0] + q[Cc.ld + 1] + q[Cc.ld] + q[1]) * T(0.25);
        L.v[idx] = p + L.v[idx];
    }
    cl.sync();
}

// poisson(psi, rhs, nlev, vel) (rcsc.f:1118-1195) on the staged arrays.
__global__ void __maxnreg__(255) k_str_solve(const __grid_constant__ StrDev d)
{
    __shared__ ClMaxState s_max;
    const Cluster cl = Cluster::self();
    if (d.abort && *d.abort) return;   // the same for every CTA: nothing sets it while the solve runs
    int turn = 0;
    const int nlev = d.nlev;
    const StrView<double> L = str_view(d.lev[1], 0.0);
    const int tp = L.ld * (L.n2 + 1);
    for (int idx = cl.tid(); idx < tp; idx += cl.nthr()) {
        const_cast<double *>(L.f)[idx] = d.io_rhs[idx];
        L.v[idx] = d.io_psi[idx];
    }
    cl.sync();
    // relax on level l and the residual for the restriction or the test
    // that follows; the norm matters on level 1 only (rcsc.f:1180)
    double res1 = 0.0;
    int status = GB_MAXSWEEPS, sweeps = d.maxsweeps, nan1 = 0;
    auto relax = [&](int l, bool restricted) {
        str_sweeps<double>(d, l);
        if (l != 1 && !restricted) return;
        int nan;
        const double m = str_residual<double>(d.lev[l], d.rc, &nan);
        if (l == 1) {
            res1 = cl_max(cl, s_max, turn, m, nan);
            nan1 = nan;
        } else {
            cl.sync();
        }
    };
    for (int sweep = 1; sweep <= d.maxsweeps; ++sweep) {
        if (sweep == 1 || nlev == 1) relax(1, true);
        for (int l = 1; l <= nlev - 1; ++l) {
            str_corser<double>(d.lev[l + 1], d.rc);
            relax(l + 1, l + 1 < nlev);
        }
        for (int l = nlev; l >= 2; --l) {
            str_finer<double>(d.lev[l], d.lev[l - 1]);
            relax(l - 1, false);
        }
        if (nan1) {
            status = GB_NAN;
            sweeps = sweep;
            break;
        }
        if (res1 < d.tolcon) {
            for (int idx = cl.tid(); idx < tp; idx += cl.nthr()) d.io_psi[idx] = L.v[idx];
            status = GB_OK;
            sweeps = sweep;
            break;
        }
    }
    if (cl.tid() == 0) {
        d.status[0] = status;
        d.status[1] = sweeps;
        if (status == GB_NAN && d.abort) *d.abort = 1;
    }
    cl.sync();   // no CTA leaves while another may still read its reduction slot
}

// ---------------------------------------------------------------------------
// Mixed precision (FP32 V-cycles inside FP64 defect correction): each outer
// iteration forms the FP64 residual r = f - L psi of the level-1 iterate
// (relax's own residual expression), stops when max |r| < tolcon, else runs
// one FP32 V-cycle of the same schedule on L e = r from e = 0 and updates
// psi += e in FP64 (rcsc.f's solve has no over-relaxation).
// ---------------------------------------------------------------------------
__global__ void __maxnreg__(255) k_str_solve_mixed(const __grid_constant__ StrDev d)
{
    __shared__ ClMaxState s_max;
    const Cluster cl = Cluster::self();
    if (d.abort && *d.abort) return;
    int turn = 0;
    const int nlev = d.nlev;
    const StrView<double> L = str_view(d.lev[1], 0.0);
    const StrView<float> L32 = str_view(d.lev[1], 0.f);
    const int tp = L.ld * (L.n2 + 1);
    for (int idx = cl.tid(); idx < tp; idx += cl.nthr()) {
        const_cast<double *>(L.f)[idx] = d.io_rhs[idx];
        L.v[idx] = d.io_psi[idx];
        L32.v[idx] = 0.f;
        const_cast<float *>(L32.f)[idx] = 0.f;
    }
    cl.sync();
    auto relax = [&](int l, bool restricted) {
        str_sweeps<float>(d, l);
        if (!restricted) return;
        int nan;
        str_residual<float>(d.lev[l], d.rc32, &nan);
        cl.sync();
    };
    int status = GB_MAXSWEEPS, cycles = 0;
    for (int it = 0;; ++it) {
        int nan;
        const double m = str_residual<double>(d.lev[1], const_cast<float *>(L32.f), &nan);
        const double res = cl_max(cl, s_max, turn, m, nan);
        if (nan) { status = GB_NAN; break; }
        if (res < d.tolcon) { status = GB_OK; break; }
        if (it == d.maxsweeps) break;
        relax(1, nlev > 1);
        for (int l = 1; l <= nlev - 1; ++l) {
            str_corser<float>(d.lev[l + 1], d.rc32);
            relax(l + 1, l + 1 < nlev);
        }
        for (int l = nlev; l >= 2; --l) {
            str_finer<float>(d.lev[l], d.lev[l - 1]);
            relax(l - 1, false);
        }
        // psi += e, and e = 0 for the next cycle
        for (int idx = cl.tid(); idx < tp; idx += cl.nthr()) {
            L.v[idx] += (double)L32.v[idx];
            L32.v[idx] = 0.f;
        }
        cl.sync();
        cycles = it + 1;
    }
    if (status == GB_OK)
        for (int idx = cl.tid(); idx < tp; idx += cl.nthr()) d.io_psi[idx] = L.v[idx];
    if (cl.tid() == 0) {
        d.status[0] = status;
        d.status[1] = cycles;
        if (status == GB_NAN && d.abort) *d.abort = 1;
    }
    cl.sync();
}

#undef V
#undef F

// FP32 copies of a level's tables and its line tables: block row y takes
// level y + 1, one thread per r-line, then per z-line.
__global__ void k_str_factors32(const __grid_constant__ StrDev d)
{
    const StrLevel &L = d.lev[1 + blockIdx.y];
    const int a = L.n1, b = L.n2;
    if (blockIdx.x == 0) {
        for (int i = threadIdx.x; i <= a; i += blockDim.x) L.r32[i] = (float)L.r[i];
        for (int q = threadIdx.x; q < 3 * (a - 1); q += blockDim.x) L.cr32[q] = (float)L.cr[q];
        for (int q = threadIdx.x; q < 4 * (a - 1); q += blockDim.x) L.crr32[q] = (float)L.crr[q];
        for (int q = threadIdx.x; q < 4 * (b - 1); q += blockDim.x) L.czz32[q] = (float)L.czz[q];
    }
    const int nr = a - 1, nz = b - 1;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < nz) pdma32_fold(L.fac_r + (size_t)t * pdma_fac_len(nr), nr, L.fac_r32 + (size_t)t * pdma32_len(nr));
    else if (t < nz + nr)
        pdma32_fold(L.fac_z + (size_t)(t - nz) * pdma_fac_len(nz), nz, L.fac_z32 + (size_t)(t - nz) * pdma32_len(nz));
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
struct gb_str {
    StrDev dev;
    double *pool = nullptr;
    int *status = nullptr;
    cudaStream_t stream = nullptr;
    int ctas = 1;             // CTAs per four-colour FP64 solve
    MerDev mer;               // the resident mixed solve (meridian.cu), where its plan fits
    int mer_ctas = 0;         // its CTAs; 0: k_str_solve_mixed
    void *mer_mem = nullptr;
};

// The resident solve's weights: grid.f's in FP32 for every level and in FP64
// for level 1's residual.
__global__ void k_str_weights(const __grid_constant__ StrDev d, const __grid_constant__ MerDev m)
{
    const int l = 1 + blockIdx.y, t = blockIdx.x * blockDim.x + threadIdx.x;
    const StrLevel &L = d.lev[l];
    if (t >= 1 && t < L.n1) {
        const int i = t;
        float4 *c = const_cast<float4 *>(m.lev[l].ci) + 2 * i;
        const float *crr = L.crr32 + 4 * (i - 1), *cr = L.cr32 + 3 * (i - 1);
        c[0] = make_float4(crr[0], crr[1], crr[2], crr[3]);
        c[1] = make_float4(cr[0], cr[1], cr[2], 1.0f / L.r32[i]);
        if (l == 1) {
            const double r = L.r[i];
            const_cast<MerRow *>(m.d_i)[i] = MerRow{{CRR(i, 1), CRR(i, 2), CRR(i, 3), CRR(i, 4)}, {CR(i, 1), CR(i, 2), CR(i, 3)},
                                                    r, L.ir[i], r * r, L.irr[i], 0.0};
        }
    }
    if (t >= 1 && t < L.n2) {
        const int j = t;
        const float *czz = L.czz32 + 4 * (j - 1);
        const_cast<float4 *>(m.lev[l].cj)[j] = make_float4(czz[0], czz[1], czz[2], czz[3]);
        if (l == 1)
            const_cast<MerCol *>(m.d_j)[j] = MerCol{{CZZ(j, 1), CZZ(j, 2), CZZ(j, 3), CZZ(j, 4)}};
    }
}

// Prepares the resident mixed solve; a grid it cannot hold leaves mer_ctas 0.
static cudaError_t str_mer_create(gb_str *h)
{
    const StrDev &d = h->dev;
    MerDev &m = h->mer;
    memset(&m, 0, sizeof(m));
    m.nlev = d.nlev;
    m.penta = 1;
    for (int l = 1; l <= d.nlev; ++l) {
        MerLevel &L = m.lev[l];
        L.n1 = d.lev[l].n1;
        L.n2 = d.lev[l].n2;
        L.fac_r = d.lev[l].fac_r32;
        L.fac_z = d.lev[l].fac_z32;
        L.fac_r_step = (int)pdma32_len(L.n1 - 1);
        L.fac_z_step = (int)pdma32_len(L.n2 - 1);
    }
    m.v = d.lev[1].v;
    h->mer_ctas = mer_fit(m, CL_MAX_CTAS);
    if (!h->mer_ctas) return cudaSuccess;
    h->mer_ctas = mer_alone(m, h->mer_ctas);
    cudaError_t e = cudaMalloc(&h->mer_mem, mer_weight_bytes(m));
    if (e != cudaSuccess) return e;
    mer_weight_layout(m, h->mer_mem);
    k_str_weights<<<dim3(gb_ceil_div((size_t)std::max(m.lev[1].n1, m.lev[1].n2), 128), m.nlev), 128>>>(d, m);
    return cudaDeviceSynchronize();
}

extern "C" int gb_str_destroy(gb_str *h)
{
    if (!h) return GB_OK;
    cudaFree(h->pool);
    cudaFree(h->status);
    cudaFree(h->mer_mem);
    if (h->stream) cudaStreamDestroy(h->stream);
    delete h;
    return GB_OK;
}

extern "C" int gb_str_create(int nlev, const gb_str_level *lv, double tolcon, int maxsweeps, int nrel, int smoother,
                             gb_str **out)
{
    if (!out || !lv || nlev < 1 || nlev >= STR_MAXLEV || maxsweeps < 1 || nrel < 1 ||
        (smoother != GB_SMOOTHER_LEX && smoother != GB_SMOOTHER_ZEBRA)) {
        gb_set_error("gb_str_create: invalid argument");
        return GB_ERR_INVALID;
    }
    *out = nullptr;
    const int n1 = lv[0].n1, n2 = lv[0].n2;
    if (n1 < 4 || n2 < 4 || n1 > 8192 || n2 > 8192) {
        gb_set_error("gb_str_create: level-1 grid %d x %d unsupported", n1, n2);
        return GB_ERR_INVALID;
    }
    for (int l = 0; l < nlev; ++l) {
        if (lv[l].n1 != (n1 >> l) || lv[l].n2 != (n2 >> l) || (l && (lv[l - 1].n1 & 1 || lv[l - 1].n2 & 1)) ||
            lv[l].n1 < 4 || lv[l].n2 < 4 || !lv[l].r || !lv[l].cr || !lv[l].crr || !lv[l].czz) {
            gb_set_error("gb_str_create: level %d must be %d x %d (halvings of level 1, >= 4) with all tables", l + 1,
                         n1 >> l, n2 >> l);
            return GB_ERR_INVALID;
        }
    }
    gb_str *h = new gb_str();
    StrDev &d = h->dev;
    memset(&d, 0, sizeof(d));
    d.nlev = nlev;
    const size_t pts1 = (size_t)(n1 + 1) * (n2 + 1);
    d.nrel = nrel;
    d.maxsweeps = maxsweeps;
    d.mode = smoother;
    d.tolcon = tolcon;
    size_t need = 3 * pts1;
    for (int l = 0; l < nlev; ++l) {
        const size_t a = lv[l].n1, b = lv[l].n2;
        need += 3 * (a + 1) + 3 * (a - 1) + 4 * (a - 1) + 4 * (b - 1) + 2 * (a + 1) * (b + 1);
        need += (b - 1) * pdma_fac_len((int)a - 1) + (a - 1) * pdma_fac_len((int)b - 1);
    }
    // FP32 copies: rc32 and every level's tables (half a double each, rounded up per array)
    size_t need32 = pts1 + 16;
    for (int l = 0; l < nlev; ++l) {
        const size_t a = lv[l].n1, b = lv[l].n2;
        need32 += (a + 1) + 3 * (a - 1) + 4 * (a - 1) + 4 * (b - 1) + 2 * (a + 1) * (b + 1);
        need32 += (b - 1) * pdma32_len((int)a - 1) + (a - 1) * pdma32_len((int)b - 1) + 16;
    }
    const size_t need64 = need;
    need += (need32 + 1) / 2;
    cudaError_t e = cudaMalloc(&h->pool, sizeof(double) * need);
    if (e != cudaSuccess) { delete h; gb_set_error("gb_str_create: %s", cudaGetErrorString(e)); return GB_ERR_ALLOC; }
    cudaMemset(h->pool, 0, sizeof(double) * need);
    double *b = h->pool;
    d.rc = b; b += pts1;
    d.io_psi = b; b += pts1;
    d.io_rhs = b; b += pts1;
    std::vector<StrJob> jobs;
    int wmax = 0;
    for (int l = 0; l < nlev; ++l) {
        StrLevel &L = d.lev[l + 1];
        const int a = lv[l].n1, bb = lv[l].n2;
        L.n1 = a;
        L.n2 = bb;
        L.r = b; b += a + 1;
        L.ir = b; b += a + 1;
        L.irr = b; b += a + 1;
        L.cr = b; b += 3 * (size_t)(a - 1);
        L.crr = b; b += 4 * (size_t)(a - 1);
        L.czz = b; b += 4 * (size_t)(bb - 1);
        L.v = b; b += (size_t)(a + 1) * (bb + 1);
        L.f = b; b += (size_t)(a + 1) * (bb + 1);
        L.fac_r = b; b += (size_t)(bb - 1) * pdma_fac_len((int)a - 1);
        L.fac_z = b; b += (size_t)(a - 1) * pdma_fac_len((int)bb - 1);
        cudaMemcpy(L.r, lv[l].r, sizeof(double) * (a + 1), cudaMemcpyHostToDevice);
        {
            std::vector<double> inv(2 * (size_t)(a + 1));
            for (int i = 0; i <= a; ++i) {
                const double r = lv[l].r[i];
                inv[i] = 1.0 / r;
                inv[a + 1 + i] = 1.0 / (r * r);
            }
            cudaMemcpy(L.ir, inv.data(), sizeof(double) * inv.size(), cudaMemcpyHostToDevice);
        }
        cudaMemcpy(L.cr, lv[l].cr, sizeof(double) * 3 * (a - 1), cudaMemcpyHostToDevice);
        cudaMemcpy(L.crr, lv[l].crr, sizeof(double) * 4 * (a - 1), cudaMemcpyHostToDevice);
        cudaMemcpy(L.czz, lv[l].czz, sizeof(double) * 4 * (bb - 1), cudaMemcpyHostToDevice);
        for (int j = 1; j <= bb - 1; ++j) jobs.push_back({l + 1, 0, j});
        for (int i = 1; i <= a - 1; ++i) jobs.push_back({l + 1, 1, i});
        wmax = std::max(wmax, std::max(a, bb));
    }
    if ((size_t)(b - h->pool) != need64) {
        gb_str_destroy(h);
        gb_set_error("gb_str_create: pool layout mismatch");
        return GB_ERR_CUDA;
    }
    {
        float *fb = (float *)b;
        float *fend = (float *)(h->pool + need);
        d.rc32 = fb; fb += pts1;
        for (int l = 1; l <= nlev; ++l) {
            StrLevel &L = d.lev[l];
            const size_t a = L.n1, bb = L.n2;
            L.r32 = fb; fb += a + 1;
            L.cr32 = fb; fb += 3 * (a - 1);
            L.crr32 = fb; fb += 4 * (a - 1);
            L.czz32 = fb; fb += 4 * (bb - 1);
            L.v32 = fb; fb += (a + 1) * (bb + 1);
            L.f32 = fb; fb += (a + 1) * (bb + 1);
            fb = (float *)(((uintptr_t)fb + 15) & ~(uintptr_t)15);   // the tables are copied 16 bytes at a time
            L.fac_r32 = fb; fb += (bb - 1) * pdma32_len((int)a - 1);
            L.fac_z32 = fb; fb += (a - 1) * pdma32_len((int)bb - 1);
        }
        if (fb > fend) {
            gb_str_destroy(h);
            gb_set_error("gb_str_create: FP32 pool layout overflow");
            return GB_ERR_CUDA;
        }
    }
    const int wstride = 7 * wmax;
    StrJob *djobs = nullptr;
    double *work = nullptr;
    e = cudaMalloc(&djobs, sizeof(StrJob) * jobs.size());
    if (e == cudaSuccess) e = cudaMalloc(&work, sizeof(double) * (size_t)wstride * jobs.size());
    if (e != cudaSuccess) {
        cudaFree(djobs);
        gb_str_destroy(h);
        gb_set_error("gb_str_create: factor scratch");
        return GB_ERR_ALLOC;
    }
    cudaMemcpy(djobs, jobs.data(), sizeof(StrJob) * jobs.size(), cudaMemcpyHostToDevice);
    k_str_factors<<<gb_ceil_div(jobs.size(), 64), 64>>>(d, djobs, (int)jobs.size(), work, wstride);
    e = cudaDeviceSynchronize();
    cudaFree(djobs);
    cudaFree(work);
    if (e == cudaSuccess) {
        k_str_factors32<<<dim3(gb_ceil_div((size_t)n1 + n2, 32), nlev), 32>>>(d);
        e = cudaDeviceSynchronize();
    }
    if (e != cudaSuccess) { gb_set_error("gb_str_create: factors: %s", cudaGetErrorString(e)); gb_str_destroy(h); return GB_ERR_CUDA; }
    e = cudaMalloc(&h->status, 64);
    if (e != cudaSuccess) { gb_str_destroy(h); gb_set_error("gb_str_create: status"); return GB_ERR_ALLOC; }
    d.status = h->status;
    e = cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking);
    if (e != cudaSuccess) { gb_str_destroy(h); gb_set_error("gb_str_create: stream"); return GB_ERR_CUDA; }
    e = cl_prepare(k_str_solve, STR_SMEM_BYTES);
    if (e == cudaSuccess) e = cl_prepare(k_str_solve_mixed, STR_SMEM_BYTES);
    if (e != cudaSuccess) { gb_str_destroy(h); gb_set_error("gb_str_create: shared memory: %s", cudaGetErrorString(e)); return GB_ERR_CUDA; }
    h->ctas = cl_fit(k_str_solve, cl_small_grid(n1, n2) ? 1 : CL_MAX_CTAS, STR_THREADS, STR_SMEM_BYTES);
    e = str_mer_create(h);
    if (e != cudaSuccess) { gb_set_error("gb_str_create: %s", cudaGetErrorString(e)); gb_str_destroy(h); return GB_ERR_CUDA; }
    *out = h;
    return GB_OK;
}

// CTAs per solve.  The reference's line order is one chain of lines, so one
// CTA; otherwise the whole cluster.
static int str_ctas(const gb_str *h, int mode)
{
    if (mode == GB_SMOOTHER_LEX) return 1;
    return h->ctas;
}

// The solve on device arrays (0:n1, 0:n2) with leading dimension n1 + 1,
// queued on stream s with the given tolerance, sweep limit, relaxation count
// and line order: psi is read and, on convergence, written in place; the
// status and sweep (mixed: outer iteration) count go to status[0..1]; abort
// as in StrDev.  mixed != 0 runs the FP32-inner / FP64-outer solve.
cudaError_t gb_str_launch_device(const gb_str *h, double *psi, const double *rhs, int *status, int *abort, int mixed,
                                 double tolcon, int maxsweeps, int nrel, int mode, cudaStream_t s)
{
    StrDev d = h->dev;
    d.tolcon = tolcon;
    d.maxsweeps = maxsweeps;
    d.nrel = nrel;
    d.mode = mode;
    d.io_psi = psi;
    d.io_rhs = const_cast<double *>(rhs);
    d.status = status;
    d.abort = abort;
    if (mixed && mode == GB_SMOOTHER_ZEBRA && h->mer_ctas) {
        MerDev m = h->mer;
        m.tolcon = tolcon;
        m.maxcycles = maxsweeps;
        m.nrel = nrel;
        m.psi = psi;
        m.rhs = rhs;
        m.status = status;
        m.abort = abort;
        return mer_launch(m, h->mer_ctas, s);
    }
    const int ctas = str_ctas(h, mode);
    if (mixed) return cl_launch(k_str_solve_mixed, 1, ctas, STR_THREADS, STR_SMEM_BYTES, s, d);
    return cl_launch(k_str_solve, 1, ctas, STR_THREADS, STR_SMEM_BYTES, s, d);
}

extern "C" int gb_str_poisson(gb_str *h, double *psi, const double *rhs, int ld, int *sweeps)
{
    if (!h || !psi || !rhs) { gb_set_error("gb_str_poisson: null argument"); return GB_ERR_INVALID; }
    const StrDev &d = h->dev;
    const int n1 = d.lev[1].n1, n2 = d.lev[1].n2;
    if (ld < n1 + 1) { gb_set_error("gb_str_poisson: ld %d < n1+1", ld); return GB_ERR_INVALID; }
    const size_t row = sizeof(double) * (size_t)(n1 + 1);
    GB_CUDA_TRY(cudaMemcpy2DAsync(d.io_psi, row, psi, sizeof(double) * (size_t)ld, row, n2 + 1, cudaMemcpyHostToDevice,
                                  h->stream));
    GB_CUDA_TRY(cudaMemcpy2DAsync(d.io_rhs, row, rhs, sizeof(double) * (size_t)ld, row, n2 + 1, cudaMemcpyHostToDevice,
                                  h->stream));
    GB_CUDA_TRY(cl_launch(k_str_solve, 1, str_ctas(h, d.mode), STR_THREADS, STR_SMEM_BYTES, h->stream, d));
    int st[2] = {0, 0};
    GB_CUDA_TRY(cudaMemcpyAsync(st, d.status, sizeof(st), cudaMemcpyDeviceToHost, h->stream));
    GB_CUDA_TRY(cudaStreamSynchronize(h->stream));
    if (st[0] == GB_OK)
        GB_CUDA_TRY(cudaMemcpy2D(psi, sizeof(double) * (size_t)ld, d.io_psi, row, row, n2 + 1, cudaMemcpyDeviceToHost));
    if (sweeps) *sweeps = st[1];
    return st[0];
}
