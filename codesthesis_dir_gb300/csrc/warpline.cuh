// FP32 line eliminations by the lanes of a warp (the correction cycles of the
// mixed-precision solves).
//
// One thread per line is a chain of 2 n dependent rows whose shared-memory
// loads it also has to issue alone: 90 cycles a row, 23 k cycles for the 255
// rows of a 257 x 257 grid's line.  Here W lanes share a line, lane l holding
// rows l M .. l M + M - 1 in registers.  Both halves of an elimination are
// linear recurrences, so a lane first runs its rows from a zero state together
// with the recurrence's homogeneous solutions, the lanes combine (state map,
// state) pairs in a scan of log2 W steps, and each lane repeats its M rows
// from its true incoming state.  The maps' entries decay with the matrix's
// diagonal dominance, as the recurrences themselves do, so a scan step (150
// cycles of shuffles) is only worth taking while the product of the maps it
// reaches over is more than 2^-30, far below FP32 rounding: the fold measures
// that product per line and stores the number of steps with the table (one on
// a square mesh, where a row passes on 0.27 of its state; all log2 W along
// strongly coupled lines).
//
// M is 8 up to 256 rows (W = 4 .. 32, so a warp takes 32 / W lines) and 16 up
// to 512; W is a run-time value.  With M fitted to each level instead (one
// row per lane on the coarsest) every level ran code of its own, and the
// short phases waited for instructions: 2.0 k cycles for a 31-row line.
//
// The pivots are folded into the factors (in FP64, rounded once), so that a
// row is one dependent fused multiply-add:
//   pentadiagonal  z(k) = S(k) r(k) - A(k) z(k-2) - B(k) z(k-1)
//                  x(k) = z(k) - E(k) x(k+2) - D(k) x(k+1)
//   tridiagonal    z(k) = r(k) - F(k) z(k-1),   x(k) = I(k) z(k) - G(k) x(k+1)
// Rows past the end have zero coefficients and leave the state at zero.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

#define WL_MAXM 16

// log2 of the rows per lane and of the lanes per line; lines longer than
// 32 WL_MAXM rows take several segments of that many, one after the other.
__host__ __device__ __forceinline__ int wl_log2m(int n) { return n <= 256 ? 3 : 4; }
__host__ __device__ __forceinline__ int wl_log2w(int n) { return n <= 32 ? 2 : n <= 64 ? 3 : n <= 128 ? 4 : 5; }
__host__ __device__ __forceinline__ int wl_segments(int n) { return n <= 256 ? 1 : (n + 511) / 512; }
// Padded rows of a line, the floats of its table (four words, the first the
// scan steps, then 5 or 3 coefficients a row as
// [segment][coefficient][row in lane][lane]; a multiple of 16 bytes) and the
// pitch of its right-hand side in shared memory (a lane's rows padded to an
// odd stride, lines to an odd pitch: no bank conflicts in either direction).
__host__ __device__ __forceinline__ int wl_rows(int n) { return wl_segments(n) << (wl_log2m(n) + wl_log2w(n)); }
__host__ __device__ __forceinline__ size_t pdma32_len(int n) { return 4 + 5 * (size_t)wl_rows(n); }
__host__ __device__ __forceinline__ size_t tdma32_len(int n) { return 4 + 3 * (size_t)wl_rows(n); }
__host__ __device__ __forceinline__ int wl_slot(int lg, int q) { return q + (q >> lg); }
__host__ __device__ __forceinline__ int wl_pitch(int n) { return (wl_rows(n) + (wl_rows(n) >> wl_log2m(n))) | 1; }

__device__ __forceinline__ size_t wl_table_at(int n, int ncoef, int coef, int k)
{
    const int lg = wl_log2m(n), lw = wl_log2w(n);
    const int seg = k >> (lg + lw), q = k - (seg << (lg + lw));
    return 4 + ((((size_t)(seg * ncoef + coef) << lg) + (q & ((1 << lg) - 1))) << lw) + (q >> lg);
}

// Scan steps a recurrence y(k) = t(k) - b(k) y(k-1) - a(k) y(k-2) needs:
// the smallest s for which every product of 2^s consecutive lanes' state maps
// is below 2^-30 (at most log2 W).  Coefficients cb, ca of the table g (ca < 0:
// first order); back: from the last row to the first.
__device__ inline int wl_scan_steps(const float *g, int n, int ncoef, int cb, int ca, bool back)
{
    const int lw = wl_log2w(n), W = 1 << lw, rows = wl_rows(n), M = rows >> lw;
    if (wl_segments(n) > 1) return lw;
    float T[32][4];   // (y(-1), y(-2)) -> (y(M-1), y(M-2)): row 1, row 2
    for (int l = 0; l < W; ++l) {
        float p1 = 1.f, p2 = 0.f, q1 = 0.f, q2 = 1.f;
        for (int u = 0; u < M; ++u) {
            const int k = back ? rows - 1 - (l * M + u) : l * M + u;
            const float b = g[wl_table_at(n, ncoef, cb, k)], a = ca >= 0 ? g[wl_table_at(n, ncoef, ca, k)] : 0.f;
            const float p = -b * p1 - a * p2, q = -b * q1 - a * q2;
            p2 = p1;
            p1 = p;
            q2 = q1;
            q1 = q;
        }
        T[l][0] = p1;
        T[l][1] = q1;
        T[l][2] = p2;
        T[l][3] = q2;
    }
    for (int s = 0; s < lw; ++s) {
        float m = 0.f;
        for (int l = 1 << s; l < W; ++l) m = fmaxf(m, fmaxf(fabsf(T[l][0]) + fabsf(T[l][1]), fabsf(T[l][2]) + fabsf(T[l][3])));
        if (m < 9.313226e-10f) return s;
        for (int l = W - 1; l >= 1 << s; --l) {
            const float *A = T[l], *B = T[l - (1 << s)];
            const float r0 = A[0] * B[0] + A[1] * B[2], r1 = A[0] * B[1] + A[1] * B[3];
            const float r2 = A[2] * B[0] + A[3] * B[2], r3 = A[2] * B[1] + A[3] * B[3];
            T[l][0] = r0;
            T[l][1] = r1;
            T[l][2] = r2;
            T[l][3] = r3;
        }
    }
    return lw;
}

// The tables from factor_pdma's and factor_tdma's FP64 factors (the caller
// has zeroed them).
__device__ inline void pdma32_fold(const double *fac, int n, float *g)
{
    for (int k = 0; k < n; ++k) {
        const double c = k < n - 1 ? fac[k] : fac[5 * n];
        g[wl_table_at(n, 5, 0, k)] = (float)(1.0 / c);
        if (k >= 1) g[wl_table_at(n, 5, 1, k)] = (float)(fac[n + k - 1] / c);
        if (k >= 2) g[wl_table_at(n, 5, 2, k)] = (float)(fac[2 * n + k] / c);
        if (k < n - 1) g[wl_table_at(n, 5, 3, k)] = (float)fac[3 * n + k];
        if (k < n - 2) g[wl_table_at(n, 5, 4, k)] = (float)fac[4 * n + k];
    }
    g[0] = __int_as_float(max(wl_scan_steps(g, n, 5, 1, 2, false), wl_scan_steps(g, n, 5, 3, 4, true)));
}
__device__ inline void tdma32_fold(const double *fac, int n, float *g)
{
    for (int k = 0; k < n; ++k) {
        const double b = fac[n + k];
        if (k >= 1) g[wl_table_at(n, 3, 0, k)] = (float)fac[k];
        g[wl_table_at(n, 3, 1, k)] = (float)(1.0 / b);
        if (k < n - 1) g[wl_table_at(n, 3, 2, k)] = (float)(fac[2 * n + k] / b);
    }
    g[0] = __int_as_float(max(wl_scan_steps(g, n, 3, 0, -1, false), wl_scan_steps(g, n, 3, 2, -1, true)));
}

// Gives a set of nlines tables (len floats apart) the largest scan-step count
// among them: a warp's lines scan together, and the result must not depend on
// which lines share a warp.  One block.
__device__ inline void wl_common_steps(float *tab, size_t len, int nlines)
{
    __shared__ int most;
    if (threadIdx.x == 0) most = 0;
    __syncthreads();
    for (int q = threadIdx.x; q < nlines; q += blockDim.x) atomicMax(&most, __float_as_int(tab[q * len]));
    __syncthreads();
    for (int q = threadIdx.x; q < nlines; q += blockDim.x) tab[q * len] = __int_as_float(most);
    __syncthreads();
}

// Second-order recurrence y(u) = t(u) - b(u) y(u-1) - a(u) y(u-2) over the
// W = 2^lw lanes' W M rows, in place in t; (c1, c2) carries y(-1), y(-2) in
// and the last two rows out.  BACK runs it from the last row to the first.
// All 32 lanes of the warp take part, with the same `steps`.
template <int M, bool BACK>
__device__ __forceinline__ void wl_recur2(int lw, int steps, const float (&b)[M], const float (&a)[M], float (&t)[M], float &c1, float &c2)
{
    const unsigned full = 0xffffffffu;
    const int W = 1 << lw, lane = threadIdx.x & (W - 1);
    const int pos = BACK ? W - 1 - lane : lane;
    float w1 = 0.f, w2 = 0.f, p1 = 1.f, p2 = 0.f, q1 = 0.f, q2 = 1.f;
#pragma unroll
    for (int s = 0; s < M; ++s) {
        const int u = BACK ? M - 1 - s : s;
        const float w = __fmaf_rn(-b[u], w1, __fmaf_rn(-a[u], w2, t[u]));
        const float p = __fmaf_rn(-b[u], p1, -a[u] * p2);
        const float q = __fmaf_rn(-b[u], q1, -a[u] * q2);
        w2 = w1;
        w1 = w;
        p2 = p1;
        p1 = p;
        q2 = q1;
        q1 = q;
    }
#pragma unroll 1
    for (int d = 1; d < 1 << steps; d <<= 1) {
        const int src = BACK ? lane + d : lane - d;   // outside the group: discarded below
        const float v1 = __shfl_sync(full, w1, src, W), v2 = __shfl_sync(full, w2, src, W);
        const float g1 = __shfl_sync(full, p1, src, W), g2 = __shfl_sync(full, p2, src, W);
        const float h1 = __shfl_sync(full, q1, src, W), h2 = __shfl_sync(full, q2, src, W);
        if (pos >= d) {
            w1 = __fmaf_rn(p1, v1, __fmaf_rn(q1, v2, w1));
            w2 = __fmaf_rn(p2, v1, __fmaf_rn(q2, v2, w2));
            const float n1 = __fmaf_rn(p1, g1, q1 * g2), n2 = __fmaf_rn(p2, g1, q2 * g2);
            q1 = __fmaf_rn(p1, h1, q1 * h2);
            q2 = __fmaf_rn(p2, h1, q2 * h2);
            p1 = n1;
            p2 = n2;
        }
    }
    // states after each lane's rows, handed to the next lane
    const float s1 = __fmaf_rn(p1, c1, __fmaf_rn(q1, c2, w1));
    const float s2 = __fmaf_rn(p2, c1, __fmaf_rn(q2, c2, w2));
    const int prev = BACK ? lane + 1 : lane - 1;
    float y1 = __shfl_sync(full, s1, prev, W), y2 = __shfl_sync(full, s2, prev, W);
    if (pos == 0) {
        y1 = c1;
        y2 = c2;
    }
    c1 = __shfl_sync(full, s1, BACK ? 0 : W - 1, W);
    c2 = __shfl_sync(full, s2, BACK ? 0 : W - 1, W);
#pragma unroll
    for (int s = 0; s < M; ++s) {
        const int u = BACK ? M - 1 - s : s;
        const float y = __fmaf_rn(-b[u], y1, __fmaf_rn(-a[u], y2, t[u]));
        t[u] = y;
        y2 = y1;
        y1 = y;
    }
}

// First-order recurrence y(u) = t(u) - b(u) y(u-1), the same way.
template <int M, bool BACK>
__device__ __forceinline__ void wl_recur1(int lw, int steps, const float (&b)[M], float (&t)[M], float &c1)
{
    const unsigned full = 0xffffffffu;
    const int W = 1 << lw, lane = threadIdx.x & (W - 1);
    const int pos = BACK ? W - 1 - lane : lane;
    float w1 = 0.f, p1 = 1.f;
#pragma unroll
    for (int s = 0; s < M; ++s) {
        const int u = BACK ? M - 1 - s : s;
        w1 = __fmaf_rn(-b[u], w1, t[u]);
        p1 = -b[u] * p1;
    }
#pragma unroll 1
    for (int d = 1; d < 1 << steps; d <<= 1) {
        const int src = BACK ? lane + d : lane - d;
        const float v1 = __shfl_sync(full, w1, src, W), g1 = __shfl_sync(full, p1, src, W);
        if (pos >= d) {
            w1 = __fmaf_rn(p1, v1, w1);
            p1 = p1 * g1;
        }
    }
    const float s1 = __fmaf_rn(p1, c1, w1);
    float y1 = __shfl_sync(full, s1, BACK ? lane + 1 : lane - 1, W);
    if (pos == 0) y1 = c1;
    c1 = __shfl_sync(full, s1, BACK ? 0 : W - 1, W);
#pragma unroll
    for (int s = 0; s < M; ++s) {
        const int u = BACK ? M - 1 - s : s;
        y1 = __fmaf_rn(-b[u], y1, t[u]);
        t[u] = y1;
    }
}

// A line's table in registers: W lanes load their rows' coefficients.
template <int M, bool PENTA> struct WlTab {
    float b[M], a[PENTA ? M : 1], s[M], d[M], e[PENTA ? M : 1];
    int steps;   // the same for all lines of a set
    __device__ __forceinline__ void load(const float *line, int lw, size_t seg = 0)
    {
        steps = __float_as_int(line[0]);
        const float *T = line + 4 + seg * (size_t)((PENTA ? 5 : 3) * (M << lw)) + (threadIdx.x & ((1 << lw) - 1));
#pragma unroll
        for (int u = 0; u < M; ++u) {
            if (PENTA) {
                s[u] = T[u << lw];
                b[u] = T[(M + u) << lw];
                a[PENTA ? u : 0] = T[(2 * M + u) << lw];
                d[u] = T[(3 * M + u) << lw];
                e[PENTA ? u : 0] = T[(4 * M + u) << lw];
            } else {
                b[u] = T[u << lw];
                s[u] = T[(M + u) << lw];
                d[u] = T[(2 * M + u) << lw];
            }
        }
    }
    __device__ __forceinline__ void down(int lw, float (&t)[M], float &c1, float &c2) const
    {
        if constexpr (PENTA) {
#pragma unroll
            for (int u = 0; u < M; ++u) t[u] *= s[u];
            wl_recur2<M, false>(lw, steps, b, a, t, c1, c2);
        } else {
            wl_recur1<M, false>(lw, steps, b, t, c1);
        }
    }
    __device__ __forceinline__ void up(int lw, float (&t)[M], float &c1, float &c2) const
    {
        if constexpr (PENTA) {
            wl_recur2<M, true>(lw, steps, d, e, t, c1, c2);
        } else {
#pragma unroll
            for (int u = 0; u < M; ++u) t[u] *= s[u];
            wl_recur1<M, true>(lw, steps, d, t, c1);
        }
    }
    // a line of one segment
    __device__ __forceinline__ void solve(int lw, float (&t)[M]) const
    {
        float c1 = 0.f, c2 = 0.f;
        down(lw, t, c1, c2);
        c1 = c2 = 0.f;
        up(lw, t, c1, c2);
    }
};

// Lines t0, t0 + tstep, ... < nl of n rows, in place in shared memory: line t
// at x + t * xpitch (its slots) with its table at tab + t * tpitch (shared or
// global).  One warp; all its lanes call.
template <int M, bool PENTA>
__device__ __forceinline__ void wl_lines_m(const float *tab, size_t tpitch, int n, float *x, int xpitch, int nl, int warp, int nwarps)
{
    const int lw = wl_log2w(n), nseg = wl_segments(n), per = 32 >> lw;
    const int sub = (threadIdx.x & 31) >> lw, lane = threadIdx.x & ((1 << lw) - 1);
    for (int t0 = warp * per; t0 < nl; t0 += nwarps * per) {
        const bool live = t0 + sub < nl;
        const int t = live ? t0 + sub : t0;   // idle groups repeat line t0 and store nothing
        WlTab<M, PENTA> T;
        float c1 = 0.f, c2 = 0.f, r[M];
        for (int g = 0; g < nseg; ++g) {
            float *xs = x + (size_t)t * xpitch + ((g << lw) + lane) * (M + 1);
            T.load(tab + t * tpitch, lw, g);
#pragma unroll
            for (int u = 0; u < M; ++u) r[u] = xs[u];
            T.down(lw, r, c1, c2);
            if (g < nseg - 1) {
#pragma unroll
                for (int u = 0; u < M; ++u) xs[u] = r[u];
            }
        }
        c1 = c2 = 0.f;
        for (int g = nseg - 1; g >= 0; --g) {
            float *xs = x + (size_t)t * xpitch + ((g << lw) + lane) * (M + 1);
            if (g < nseg - 1) {
                T.load(tab + t * tpitch, lw, g);
#pragma unroll
                for (int u = 0; u < M; ++u) r[u] = xs[u];
            }
            T.up(lw, r, c1, c2);
            if (live) {
#pragma unroll
                for (int u = 0; u < M; ++u) xs[u] = r[u];
            }
        }
    }
}
template <bool PENTA>
__device__ __forceinline__ void wl_lines(const float *tab, size_t tpitch, int n, float *x, int xpitch, int nl)
{
    const int warp = threadIdx.x >> 5, nwarps = (int)blockDim.x >> 5;
    if (wl_log2m(n) == 3) wl_lines_m<8, PENTA>(tab, tpitch, n, x, xpitch, nl, warp, nwarps);
    else wl_lines_m<16, PENTA>(tab, tpitch, n, x, xpitch, nl, warp, nwarps);
}

// Asynchronous copy of n elements into shared memory by the block (16 bytes
// at a time where both ends and the length allow, else per element); the
// caller waits with async_copy_wait before the __syncthreads that publishes
// it.
template <class T> __device__ __forceinline__ void async_copy(T *dst, const T *src, int n, int tid, int nthr)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    const int per = 16 / (int)sizeof(T);
    if (((d | (unsigned)(size_t)src) & 15u) == 0 && n % per == 0) {
        for (int q = tid; q < n / per; q += nthr)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + 16u * q), "l"((const char *)src + 16 * (size_t)q) : "memory");
    } else {
        for (int q = tid; q < n; q += nthr)
            asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(d + (unsigned)sizeof(T) * q), "l"(src + q), "n"(sizeof(T))
                         : "memory");
    }
}
__device__ __forceinline__ void async_copy_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
