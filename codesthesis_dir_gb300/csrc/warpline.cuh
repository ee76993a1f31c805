// FP32 line eliminations by the lanes of a warp (the correction cycles of the
// mixed-precision solves).
//
// One thread per line is a chain of 2 n dependent rows whose shared-memory
// loads it also has to issue alone: 90 cycles a row, 23 k cycles for the 255
// rows of a 257 x 257 grid's line.  Here W lanes share a line, lane l holding
// rows l M .. l M + M - 1 and their coefficients in registers.  Both halves of
// an elimination are recurrences, so every lane runs its rows from the state
// the lane before it last reached (zero at first) and the lanes repeat this
// until no lane's incoming state changes.  That is the serial elimination's
// result to the bit: lane l is final after pass l + 1 at the latest, and once
// no state changes another pass would change nothing.  It takes few passes
// because a row passes on only a part of its state (0.27 on a square mesh, so
// eight rows forget 15 bits and three passes reach FP32's rounding), up to W
// along strongly coupled lines.  A scan over the lanes' state maps takes about
// as long (two passes' arithmetic and 150 cycles a scan step) but rounds
// differently, and a solve stopped after one or two cycles keeps that: 5e-8
// of the streamfunction at a loose tolerance.
//
// M is 8 up to 256 rows (W = 4 .. 32, so a warp takes 32 / W lines) and 16 up
// to 512; W is a run-time value.  With M fitted to each level instead (one
// row per lane on the coarsest) every level ran code of its own, and the
// short phases waited for instructions: 2.0 k cycles for a 31-row line.
//
// The rows, rounded as written (no fused multiply-add), S and I being the
// pivots' reciprocals (taken in FP64, rounded once):
//   pentadiagonal  z(k) = ((r(k) - A(k) z(k-2)) - B(k) z(k-1)) S(k)
//                  x(k) = (z(k) - D(k) x(k+1)) - E(k) x(k+2)
//   tridiagonal    z(k) = r(k) - F(k) z(k-1),   x(k) = (z(k) - C(k) x(k+1)) I(k)
// Rows past the end have zero coefficients and leave the state at zero.
//
// FUSED tables have the pivots folded in (in FP64, rounded once), so that a row
// is one dependent fused multiply-add, a third of the rows above:
//   pentadiagonal  z(k) = S r(k) - (A S) z(k-2) - (B S) z(k-1)
//                  x(k) = z(k) - E x(k+2) - D x(k+1)
//   tridiagonal    z(k) = r(k) - F z(k-1),   x(k) = I z(k) - (C I) x(k+1)
// The 3D solves use them: their rings' eliminations round differently from a
// serial one in any case, and it takes 10 to 80 cycles to a solve, which leave
// 4e-10 of that.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

#define WL_MAXM 16

// log2 of the rows per lane and of the lanes per line; lines longer than
// 32 WL_MAXM rows take several segments of that many, one after the other.
__host__ __device__ __forceinline__ int wl_log2m(int n) { return n <= 256 ? 3 : 4; }
__host__ __device__ __forceinline__ int wl_log2w(int n) { return n <= 32 ? 2 : n <= 64 ? 3 : n <= 128 ? 4 : 5; }
// log2 of the lanes that hold a line's rows: the passes of a line go over no more
// (a line of up to 8 rows is one lane's and takes one pass).
__host__ __device__ __forceinline__ int wl_log2p(int n) { return n <= 8 ? 0 : n <= 16 ? 1 : wl_log2w(n); }
__host__ __device__ __forceinline__ int wl_segments(int n) { return n <= 256 ? 1 : (n + 511) / 512; }
// Padded rows of a line, the floats of its table (5 or 3 coefficients a row
// as [segment][coefficient][row in lane][lane]; a multiple of 16 bytes) and the
// pitch of its right-hand side in shared memory (a lane's rows padded to an
// odd stride, lines to an odd pitch: no bank conflicts in either direction).
__host__ __device__ __forceinline__ int wl_rows(int n) { return wl_segments(n) << (wl_log2m(n) + wl_log2w(n)); }
__host__ __device__ __forceinline__ size_t pdma32_len(int n) { return 5 * (size_t)wl_rows(n); }
__host__ __device__ __forceinline__ size_t tdma32_len(int n) { return 3 * (size_t)wl_rows(n); }
__host__ __device__ __forceinline__ int wl_slot(int lg, int q) { return q + (q >> lg); }
__host__ __device__ __forceinline__ int wl_pitch(int n) { return (wl_rows(n) + (wl_rows(n) >> wl_log2m(n))) | 1; }

__device__ __forceinline__ size_t wl_table_at(int n, int ncoef, int coef, int k)
{
    const int lg = wl_log2m(n), lw = wl_log2w(n);
    const int seg = k >> (lg + lw), q = k - (seg << (lg + lw));
    return ((((size_t)(seg * ncoef + coef) << lg) + (q & ((1 << lg) - 1))) << lw) + (q >> lg);
}

// The tables from factor_pdma's and factor_tdma's FP64 factors (the caller
// has zeroed them).
template <bool FUSED = false> __device__ inline void pdma32_fold(const double *fac, int n, float *g)
{
    for (int k = 0; k < n; ++k) {
        const double c = k < n - 1 ? fac[k] : fac[5 * n], q = FUSED ? c : 1.0;
        g[wl_table_at(n, 5, 0, k)] = (float)(1.0 / c);
        if (k >= 1) g[wl_table_at(n, 5, 1, k)] = (float)(fac[n + k - 1] / q);
        if (k >= 2) g[wl_table_at(n, 5, 2, k)] = (float)(fac[2 * n + k] / q);
        if (k < n - 1) g[wl_table_at(n, 5, 3, k)] = (float)fac[3 * n + k];
        if (k < n - 2) g[wl_table_at(n, 5, 4, k)] = (float)fac[4 * n + k];
    }
}
template <bool FUSED = false> __device__ inline void tdma32_fold(const double *fac, int n, float *g)
{
    for (int k = 0; k < n; ++k) {
        const double q = FUSED ? fac[n + k] : 1.0;
        if (k >= 1) g[wl_table_at(n, 3, 0, k)] = (float)fac[k];
        g[wl_table_at(n, 3, 1, k)] = (float)(1.0 / fac[n + k]);
        if (k < n - 1) g[wl_table_at(n, 3, 2, k)] = (float)(fac[2 * n + k] / q);
    }
}

// A recurrence of up to second order over the rows of W = 2^lw lanes, M each:
// y(u) = row(u, y(u-1), y(u-2)), into y; (c1, c2) carries the two states
// before the first row in and the last two out.  BACK runs it from the last
// row to the first.  All 32 lanes of the warp take part.
template <int M, bool BACK, bool SECOND, class Row>
__device__ __forceinline__ void wl_chain(int lw, float (&y)[M], float &c1, float &c2, const Row &row)
{
    const unsigned full = 0xffffffffu;
    const int W = 1 << lw, lane = threadIdx.x & (W - 1);
    const int pos = BACK ? W - 1 - lane : lane, prev = BACK ? lane + 1 : lane - 1;
    float in1 = pos == 0 ? c1 : 0.f, in2 = pos == 0 ? c2 : 0.f, s1, s2;
#pragma unroll 1
    for (int pass = 0;; ++pass) {
        s1 = in1;
        s2 = in2;
#pragma unroll
        for (int s = 0; s < M; ++s) {
            const int u = BACK ? M - 1 - s : s;
            y[u] = row(u, s1, s2);
            s2 = s1;
            s1 = y[u];
        }
        if (pass == W - 1) break;
        float n1 = __shfl_sync(full, s1, prev, W), n2 = SECOND ? __shfl_sync(full, s2, prev, W) : 0.f;
        if (pos == 0) {
            n1 = in1;
            n2 = in2;
        }
        const bool moved = __float_as_int(n1) != __float_as_int(in1) || (SECOND && __float_as_int(n2) != __float_as_int(in2));
        if (!__any_sync(full, moved)) break;
        in1 = n1;
        in2 = n2;
    }
    c1 = __shfl_sync(full, s1, BACK ? 0 : W - 1, W);
    if (SECOND) c2 = __shfl_sync(full, s2, BACK ? 0 : W - 1, W);
}

// A line's table in registers: W lanes load their rows' coefficients.
template <int M, bool PENTA, bool FUSED = false> struct WlTab {
    float b[M], a[PENTA ? M : 1], s[M], d[M], e[PENTA ? M : 1];
    __device__ __forceinline__ const float *rows(const float *line, int lw, size_t seg) const
    {
        return line + seg * (size_t)((PENTA ? 5 : 3) * (M << lw)) + (threadIdx.x & ((1 << lw) - 1));
    }
    __device__ __forceinline__ void load_down(const float *line, int lw, size_t seg)
    {
        const float *T = rows(line, lw, seg);
#pragma unroll
        for (int u = 0; u < M; ++u) {
            if (PENTA) {
                s[u] = T[u << lw];
                b[u] = T[(M + u) << lw];
                a[PENTA ? u : 0] = T[(2 * M + u) << lw];
            } else {
                b[u] = T[u << lw];
            }
        }
    }
    __device__ __forceinline__ void load_up(const float *line, int lw, size_t seg)
    {
        const float *T = rows(line, lw, seg);
#pragma unroll
        for (int u = 0; u < M; ++u) {
            if (PENTA) {
                d[u] = T[(3 * M + u) << lw];
                e[PENTA ? u : 0] = T[(4 * M + u) << lw];
            } else {
                s[u] = T[(M + u) << lw];
                d[u] = T[(2 * M + u) << lw];
            }
        }
    }
    __device__ __forceinline__ void load(const float *line, int lw)
    {
        load_down(line, lw, 0);
        load_up(line, lw, 0);
    }
    __device__ __forceinline__ void down(int lw, const float (&t)[M], float (&z)[M], float &c1, float &c2) const
    {
        if constexpr (PENTA && FUSED)
            wl_chain<M, false, true>(lw, z, c1, c2, [&](int u, float y1, float y2) {
                return __fmaf_rn(-b[u], y1, __fmaf_rn(-a[u], y2, t[u] * s[u]));
            });
        else if constexpr (PENTA)
            wl_chain<M, false, true>(lw, z, c1, c2, [&](int u, float y1, float y2) { return ((t[u] - a[u] * y2) - b[u] * y1) * s[u]; });
        else if constexpr (FUSED)
            wl_chain<M, false, false>(lw, z, c1, c2, [&](int u, float y1, float) { return __fmaf_rn(-b[u], y1, t[u]); });
        else
            wl_chain<M, false, false>(lw, z, c1, c2, [&](int u, float y1, float) { return t[u] - b[u] * y1; });
    }
    __device__ __forceinline__ void up(int lw, const float (&z)[M], float (&x)[M], float &c1, float &c2) const
    {
        if constexpr (PENTA && FUSED)
            wl_chain<M, true, true>(lw, x, c1, c2, [&](int u, float y1, float y2) { return __fmaf_rn(-d[u], y1, __fmaf_rn(-e[u], y2, z[u])); });
        else if constexpr (PENTA)
            wl_chain<M, true, true>(lw, x, c1, c2, [&](int u, float y1, float y2) { return (z[u] - d[u] * y1) - e[u] * y2; });
        else if constexpr (FUSED)
            wl_chain<M, true, false>(lw, x, c1, c2, [&](int u, float y1, float) { return __fmaf_rn(-d[u], y1, z[u] * s[u]); });
        else
            wl_chain<M, true, false>(lw, x, c1, c2, [&](int u, float y1, float) { return (z[u] - d[u] * y1) * s[u]; });
    }
    // a line of one segment and n rows, in place
    __device__ __forceinline__ void solve(int n, float (&t)[M]) const
    {
        const int lw = wl_log2p(n);
        float c1 = 0.f, c2 = 0.f, z[M];
        down(lw, t, z, c1, c2);
        c1 = c2 = 0.f;
        up(lw, z, t, c1, c2);
    }
};

// Lines t0, t0 + tstep, ... < nl of n rows, in place in shared memory: line t
// at x + t * xpitch (its slots) with its table at tab + t * tpitch (shared or
// global).  One warp; all its lanes call.
// BRIEF: passes over the lanes that hold rows only (wl_log2p), where the kernel has
// the registers for a second width (64 x 64 x 128 mixed, two steps: 217 -> 298 ms).
template <int M, bool PENTA, bool FUSED = false, bool BRIEF = false>
__device__ __forceinline__ void wl_lines_m(const float *tab, size_t tpitch, int n, float *x, int xpitch, int nl, int warp, int nwarps)
{
    const int lw = wl_log2w(n), lp = BRIEF ? wl_log2p(n) : lw, nseg = wl_segments(n), per = 32 >> lw;
    const int sub = (threadIdx.x & 31) >> lw, lane = threadIdx.x & ((1 << lw) - 1);
    for (int t0 = warp * per; t0 < nl; t0 += nwarps * per) {
        const bool live = t0 + sub < nl;
        const int t = live ? t0 + sub : t0;   // idle groups repeat line t0 and store nothing
        WlTab<M, PENTA, FUSED> T;
        float c1 = 0.f, c2 = 0.f, r[M], z[M];
        for (int g = 0; g < nseg; ++g) {
            float *xs = x + (size_t)t * xpitch + ((g << lw) + lane) * (M + 1);
            T.load_down(tab + t * tpitch, lw, g);
#pragma unroll
            for (int u = 0; u < M; ++u) r[u] = xs[u];
            T.down(lp, r, z, c1, c2);
            if (g < nseg - 1) {
#pragma unroll
                for (int u = 0; u < M; ++u) xs[u] = z[u];
            }
        }
        c1 = c2 = 0.f;
        for (int g = nseg - 1; g >= 0; --g) {
            float *xs = x + (size_t)t * xpitch + ((g << lw) + lane) * (M + 1);
            T.load_up(tab + t * tpitch, lw, g);
            if (g < nseg - 1) {
#pragma unroll
                for (int u = 0; u < M; ++u) z[u] = xs[u];
            }
            T.up(lp, z, r, c1, c2);
            if (live) {
#pragma unroll
                for (int u = 0; u < M; ++u) xs[u] = r[u];
            }
        }
    }
}
template <bool PENTA, bool FUSED = false, bool BRIEF = false>
__device__ __forceinline__ void wl_lines(const float *tab, size_t tpitch, int n, float *x, int xpitch, int nl)
{
    const int warp = threadIdx.x >> 5, nwarps = (int)blockDim.x >> 5;
    if (wl_log2m(n) == 3) wl_lines_m<8, PENTA, FUSED, BRIEF>(tab, tpitch, n, x, xpitch, nl, warp, nwarps);
    else wl_lines_m<16, PENTA, FUSED, BRIEF>(tab, tpitch, n, x, xpitch, nl, warp, nwarps);
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
