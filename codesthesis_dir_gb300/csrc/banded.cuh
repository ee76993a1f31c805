// Banded line solvers on the device.
//
// The reference solves every line of a sweep with the same matrix
// (tdma/ptdma/pdma of velvor2dperiodicrbconv.f:3046-3164), redoing the
// elimination of the matrix for each line.  Here the matrix part of each
// elimination is done once (factor_* below, one thread, same operations in
// the same order) and every line then applies only the right-hand-side part.
// Both parts round exactly as the reference's interleaved loop does, so a
// line solved here is bit-identical to the reference algorithm on the same
// right-hand side (this file must be compiled with -fmad=false).  The
// factors also hold the reciprocals of the pivots (IEEE divisions done once),
// and every division of a line's elimination is the correctly rounded
// quotient formed from them (divrn.cuh), the same bits as the division.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

#include "divrn.cuh"

// Doubles of each factor layout.
__host__ __device__ inline size_t tdma_fac_len(int n) { return 4 * (size_t)n; }
__host__ __device__ inline size_t ptdma_fac_len(int n) { return 6 * (size_t)n + 3; }
__host__ __device__ inline size_t pdma_fac_len(int n) { return 6 * (size_t)n + 4; }

// ---------------------------------------------------------------------------
// Tridiagonal (tdma, velvor2dperiodicrbconv.f:3046-3064), n unknowns.
// Factor layout (4n doubles): fact[0..n), bp[0..n), c[0..n), 1/bp[0..n).
// ---------------------------------------------------------------------------
__device__ inline void factor_tdma(const double *a, const double *b, const double *c, int n,
                                   double *fac)
{
    double *fact = fac, *bp = fac + n, *cc = fac + 2 * n, *ibp = fac + 3 * n;
    bp[0] = b[0];
    fact[0] = 0.0;
    for (int j = 0; j < n; ++j) cc[j] = c[j];
    for (int j = 1; j < n; ++j) {
        fact[j] = a[j] / bp[j - 1];
        bp[j] = b[j] - fact[j] * c[j - 1];
    }
    for (int j = 0; j < n; ++j) ibp[j] = 1.0 / bp[j];
}

// ---------------------------------------------------------------------------
// Periodic tridiagonal (ptdma, velvor2dperiodicrbconv.f:3066-3116), n >= 4.
// Factor layout (6n + 3 doubles): f1[n), f2[n), a'[n), b'[n), c'[n), 1/b'[n),
// then fA, fB, fC.
// ---------------------------------------------------------------------------
__device__ inline void factor_ptdma(const double *a0, const double *b0, const double *c0, int n,
                                    double *fac)
{
    double *f1 = fac, *f2 = fac + n, *a = fac + 2 * n, *b = fac + 3 * n, *c = fac + 4 * n;
    const int N = n - 1;
    for (int j = 0; j < n; ++j) {
        a[j] = a0[j];
        b[j] = b0[j];
        c[j] = c0[j];
        f1[j] = 0.0;
        f2[j] = 0.0;
    }
    for (int j = 1; j <= n - 3; ++j) {
        double fact = a[j] / b[j - 1];
        f1[j] = fact;
        b[j] = b[j] - fact * c[j - 1];
        a[j] = -fact * a[j - 1];
        fact = c[N] / b[j - 1];
        f2[j] = fact;
        c[N] = -fact * c[j - 1];
        b[N] = b[N] - fact * a[j - 1];
    }
    double fA = a[n - 2] / b[n - 3];
    b[n - 2] = b[n - 2] - fA * c[n - 3];
    c[n - 2] = c[n - 2] - fA * a[n - 3];
    double fB = c[N] / b[n - 3];
    a[N] = a[N] - fB * c[n - 3];
    b[N] = b[N] - fB * a[n - 3];
    double fC = a[N] / b[n - 2];
    b[N] = b[N] - fC * c[n - 2];
    for (int j = 0; j < n; ++j) fac[5 * n + j] = 1.0 / b[j];
    fac[6 * n + 0] = fA;
    fac[6 * n + 1] = fB;
    fac[6 * n + 2] = fC;
}

__device__ inline void apply_ptdma(const double *fac, int n, double *x, int stride)
{
    const double *f1 = fac, *f2 = fac + n, *a = fac + 2 * n, *b = fac + 3 * n, *c = fac + 4 * n;
    const double *ib = fac + 5 * n;
    const double fA = fac[6 * n], fB = fac[6 * n + 1], fC = fac[6 * n + 2];
    const int N = n - 1;
    double rN = x[(size_t)N * stride];
    double prev = x[0];
    for (int j = 1; j <= n - 3; ++j) {
        double rj = x[(size_t)j * stride] - f1[j] * prev;
        rN = rN - f2[j] * prev;
        x[(size_t)j * stride] = rj;
        prev = rj;
    }
    // prev = r(n-3) final
    double rn2 = x[(size_t)(n - 2) * stride] - fA * prev;
    rN = rN - fB * prev;
    rN = rN - fC * rn2;
    double yN = div_by_rcp(rN, b[N], ib[N]);
    double y = div_by_rcp(rn2 - c[n - 2] * yN, b[n - 2], ib[n - 2]);
    x[(size_t)N * stride] = yN;
    x[(size_t)(n - 2) * stride] = y;
    for (int j = n - 3; j >= 0; --j) {
        y = div_by_rcp(x[(size_t)j * stride] - c[j] * y - a[j] * yN, b[j], ib[j]);
        x[(size_t)j * stride] = y;
    }
}

// ---------------------------------------------------------------------------
// Pentadiagonal (pdma, velvor2dperiodicrbconv.f:3118-3164), n >= 3.
// a: 2nd sub, b: sub, c: diag, d: super, e: 2nd super.
// Factor layout (6n + 4 doubles): cdiv[n), bk1[n), a[n), dn[n), en[n), cN,
// 1/cdiv[n), 1/cN, then as whole numbers the first k with a[k + 2] != 0 (n - 2
// if none) and the last j < n - 2 with en[j] != 0 (-1 if none).
// ---------------------------------------------------------------------------
__device__ inline void factor_pdma(const double *a0, const double *b0, const double *c0,
                                   const double *d0, const double *e0, int n, double *fac,
                                   double *work /* 2n doubles */)
{
    double *cdiv = fac, *bk1 = fac + n, *aa = fac + 2 * n, *d = fac + 3 * n, *e = fac + 4 * n;
    double *b = work, *c = work + n;
    for (int j = 0; j < n; ++j) {
        aa[j] = a0[j];
        b[j] = b0[j];
        c[j] = c0[j];
        d[j] = d0[j];
        e[j] = e0[j];
        cdiv[j] = 0.0;
        bk1[j] = 0.0;
    }
    for (int k = 0; k <= n - 2; ++k) {
        cdiv[k] = c[k];
        d[k] = d[k] / c[k];
        e[k] = e[k] / c[k];
        c[k] = 1.0;
        bk1[k] = b[k + 1];
        c[k + 1] = c[k + 1] - b[k + 1] * d[k];
        if (k != n - 2) d[k + 1] = d[k + 1] - b[k + 1] * e[k];
        b[k + 1] = 0.0;
        if (k != n - 2) {
            b[k + 2] = b[k + 2] - aa[k + 2] * d[k];
            c[k + 2] = c[k + 2] - aa[k + 2] * e[k];
        }
    }
    fac[5 * n] = c[n - 1];
    for (int k = 0; k <= n - 2; ++k) fac[5 * n + 1 + k] = 1.0 / cdiv[k];
    fac[6 * n + 1] = 1.0 / c[n - 1];
    int ka = n - 2, je = -1;
    for (int k = n - 3; k >= 0; --k)
        if (aa[k + 2] != 0.0) ka = k;
    for (int j = 0; j < n - 2; ++j)
        if (e[j] != 0.0) je = j;
    fac[6 * n + 2] = (double)ka;
    fac[6 * n + 3] = (double)je;
}

// Tridiagonal solve with a lazily produced right-hand side.
template <class Rhs>
__device__ inline void apply_tdma_rhs(const double *fac, int n, double *x, int stride, Rhs rhs)
{
    const double *fact = fac, *bp = fac + n, *c = fac + 2 * n, *ibp = fac + 3 * n;
    double prev = rhs(0);
    x[0] = prev;
#pragma unroll 4
    for (int j = 1; j < n; ++j) {
        double rj = rhs(j) - fact[j] * prev;
        x[(size_t)j * stride] = rj;
        prev = rj;
    }
    double y = div_by_rcp(prev, bp[n - 1], ibp[n - 1]);
    x[(size_t)(n - 1) * stride] = y;
#pragma unroll 4
    for (int j = n - 2; j >= 0; --j) {
        y = div_by_rcp(x[(size_t)j * stride] - c[j] * y, bp[j], ibp[j]);
        x[(size_t)j * stride] = y;
    }
}

template <class Rhs>
__device__ inline void apply_ptdma_rhs(const double *fac, int n, double *x, int stride, Rhs rhs)
{
    for (int j = 0; j < n; ++j) x[(size_t)j * stride] = rhs(j);
    apply_ptdma(fac, n, x, stride);
}

// ---------------------------------------------------------------------------
// Eliminations in place on a staged line, x[k * pitch] and the line's factors
// both in shared memory, one thread per line.  What bounds them is the FP64
// unit of an SM quarter: it takes one warp instruction every 64 cycles however
// many lanes are active and whether or not it depends on the last one
// (measured: 1, 2, 3, 4 independent chains 64.7, 128.5, 192.3, 256.3 cycles a
// step), so a row costs 64 cycles times its FP64 instructions.  Hence:
//   - products with a's and e's zeros are left out (only the walls' one-sided
//     rows, or half of a stretched line, have them; r - 0 q is r for every
//     finite q, the sign of a zero aside);
//   - quotients without the selection of div_by_rcp (the pivots of these
//     diagonally dominant lines are negative);
//   - factors and right-hand sides of the next rows are loaded into registers
//     while a row is eliminated (the compiler cannot move those loads above
//     the stores to x).
// A row of the layer's pentadiagonal lines: 902 cycles with all products and
// selections, 560 now (7 FP64 instructions).
// ---------------------------------------------------------------------------

// Rows k0 .. k1 - 1 of the pentadiagonal forward elimination; A: with the
// products by a.  (rk, rk1) are the current and the next row's right-hand
// sides.
template <int U, bool A>
__device__ __forceinline__ void pdma_down(const double *fac, int n, double *x, int pitch, int k0, int k1, double &rk, double &rk1)
{
    if (k0 >= k1) return;
    const double *cdiv = fac, *bk1 = fac + n, *aa = fac + 2 * n, *icdiv = fac + 5 * n + 1;
    double c[U], ic[U], b[U], a[U], r[U];
    auto fetch = [&](int k2) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int k = min(k2 + u, k1 - 1);
            c[u] = cdiv[k];
            ic[u] = icdiv[k];
            b[u] = bk1[k];
            if (A) a[u] = aa[k + 2];
            r[u] = x[(k + 2) * pitch];
        }
    };
    fetch(k0);
    for (int k = k0; k < k1; k += U) {
        double c0[U], ic0[U], b0[U], a0[U], r0[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            c0[u] = c[u];
            ic0[u] = ic[u];
            b0[u] = b[u];
            if (A) a0[u] = a[u];
            r0[u] = r[u];
        }
        if (k + U < k1) fetch(k + U);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (k + u < k1) {
                const double q = div_by_rcp_neg(rk, c0[u], ic0[u]);
                x[(k + u) * pitch] = q;
                rk = rk1 - b0[u] * q;
                rk1 = A ? r0[u] - a0[u] * q : r0[u];
            }
        }
    }
}
// Rows j0 down to j1 of the back substitution; E: with the products by e.
// (x0, x1) are the two rows above.
template <int U, bool E>
__device__ __forceinline__ void pdma_up(const double *fac, int n, double *x, int pitch, int j0, int j1, double &x0, double &x1)
{
    if (j0 < j1) return;
    const double *dn = fac + 3 * n, *en = fac + 4 * n;
    double d[U], e[U], r[U];
    auto fetch = [&](int j2) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int j = max(j2 - u, j1);
            d[u] = dn[j];
            if (E) e[u] = en[j];
            r[u] = x[j * pitch];
        }
    };
    fetch(j0);
    for (int j = j0; j >= j1; j -= U) {
        double d0[U], e0[U], r0[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            d0[u] = d[u];
            if (E) e0[u] = e[u];
            r0[u] = r[u];
        }
        if (j - U >= j1) fetch(j - U);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (j - u >= j1) {
                double xj = r0[u] - d0[u] * x0;
                if (E) xj = xj - e0[u] * x1;
                x[(j - u) * pitch] = xj;
                x1 = x0;
                x0 = xj;
            }
        }
    }
}
// Pentadiagonal, factor_pdma's layout: pdma's right-hand-side operations in its order.
template <int U = 2> __device__ __forceinline__ void pdma_staged(const double *fac, int n, double *x, int pitch)
{
    const int ka = (int)fac[6 * n + 2], je = (int)fac[6 * n + 3];
    double rk = x[0], rk1 = x[pitch];
    pdma_down<U, false>(fac, n, x, pitch, 0, ka, rk, rk1);
    pdma_down<U, true>(fac, n, x, pitch, ka, n - 2, rk, rk1);
    {   // row n - 2
        const double q = div_by_rcp_neg(rk, fac[n - 2], fac[5 * n + 1 + n - 2]);
        x[(n - 2) * pitch] = q;
        rk1 = rk1 - fac[n + n - 2] * q;
    }
    double x1 = div_by_rcp_neg(rk1, fac[5 * n], fac[6 * n + 1]);
    x[(n - 1) * pitch] = x1;
    double x0 = x[(n - 2) * pitch] - fac[3 * n + n - 2] * x1;
    x[(n - 2) * pitch] = x0;
    pdma_up<U, false>(fac, n, x, pitch, n - 3, je + 1, x0, x1);
    pdma_up<U, true>(fac, n, x, pitch, min(je, n - 3), 0, x0, x1);
}

// Tridiagonal, factor_tdma's layout: apply_tdma_rhs's operations in its order.
template <int U = 2> __device__ __forceinline__ void tdma_staged(const double *fac, int n, double *x, int pitch)
{
    const double *fact = fac, *bp = fac + n, *cc = fac + 2 * n, *ibp = fac + 3 * n;
    double prev = x[0];
    double f[U], r[U], b[U], ib[U];
    auto fetch = [&](int j0) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int j = min(j0 + u, n - 1);
            f[u] = fact[j];
            r[u] = x[j * pitch];
        }
    };
    fetch(1);
    for (int j0 = 1; j0 < n; j0 += U) {
        double f0[U], r0[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            f0[u] = f[u];
            r0[u] = r[u];
        }
        if (j0 + U < n) fetch(j0 + U);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (j0 + u < n) {
                prev = r0[u] - f0[u] * prev;
                x[(j0 + u) * pitch] = prev;
            }
        }
    }
    double y = div_by_rcp_neg(prev, bp[n - 1], ibp[n - 1]);
    x[(n - 1) * pitch] = y;
    auto fetch_back = [&](int j0) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int j = max(j0 - u, 0);
            f[u] = cc[j];
            b[u] = bp[j];
            ib[u] = ibp[j];
            r[u] = x[j * pitch];
        }
    };
    if (n >= 2) fetch_back(n - 2);
    for (int j0 = n - 2; j0 >= 0; j0 -= U) {
        double f0[U], b0[U], ib0[U], r0[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            f0[u] = f[u];
            b0[u] = b[u];
            ib0[u] = ib[u];
            r0[u] = r[u];
        }
        if (j0 - U >= 0) fetch_back(j0 - U);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (j0 - u >= 0) {
                y = div_by_rcp_neg(r0[u] - f0[u] * y, b0[u], ib0[u]);
                x[(j0 - u) * pitch] = y;
            }
        }
    }
}
