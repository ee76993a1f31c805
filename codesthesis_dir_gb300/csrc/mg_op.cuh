// Pointwise arithmetic of the velocity multigrid, shared by its two kernels
// (prb_mg.cu on global memory, prb_resident.cu in shared memory), which give
// the same bits.  Compiled with -fmad=false.
#pragma once

#include <cuda_runtime.h>

// The level operator applied at row i of a line (the part of relax2/relax3's
// residual before it is subtracted from f): PRB:2306-2357 (v), PRB:2553-2587
// (u), and the annulus forms of velvor2dnewsch3.4.f:2300-2346 and
// :2546-2579.  v(q) is the line's row q, va and vm the rows i of the lines
// after and before it.  Instantiated for double (bit-identical to the
// reference) and for float (the mixed-precision correction cycle).
template <class T, class At>
__device__ __forceinline__ T mg_apply_op(At v, T va, T vm, int i, int which, int polar, int n1, T hhri, T hhpi, T hri,
                                         const T *rvi, const T *rvq)
{
    const T two = T(2.0), c53 = T(5.0 / 3.0), c02 = T(0.2), c15 = T(1.5), c43 = T(4.0 / 3.0);
    const T v0 = v(i);
    T temp;
    if (polar && which == 2) {
        temp = (va - two * v0 + vm) * hhpi * rvq[i] + v0 * rvq[i];
        if (i == 1)
            temp = temp + (-two * v0 + c53 * v(i + 1) - c02 * v(i + 2)) * hhri + c43 * v(i + 1) * hri * rvi[i];
        else if (i == n1)
            temp = temp + (-two * v0 + c53 * v(i - 1) - c02 * v(i - 2)) * hhri - c43 * v(i - 1) * hri * rvi[i];
        else
            temp = temp + (v(i - 1) - two * v0 + v(i + 1)) * hhri + c15 * (v(i + 1) - v(i - 1)) * hri * rvi[i];
    } else if (polar) {
        temp = (v(i + 1) + v(i - 1)) * hhri + c15 * (v(i + 1) - v(i - 1)) * hri * rvi[i] + v0 * rvq[i] +
               (va + vm) * hhpi * rvq[i] - v0 * (two * hhri + two * hhpi * rvq[i]);
    } else if (which == 2) {
        temp = (va - two * v0 + vm) * hhpi;
        if (i == 1)
            temp = temp + (-two * v0 + c53 * v(i + 1) - c02 * v(i + 2)) * hhri;
        else if (i == n1)
            temp = temp + (-two * v0 + c53 * v(i - 1) - c02 * v(i - 2)) * hhri;
        else
            temp = temp + (v(i - 1) - two * v0 + v(i + 1)) * hhri;
    } else {
        temp = (v(i + 1) + v(i - 1)) * hhri + (va + vm) * hhpi - v0 * (two * hhri + two * hhpi);
    }
    return temp;
}

// corser's weighting (PRB:2603-2718) of a fine residual and its neighbours
// (i +- 1: ip, im; k +- 1: kp, km; corners ip/im x kp/km): the reference's sums in
// its order, or in FP32 1/4, 1/8 and 1/16.
__device__ __forceinline__ double mg_full_weight(double c0, double ip, double im, double kp, double km, double pp, double pm,
                                                 double mp, double mm)
{
    double t = c0;
    t = t + t;
    t = t + ip;
    t = t + im;
    t = t + c0;
    t = t + c0;
    t = t + kp;
    t = t + km;
    t = t + t;
    t = t + ip;
    t = t + ip;
    t = t + im;
    t = t + im;
    t = t + pp;
    t = t + pm;
    t = t + mp;
    t = t + mm;
    t = t + kp;
    t = t + km;
    t = t + kp;
    t = t + km;
    t = t + t;
    t = t + pp;
    t = t + pm;
    t = t + pp;
    t = t + pm;
    t = t + mp;
    t = t + mm;
    t = t + mp;
    t = t + mm;
    return t * 0.015625;
}
__device__ __forceinline__ float mg_full_weight(float c0, float ip, float im, float kp, float km, float pp, float pm, float mp,
                                                float mm)
{
    return 0.25f * c0 + 0.125f * (ip + im + kp + km) + 0.0625f * (pp + pm + mp + mm);
}

// finer's interpolation (PRB:2721-2803): coarse values at (i1, k1), (i1 + 1,
// k1), (i1, k1 + 1), (i1 + 1, k1 + 1); io, ko: fine index odd.
template <class T> __device__ __forceinline__ T mg_prolong(bool io, bool ko, T q00, T q10, T q01, T q11)
{
    if (!io) return !ko ? q00 : (q00 + q01) * T(0.5);
    if (!ko) return (q00 + q10) * T(0.5);
    return (q00 + q10 + q01 + q11) * T(0.25);
}
