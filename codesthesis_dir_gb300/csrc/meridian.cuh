// Mixed-precision streamfunction solve in the (r, z) plane with the FP32
// correction cycles resident in a cluster's shared memory (meridian.cu).
#pragma once

#include "gbcommon.cuh"

#define MER_MAXLEV 8

struct __align__(16) MerW {
    double x, y, z, w;
};

// One level.  Off-diagonal weights of row i in r: c4i[i] = (i-1, i+1, far,
// diagonal), far being i + 2 for i <= n1/2 and i - 2 beyond it (the stretched
// grid's one-sided points; the uniform grid's far weight is zero), and of
// row j in z: c4j[j] the same with n2.
struct MerLevel {
    int n1, n2;
    const float4 *c4i, *c4j;        // i = 0..n1, j = 0..n2
    const float *fac_r, *fac_z;     // folded line tables (warpline.cuh) of line 1
    int fac_r_step, fac_z_step;     // floats from one line's table to the next (0: one table for all)
    // shared-memory plan of one CTA (floats): rows per CTA, row pitch, offsets
    int rp, pitch, v, f, o4i, o4j;
    int rows;                       // addresses of the rows of v, j = 0..n2
    int xline;                      // addresses of a colour's z-lines in their owners' line buffers
};

struct MerDev {
    int nlev, maxcycles, nrel;
    double tolcon;
    MerLevel lev[MER_MAXLEV];
    const MerW *d4i, *d4j;       // level 1's weights in FP64
    double *psi;                    // in, and out on convergence; pitch n1 + 1
    const double *rhs;
    double *v;                      // the FP64 iterate, pitch n1 + 1
    int *status;                    // [0] status, [1] correction cycles
    int *abort;                     // optional: the solve is skipped while it is set; set to 1 on a NaN
    int rc, x, stage, smem_floats;  // residual buffer, z-line buffer, neighbour rows, total
    int tab, tab_floats;            // the two stages of line tables, floats of one
    int penta;                      // pentadiagonal lines, four colours; else tridiagonal, two colours
};

// Lays out one CTA's shared memory for clusters of `ctas`; false when a level
// has lines longer than a warp holds (512 rows) or the arrays do not fit.
bool mer_plan(MerDev &d, int ctas);
// The weights of every level and of level 1 in FP64, in one allocation sized
// by mer_weight_bytes; the levels' n1, n2 must be set.
size_t mer_weight_bytes(const MerDev &d);
void mer_weight_layout(MerDev &d, void *mem);
// Clusters of this size that fit the device for d's plan (halved from want).
int mer_fit(MerDev &d, int want);
cudaError_t mer_launch(const MerDev &d, int ctas, cudaStream_t s);
// n solves in one launch: d_devs on the device, all planned for `ctas`.
cudaError_t mer_launch_many(const MerDev *d_devs, int n, int penta, int ctas, size_t smem, cudaStream_t s);
