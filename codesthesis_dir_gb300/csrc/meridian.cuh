// Mixed-precision streamfunction solve in the (r, z) plane with the FP32
// correction cycles resident in a cluster's shared memory (meridian.cu).
#pragma once

#include "gbcommon.cuh"

#define MER_MAXLEV 8

// Level 1's operator in FP64, row i in r and row j in z: the same weights as
// MerLevel's, with the reciprocals of the divisors (the uniform grid uses r,
// rr and theirs only).
struct __align__(16) MerRow {
    double crr[4], cr[3], r, ir, rr, irr, pad;
};
struct __align__(16) MerCol {
    double czz[4];
};
// A divisor and its reciprocal.
struct MerOver {
    double h, ih;
};

// One level.  The FP32 cycles apply the operators term by term, in the order
// of the reference's statements.  Stretched grid (rcsc.f): row i's weights of
// d2/dr2 and of d/dr and 1/r, (crr1 .. crr4), (cr1, cr2, cr3, 1/r), and row j's
// of d2/dz2, (czz1 .. czz4); the points of row i are i-1 .. i+2 for i <= n1/2
// and i-2 .. i+1 beyond it, in z likewise.  Uniform grid (rotann2.f): row i's
// (r, r r, 1/r, 1/(r r)) and the spacings h with 1/h.
struct MerLevel {
    int n1, n2;
    const float4 *ci;               // i = 0..n1, two a row (stretched) or one
    const float4 *cj;               // j = 0..n2, stretched only
    float hr, hhr, hhz, drdz;       // uniform: 1/h's denominators, 2 (1/hhr + 1/hhz)
    float ihr, ihhr, ihhz;          // 1/h (IEEE)
    int quick;                      // every divisor lies in 2^-24 .. 2^24 (mer_quot)
    const float *fac_r, *fac_z;     // line tables (warpline.cuh) of line 1
    int fac_r_step, fac_z_step;     // floats from one line's table to the next (0: one table for all)
    // shared-memory plan of one CTA (floats): rows per CTA, row pitch, offsets
    int rp, pitch, v, f, oci, ocj;
    int rows;                       // addresses of the rows of v, j = 0..n2
    int xline;                      // addresses of a colour's z-lines in their owners' line buffers
};

struct MerDev {
    int nlev, maxcycles, nrel;
    double tolcon;
    MerLevel lev[MER_MAXLEV];
    const MerRow *d_i;              // level 1, i = 0..n1
    const MerCol *d_j;              // j = 0..n2
    MerOver hr, hhr, hhz;           // uniform grid
    double drdz;
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
// The weights of every level and level 1's in FP64, in one allocation sized
// by mer_weight_bytes; penta and the levels' n1, n2 must be set.
size_t mer_weight_bytes(const MerDev &d);
void mer_weight_layout(MerDev &d, void *mem);
// The largest cluster, up to `want`, that the device holds and d fits (0: none).
int mer_fit(MerDev &d, int want);
// CTAs of a solve of its own, planned for: `most`, or one for a small grid.
int mer_alone(MerDev &d, int most);
// One cluster size for n solves of a launch: the power of two `want` or, up to
// `most`, as many more CTAs as the largest needs.  Plans the solves for it;
// fits[q]: solve q does fit.  *smem: the most any of those takes.
int mer_plan_many(MerDev *d, int n, int want, int most, size_t *smem, char *fits);
[[nodiscard]] cudaError_t mer_launch(const MerDev &d, int ctas, cudaStream_t s);
// n solves in one launch: d_devs on the device, all planned for `ctas`.
[[nodiscard]] cudaError_t mer_launch_many(const MerDev *d_devs, int n, int penta, int ctas, size_t smem, cudaStream_t s);
