// 3D rotating annulus of rot3dmg.f on sm_103a: the Dufort-Frankel transport
// of the vorticity components A, B, C and the temperature, the wall
// vorticities, the right-hand sides of the three velocity Poisson equations,
// and their multigrid solves, FP64, bit-identical to the oracle (every
// expression in the reference's order, -fmad=false, IEEE division).
//
// Layout: every field is a (0:nr+1, 0:nz+1, 0:np) column-major array in HBM
// (i fastest), the reference's COMMON arrays cut to the run's size.  Each
// multigrid level holds its correction v, right-hand side f and residual
// res as (0:n1, 0:n2, 0:n3) arrays.
//
// Multigrid: one persistent cooperative launch per Poisson solve runs the
// whole sweep loop of poisson1/2/3.  A relaxation pass in one direction is
// a sequence of phases of independent lines separated by bounded grid
// barriers; each thread solves whole lines in place.  The line matrices
// depend only on the level and the line's radius, so the banded solvers'
// matrix eliminations are done once at creation (k_r3d_factors) and a line
// solve only carries its right-hand side through the recorded multipliers:
// the same operations, in the same order, as the reference's tdma, ptdma
// and pdma (rot3dmg.f:2570-2689).  Phases: GB_SMOOTHER_LEX runs the
// reference's sequential order as anti-diagonal wavefronts (a line reads
// the new values of the lines before it in the reference's order and the old
// values of those after it, and every such neighbour sits on an earlier or
// a later anti-diagonal), GB_SMOOTHER_ZEBRA the two-colour order with the
// one-sided boundary rows last.
#include "gbcommon.cuh"
#include "banded.cuh"
#include "cluster.cuh"
#include "convert.cuh"
#include "gridsync.cuh"
#include "r3d_stage.cuh"
#include "warpline.cuh"

#include <math.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <functional>
#include <vector>

#define R3_MAXLEV 8
#define R3_SYNC_STRIDE 32           // unsigneds between the components' barriers

// Work arrays of one level of one component's solve (the w and v solves
// of a step run concurrently, each on its own arrays).
struct R3Work {
    double *v, *f, *res;
    float *v32, *f32, *res32;
};

struct R3Lev {
    int n1, n2, n3, L1, L2;
    double hr, hz, hp, hhr, hhz, hhp;
    double ihr, ihhr, ihhz, ihhp;   // reciprocals (IEEE)
    double *rvc, *rvv;          // r0 + (i - 1/2) hr and i hr + r0, i = 0..n1+1
    double *dirc, *dirv, *diqc, *diqv;   // 1/r and 1/(r r) of both (IEEE)
    double *fac[4][3];          // [component][direction] factor tables
    int *lines[4][3];           // packed p | q << 16, phase by phase
    int *poff[4][3];            // phase offsets (nphase + 1)
    int nphase[4][3];
    // FP32 inner cycles (GB_PRB_MIXED)
    // weights of the FP32 operator, per component: of the rows i (i-1, i+1,
    // far, diagonal) and (phi neighbours), of the rows j (j-1, j+1, far, diagonal);
    // far is the one-sided rows' point two over
    float4 *wi[4], *wj[4];
    float *wp[4];
    float *fac32[4][3];         // fused line tables (warpline.cuh); phi-lines: R3Ring per radius
};

struct R3Dev {
    int nr, nz, np, ni, nj, nk, nlev;
    double dt, r0, rmax, zmax, Ra, Re, Gr, Ptl, dr, dz, dp;
    double nu_num, nu_den;      // -r0 ln(r0/rmax) and zmax 2 pi (host libm)
    double tolcon, sor;
    int nrel, maxsweeps;
    double *fld[GB_R_COUNT];
    R3Lev lev[R3_MAXLEV];
    R3Work work[4][R3_MAXLEV];  // [component 1..3][level]
    unsigned long long *resmax; // two slots per component, bit patterns of non-negative doubles
    int *nanflag;               // two slots per component
    int *abort;                 // nonzero: a solve failed, later kernels return
    int *steps_done;
    double *trans;              // per-k heat flux sums (np + 1)
    double *hist_nu;
    int *hist_sw;
    int *solve_status, *solve_sweeps;   // per component
    GridSync gs[4];             // per component (the w and v solves run concurrently)
    // rot3dmghor.f (GB_R3D_HORIZONTAL): gravity across the axis, both walls'
    // heat flux, the inner wall hot, plain V-cycles
    int horizontal;
    const double *sinth, *costh;        // libm sin, cos of 6.283185307/np k, k = 0..np
    double nu2_num;                     // nz/6 rmax ln(r0/rmax); nu_num is nz/6 r0 ln(r0/rmax) there
    double *trans2;                     // outer-wall per-k sums (np + 1)
    double *hist_nu2;
};

#define FX(a, i, j, k) ((a)[(size_t)(i) + (size_t)ni * ((size_t)(j) + (size_t)nj * (size_t)(k))])

// ---------------------------------------------------------------------------
// Transport (rot3dmg.f:341-873): one thread per point
// ---------------------------------------------------------------------------

__global__ void k_r3d_avort(R3Dev d)
{
    if (*(volatile int *)d.abort) return;
    const int nr = d.nr, nz = d.nz, np = d.np, ni = d.ni, nj = d.nj;
    const long long total = (long long)nr * (nz - 1) * (np + 1);
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= total) return;
    const int i = 1 + (int)(t % nr);
    const long long rest = t / nr;
    const int j = 1 + (int)(rest % (nz - 1));
    const int k = (int)(rest / (nz - 1));
    const double dr = d.dr, dz = d.dz, dp = d.dp, dt = d.dt, Ptl = d.Ptl;
    const double Ra = d.Ra, Re = d.Re, Gr = d.Gr;
    const double *A = d.fld[GB_R_A], *Ap = d.fld[GB_R_Ap], *B = d.fld[GB_R_B], *C = d.fld[GB_R_C];
    const double *th = d.fld[GB_R_th];
    const double *uel = d.fld[GB_R_uel], *vel = d.fld[GB_R_vel], *wel = d.fld[GB_R_wel];
    double *An = d.fld[GB_R_An];
    const int im = i - 1, jp = j + 1;
    const int km = k == 0 ? np - 1 : k - 1;
    const int ka = k == np ? 1 : k + 1;
    const double r = d.r0 + ((double)i - 0.5) * dr;
    const double u = (FX(uel, i, j, k) + FX(uel, i, jp, k) + FX(uel, i, j, ka) + FX(uel, i, jp, ka) +
                      FX(uel, im, j, k) + FX(uel, im, jp, k) + FX(uel, im, j, ka) + FX(uel, im, jp, ka)) *
                     0.125;
    const double v = (FX(vel, i, jp, k) + FX(vel, i, j, k)) * 0.5;
    const double w = (FX(wel, i, j, ka) + FX(wel, i, j, k)) * 0.5;
    const double tem = (FX(th, i, j, k) + FX(th, i, j, ka) + FX(th, i, jp, k) + FX(th, i, jp, ka)) * 0.25;
    const double BB = (FX(B, i, j, k) + FX(B, im, j, k) + FX(B, i, j, ka) + FX(B, im, j, ka)) * 0.25;
    const double CC = (FX(C, i, j, k) + FX(C, i, jp, k) + FX(C, im, j, k) + FX(C, im, jp, k)) * 0.25;
    double Arra, Ara, Ar, cnr;
    if (i == 1) {
        Arra = (3.2 * FX(A, i - 1, j, k) + 2.0 * FX(A, i + 1, j, k) - 0.2 * FX(A, i + 2, j, k)) / (dr * dr);
        Ara = (-4.0 * FX(A, i - 1, j, k) / 3.0 + FX(A, i + 1, j, k) / 3.0) / dr;
        Ar = (-4.0 * FX(A, i - 1, j, k) / 3.0 + FX(A, i, j, k) + FX(A, i + 1, j, k) / 3.0) / dr;
        cnr = -2.5 / (dr * dr) + 0.5 / dr / r;
    } else if (i == nr) {
        Arra = (3.2 * FX(A, i + 1, j, k) + 2.0 * FX(A, i - 1, j, k) - 0.2 * FX(A, i - 2, j, k)) / (dr * dr);
        Ara = (-FX(A, i - 1, j, k) / 3.0 + 4.0 * FX(A, i + 1, j, k) / 3.0) / dr;
        // the inner-wall formula again (rot3dmg.f:390)
        Ar = (-4.0 * FX(A, i - 1, j, k) / 3.0 + FX(A, i, j, k) + FX(A, i + 1, j, k) / 3.0) / dr;
        cnr = -2.5 / (dr * dr) - 0.5 / dr / r;
    } else {
        Arra = (FX(A, i - 1, j, k) + FX(A, i + 1, j, k)) / (dr * dr);
        Ara = (FX(A, i + 1, j, k) - FX(A, i - 1, j, k)) * 0.5 / dr;
        Ar = Ara;
        cnr = -1.0 / (dr * dr);
        const double Pe = fabs(u * dr / Ptl);
        if (Pe > 2.0) {
            if (u > 0.0) Ar = (FX(A, i, j, k) - FX(A, i - 1, j, k)) / dr;
            else if (u < 0.0) Ar = (FX(A, i + 1, j, k) - FX(A, i, j, k)) / dr;
        }
    }
    const double uelr = ((FX(uel, i, j, k) + FX(uel, i, jp, k) + FX(uel, i, j, ka) + FX(uel, i, jp, ka)) * 0.25 -
                         (FX(uel, im, j, k) + FX(uel, im, jp, k) + FX(uel, im, j, ka) + FX(uel, im, jp, ka)) * 0.25) /
                        dr;
    const double Azza = (FX(A, i, j - 1, k) + FX(A, i, j + 1, k)) / (dz * dz);
    double Az = (FX(A, i, j + 1, k) - FX(A, i, j - 1, k)) * 0.5 / dz;
    {
        const double Pe = fabs(w * dz / Ptl);
        if (Pe > 2.0) {
            if (w > 0.0) Az = (FX(A, i, j, k) - FX(A, i, j - 1, k)) / dz;
            else if (w < 0.0) Az = (FX(A, i, j + 1, k) - FX(A, i, j, k)) / dz;
        }
    }
    const double uelz = ((FX(uel, i, jp, k) + FX(uel, i, jp, ka) + FX(uel, im, jp, k) + FX(uel, im, jp, ka)) * 0.25 -
                         (FX(uel, i, j, k) + FX(uel, i, j, ka) + FX(uel, im, j, k) + FX(uel, im, j, ka)) * 0.25) /
                        dz;
    const double thz = (FX(th, i, jp, k) + FX(th, i, jp, ka) - FX(th, i, j, k) - FX(th, i, j, ka)) * 0.5 / dz;
    const double thh = (FX(th, i, j, ka) + FX(th, i, jp, ka) - FX(th, i, j, k) - FX(th, i, jp, k)) * 0.5 / dp;
    const double Ahha = (FX(A, i, j, ka) + FX(A, i, j, km)) / (dp * dp);
    double Ah = (FX(A, i, j, ka) - FX(A, i, j, km)) * 0.5 / dp;
    {
        const double Pe = fabs(v * dp * r / Ptl);
        if (Pe > 2.0) {
            if (v > 0.0) Ah = (FX(A, i, j, k) - FX(A, i, j, km)) / dp;
            else if (v < 0.0) Ah = (FX(A, i, j, ka) - FX(A, i, j, k)) / dp;
        }
    }
    const double Bh = (FX(B, i, j, ka) + FX(B, im, j, ka) - FX(B, i, j, k) - FX(B, im, j, k)) * 0.5 / dp;
    const double uelh = ((FX(uel, i, j, ka) + FX(uel, i, jp, ka) + FX(uel, im, j, ka) + FX(uel, im, jp, ka)) * 0.25 -
                         (FX(uel, i, j, k) + FX(uel, i, jp, k) + FX(uel, im, j, k) + FX(uel, im, jp, k)) * 0.25) /
                        dp;
    const double cnz = -1.0 / (dz * dz);
    const double cnh = -1.0 / (dp * dp) / (r * r);
    const double RHS1 = Arra + Ara / r + Ahha / (r * r) + Azza - 2.0 * Bh / (r * r) + FX(A, i, j, k) / (Ptl * dt);
    const double ULT = (u * Ar + v * Ah / r + w * Az - uelh * BB / r - uelz * CC) / Ptl;
    const double RHS2 = d.horizontal ? d.sinth[k] * Gr * Ptl * thz   // rot3dmghor.f:479
                                     : -2.0 * Re * uelz + 2.0 * Ra * (tem * uelz + thz * u) / Re / Ptl - Gr * Ptl / r * thh;
    const double cf1 = 1.0 / (Ptl * dt) - uelr / (2.0 * Ptl) + 1.0 / (2.0 * (r * r)) - cnr - cnz - cnh;
    const double cf2 = uelr / (2.0 * Ptl) - 1.0 / (2.0 * (r * r)) + cnr + cnz + cnh;
    FX(An, i, j, k) = (cf2 * FX(Ap, i, j, k) - ULT - RHS2 + RHS1) / cf1;
}

__global__ void k_r3d_bvort(R3Dev d)
{
    if (*(volatile int *)d.abort) return;
    const int nr = d.nr, nz = d.nz, np = d.np, ni = d.ni, nj = d.nj;
    const long long total = (long long)(nr - 1) * (nz - 1) * (np + 1);
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= total) return;
    const int i = 1 + (int)(t % (nr - 1));
    const long long rest = t / (nr - 1);
    const int j = 1 + (int)(rest % (nz - 1));
    const int k = (int)(rest / (nz - 1));
    const double dr = d.dr, dz = d.dz, dp = d.dp, dt = d.dt, Ptl = d.Ptl;
    const double Ra = d.Ra, Re = d.Re, Gr = d.Gr;
    const double *A = d.fld[GB_R_A], *B = d.fld[GB_R_B], *Bp = d.fld[GB_R_Bp], *C = d.fld[GB_R_C];
    const double *th = d.fld[GB_R_th];
    const double *uel = d.fld[GB_R_uel], *vel = d.fld[GB_R_vel], *wel = d.fld[GB_R_wel];
    double *Bn = d.fld[GB_R_Bn];
    const int ip = i + 1, jp = j + 1;
    const int km = k == 0 ? np - 1 : k - 1;
    const int ka = k == np ? 1 : k + 1;
    const double r = d.r0 + (double)i * dr;
    const double u = (FX(uel, i, j, k) + FX(uel, i, jp, k)) * 0.5;
    const double v = (FX(vel, i, j, km) + FX(vel, i, jp, km) + FX(vel, i, j, k) + FX(vel, i, jp, k) +
                      FX(vel, ip, j, km) + FX(vel, ip, jp, km) + FX(vel, ip, j, k) + FX(vel, ip, jp, k)) *
                     0.125;
    const double w = (FX(wel, i, j, k) + FX(wel, ip, j, k)) * 0.5;
    const double tem = (FX(th, i, jp, k) + FX(th, ip, jp, k) + FX(th, i, j, k) + FX(th, ip, j, k)) * 0.25;
    const double AA = (FX(A, i, j, k) + FX(A, ip, j, k) + FX(A, i, j, km) + FX(A, ip, j, km)) * 0.25;
    const double CC = (FX(C, i, j, k) + FX(C, i, jp, k) + FX(C, i, j, km) + FX(C, i, jp, km)) * 0.25;
    const double Brra = (FX(B, i - 1, j, k) + FX(B, i + 1, j, k)) / (dr * dr);
    const double Bra = (FX(B, i + 1, j, k) - FX(B, i - 1, j, k)) * 0.5 / dr;
    double Br = Bra;
    {
        const double Pe = fabs(u * dr / Ptl);
        if (Pe > 2.0) {
            if (u > 0.0) Br = (FX(B, i, j, k) - FX(B, i - 1, j, k)) / dr;
            else if (u < 0.0) Br = (FX(B, i + 1, j, k) - FX(B, i, j, k)) / dr;
        }
    }
    const double velr = ((FX(vel, ip, j, km) + FX(vel, ip, jp, km) + FX(vel, ip, j, k) + FX(vel, ip, jp, k)) * 0.25 -
                         (FX(vel, i, j, km) + FX(vel, i, jp, km) + FX(vel, i, j, k) + FX(vel, i, jp, k)) * 0.25) /
                        dr;
    const double Bzza = (FX(B, i, j - 1, k) + FX(B, i, j + 1, k)) / (dz * dz);
    double Bz = (FX(B, i, j + 1, k) - FX(B, i, j - 1, k)) * 0.5 / dz;
    {
        const double Pe = fabs(w * dz / Ptl);
        if (Pe > 2.0) {
            if (w > 0.0) Bz = (FX(B, i, j, k) - FX(B, i, j - 1, k)) / dz;
            else if (w < 0.0) Bz = (FX(B, i, j + 1, k) - FX(B, i, j, k)) / dz;
        }
    }
    const double velz = ((FX(vel, i, jp, km) + FX(vel, ip, jp, km) + FX(vel, i, jp, k) + FX(vel, ip, jp, k)) * 0.25 -
                         (FX(vel, i, j, km) + FX(vel, ip, j, km) + FX(vel, i, j, k) + FX(vel, ip, j, k)) * 0.25) /
                        dz;
    const double thz = (FX(th, i, jp, k) + FX(th, ip, jp, k) - FX(th, i, j, k) - FX(th, ip, j, k)) * 0.5 / dz;
    const double thr = (FX(th, ip, jp, k) + FX(th, ip, j, k) - FX(th, i, jp, k) - FX(th, i, j, k)) * 0.5 / dr;
    const double Bhha = (FX(B, i, j, ka) + FX(B, i, j, km)) / (dp * dp);
    double Bh = (FX(B, i, j, ka) - FX(B, i, j, km)) * 0.5 / dp;
    {
        const double Pe = fabs(v * dp * r / Ptl);
        if (Pe > 2.0) {
            if (v > 0.0) Bh = (FX(B, i, j, k) - FX(B, i, j, km)) / dp;
            else if (v < 0.0) Bh = (FX(B, i, j, ka) - FX(B, i, j, k)) / dp;
        }
    }
    const double Ah = (FX(A, i, j, k) + FX(A, ip, j, k) - FX(A, i, j, km) - FX(A, ip, j, km)) * 0.5 / dp;
    const double velh = ((FX(vel, i, j, k) + FX(vel, ip, j, k) + FX(vel, i, jp, k) + FX(vel, ip, jp, k)) * 0.25 -
                         (FX(vel, i, j, km) + FX(vel, ip, j, km) + FX(vel, i, jp, km) + FX(vel, ip, jp, km)) * 0.25) /
                        dp;
    const double cnr = -1.0 / (dr * dr);
    const double cnz = -1.0 / (dz * dz);
    const double cnh = -1.0 / (dp * dp) / (r * r);
    const double RHS1 = Brra + Bra / r + Bhha / (r * r) + Bzza + 2.0 * Ah / (r * r) + FX(B, i, j, k) / (Ptl * dt);
    const double ULT = (u * Br + v * Bh / r + w * Bz - (velr - v / r) * AA - velz * CC) / Ptl;
    const double RHS2 = d.horizontal ? d.costh[k] * Gr * Ptl * thz   // rot3dmghor.f:606
                                     : -2.0 * Re * velz + r * Ra * thz + 2.0 * Ra * (tem * velz + thz * v) / Re / Ptl +
                                           Gr * Ptl * thr;
    const double cf1 = 1.0 / (Ptl * dt) - (u / r + velh / r) / (2.0 * Ptl) + 1.0 / (2.0 * (r * r)) - cnr - cnz - cnh;
    const double cf2 = (u / r + velh / r) / (2.0 * Ptl) - 1.0 / (2.0 * (r * r)) + cnr + cnz + cnh;
    FX(Bn, i, j, k) = (cf2 * FX(Bp, i, j, k) - ULT - RHS2 + RHS1) / cf1;
}

__global__ void k_r3d_cvort(R3Dev d)
{
    if (*(volatile int *)d.abort) return;
    const int nr = d.nr, nz = d.nz, np = d.np, ni = d.ni, nj = d.nj;
    const long long total = (long long)(nr - 1) * nz * (np + 1);
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= total) return;
    const int i = 1 + (int)(t % (nr - 1));
    const long long rest = t / (nr - 1);
    const int j = 1 + (int)(rest % nz);
    const int k = (int)(rest / nz);
    const double dr = d.dr, dz = d.dz, dp = d.dp, dt = d.dt, Ptl = d.Ptl;
    const double Ra = d.Ra, Re = d.Re;
    const double *A = d.fld[GB_R_A], *B = d.fld[GB_R_B], *C = d.fld[GB_R_C], *Cp = d.fld[GB_R_Cp];
    const double *th = d.fld[GB_R_th];
    const double *uel = d.fld[GB_R_uel], *vel = d.fld[GB_R_vel], *wel = d.fld[GB_R_wel];
    double *Cn = d.fld[GB_R_Cn];
    const int ip = i + 1, jm = j - 1;
    const int km = k == 0 ? np - 1 : k - 1;
    const int ka = k == np ? 1 : k + 1;
    const double r = d.r0 + (double)i * dr;
    const double u = (FX(uel, i, j, ka) + FX(uel, i, j, k)) * 0.5;
    const double v = (FX(vel, i, j, k) + FX(vel, ip, j, k)) * 0.5;
    const double w = (FX(wel, i, j, k) + FX(wel, ip, j, k) + FX(wel, i, j, ka) + FX(wel, ip, j, ka) +
                      FX(wel, i, jm, k) + FX(wel, ip, jm, k) + FX(wel, i, jm, ka) + FX(wel, ip, jm, ka)) *
                     0.125;
    const double AA = (FX(A, i, j, k) + FX(A, i, jm, k) + FX(A, ip, j, k) + FX(A, ip, jm, k)) * 0.25;
    const double BB = (FX(B, i, j, k) + FX(B, i, jm, k) + FX(B, i, j, ka) + FX(B, i, jm, ka)) * 0.25;
    const double tem = (FX(th, i, j, k) + FX(th, ip, j, k) + FX(th, ip, j, ka) + FX(th, i, j, ka)) * 0.25;
    const double Crra = (FX(C, i - 1, j, k) + FX(C, i + 1, j, k)) / (dr * dr);
    const double Cra = (FX(C, i + 1, j, k) - FX(C, i - 1, j, k)) * 0.5 / dr;
    double Cr = Cra;
    {
        const double Pe = fabs(u * dr / Ptl);
        if (Pe > 2.0) {
            if (u > 0.0) Cr = (FX(C, i, j, k) - FX(C, i - 1, j, k)) / dr;
            else if (u < 0.0) Cr = (FX(C, i + 1, j, k) - FX(C, i, j, k)) / dr;
        }
    }
    const double welr = ((FX(wel, ip, j, k) + FX(wel, ip, j, ka) + FX(wel, ip, jm, k) + FX(wel, ip, jm, ka)) * 0.25 -
                         (FX(wel, i, j, k) + FX(wel, i, j, ka) + FX(wel, i, jm, k) + FX(wel, i, jm, ka)) * 0.25) /
                        dr;
    const double thr = (FX(th, ip, j, k) + FX(th, ip, j, ka) - FX(th, i, j, k) - FX(th, i, j, ka)) * 0.5 / dr;
    double Czza, Cz, cnz;
    if (j == 1) {
        Czza = (3.2 * FX(C, i, j - 1, k) + 2.0 * FX(C, i, j + 1, k) - 0.2 * FX(C, i, j + 2, k)) / (dz * dz);
        Cz = (-4.0 * FX(C, i, j - 1, k) / 3.0 + FX(C, i, j, k) + FX(C, i, j + 1, k) / 3.0) / dz;
        cnz = -2.5 / (dz * dz);
    } else if (j == nz) {
        Czza = (3.2 * FX(C, i, j + 1, k) + 2.0 * FX(C, i, j - 1, k) - 0.2 * FX(C, i, j - 2, k)) / (dz * dz);
        Cz = (-FX(C, i, j - 1, k) / 3.0 - FX(C, i, j, k) + 4.0 * FX(C, i, j + 1, k) / 3.0) / dz;
        cnz = -2.5 / (dz * dz);
    } else {
        Czza = (FX(C, i, j - 1, k) + FX(C, i, j + 1, k)) / (dz * dz);
        Cz = (FX(C, i, j + 1, k) - FX(C, i, j - 1, k)) * 0.5 / dz;
        const double Pe = fabs(w * dz / Ptl);
        if (Pe > 2.0) {
            if (w > 0.0) Cz = (FX(C, i, j, k) - FX(C, i, j - 1, k)) / dz;
            else if (w < 0.0) Cz = (FX(C, i, j + 1, k) - FX(C, i, j, k)) / dz;
        }
        cnz = -1.0 / (dz * dz);
    }
    const double welz = ((FX(wel, i, j, k) + FX(wel, ip, j, k) + FX(wel, i, j, ka) + FX(wel, ip, j, ka)) * 0.25 -
                         (FX(wel, i, jm, k) + FX(wel, ip, jm, k) + FX(wel, i, jm, ka) + FX(wel, ip, jm, ka)) * 0.25) /
                        dz;
    const double Chha = (FX(C, i, j, ka) + FX(C, i, j, km)) / (dp * dp);
    double Ch = (FX(C, i, j, ka) - FX(C, i, j, km)) * 0.5 / dp;
    {
        const double Pe = fabs(v * dp * r / Ptl);
        if (Pe > 2.0) {
            if (v > 0.0) Ch = (FX(C, i, j, k) - FX(C, i, j, km)) / dp;
            else if (v < 0.0) Ch = (FX(C, i, j, ka) - FX(C, i, j, k)) / dp;
        }
    }
    const double welh = ((FX(wel, i, j, ka) + FX(wel, ip, j, ka) + FX(wel, i, jm, ka) + FX(wel, ip, jm, ka)) * 0.25 -
                         (FX(wel, i, j, k) + FX(wel, ip, j, k) + FX(wel, i, jm, k) + FX(wel, ip, jm, k)) * 0.25) /
                        dp;
    const double thh = (FX(th, i, j, ka) + FX(th, ip, j, ka) - FX(th, i, j, k) - FX(th, ip, j, k)) * 0.5 / dp;
    const double cnr = -1.0 / (dr * dr);
    const double cnh = -1.0 / (dp * dp) / (r * r);
    const double RHS1 = Crra + Cra / r + Chha / (r * r) + Czza + FX(C, i, j, k) / (Ptl * dt);
    const double ULT = (u * Cr + v * Ch / r + w * Cz - welr * AA - welh * BB / r) / Ptl;
    const double RHS2 =
        d.horizontal ? -(1.0 / r * d.Gr * Ptl * d.costh[k] * thh) - d.Gr * Ptl * d.sinth[k] * thr   // rot3dmghor.f:749
                     : -2.0 * Re * welz - Ra * thh + 2.0 * Ra * (tem * welz - thr * u - thh * v / r) / Re / Ptl;
    const double cf1 = 1.0 / (Ptl * dt) - welz / (2.0 * Ptl) - cnr - cnz - cnh;
    const double cf2 = welz / (2.0 * Ptl) + cnr + cnz + cnh;
    FX(Cn, i, j, k) = (cf2 * FX(Cp, i, j, k) - ULT - RHS2 + RHS1) / cf1;
}

__global__ void k_r3d_temp(R3Dev d)
{
    if (*(volatile int *)d.abort) return;
    const int nr = d.nr, nz = d.nz, np = d.np, ni = d.ni, nj = d.nj;
    const long long total = (long long)nr * (nz + 2) * (np + 1);
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= total) return;
    const int i = 1 + (int)(t % nr);
    const long long rest = t / nr;
    const int j = (int)(rest % (nz + 2));
    const int k = (int)(rest / (nz + 2));
    const double dr = d.dr, dz = d.dz, dp = d.dp, dt = d.dt, Ptl = d.Ptl;
    const double *th = d.fld[GB_R_th], *thp = d.fld[GB_R_thp];
    const double *uel = d.fld[GB_R_uel], *vel = d.fld[GB_R_vel], *wel = d.fld[GB_R_wel];
    double *thn = d.fld[GB_R_thn];
    const int im = i - 1, jm = j - 1;
    const int km = k == 0 ? np - 1 : k - 1;
    const int ka = k == np ? 1 : k + 1;
    const double r = d.r0 + ((double)i - 0.5) * dr;
    double u, v, w;
    if (j == 0 || j == nz + 1) {
        u = 0.0;
        v = 0.0;
        w = 0.0;
    } else {
        u = (FX(uel, i, j, k) + FX(uel, im, j, k)) * 0.5;
        v = (FX(vel, i, j, k) + FX(vel, i, j, km)) * 0.5;
        w = (FX(wel, i, j, k) + FX(wel, i, jm, k)) * 0.5;
    }
    double thrra, thra, thr, cnr;
    if (i == 1) {
        thrra = (3.2 * FX(th, i - 1, j, k) + 2.0 * FX(th, i + 1, j, k) - 0.2 * FX(th, i + 2, j, k)) / (dr * dr);
        thra = (-4.0 * FX(th, i - 1, j, k) / 3.0 + FX(th, i + 1, j, k) / 3.0) / dr;
        thr = (-4.0 * FX(th, i - 1, j, k) / 3.0 + FX(th, i, j, k) + FX(th, i + 1, j, k) / 3.0) / dr;
        cnr = -2.5 / (dr * dr) + 0.5 / dr / r;
    } else if (i == nr) {
        thrra = (3.2 * FX(th, i + 1, j, k) + 2.0 * FX(th, i - 1, j, k) - 0.2 * FX(th, i - 2, j, k)) / (dr * dr);
        thra = (-FX(th, i - 1, j, k) / 3.0 + 4.0 * FX(th, i + 1, j, k) / 3.0) / dr;
        thr = (-FX(th, i - 1, j, k) / 3.0 - FX(th, i, j, k) + 4.0 * FX(th, i + 1, j, k) / 3.0) / dr;
        cnr = -2.5 / (dr * dr) - 0.5 / dr / r;
    } else {
        thrra = (FX(th, i - 1, j, k) + FX(th, i + 1, j, k)) / (dr * dr);
        thra = (FX(th, i + 1, j, k) - FX(th, i - 1, j, k)) * 0.5 / dr;
        thr = thra;
        const double Pe = fabs(u * dr / Ptl);
        if (Pe > 2.0) {
            if (u > 0.0) thr = (FX(th, i, j, k) - FX(th, i - 1, j, k)) / dr;
            else if (u < 0.0) thr = (FX(th, i + 1, j, k) - FX(th, i, j, k)) / dr;
        }
        cnr = -1.0 / (dr * dr);
    }
    double thzza, thz, cnz;
    if (j == 1) {
        thzza = (3.2 * FX(th, i, j - 1, k) + 2.0 * FX(th, i, j + 1, k) - 0.2 * FX(th, i, j + 2, k)) / (dz * dz);
        thz = (-4.0 * FX(th, i, j - 1, k) / 3.0 + FX(th, i, j, k) + FX(th, i, j + 1, k) / 3.0) / dz;
        cnz = -2.5 / (dz * dz);
    } else if (j == nz) {
        thzza = (3.2 * FX(th, i, j + 1, k) + 2.0 * FX(th, i, j - 1, k) - 0.2 * FX(th, i, j - 2, k)) / (dz * dz);
        thz = (-FX(th, i, j - 1, k) / 3.0 - FX(th, i, j, k) + 4.0 * FX(th, i, j + 1, k) / 3.0) / dz;
        cnz = -2.5 / (dz * dz);
    } else if (j == 0) {
        thzza = 8.0 * FX(th, i, j + 1, k) / (dz * dz);
        thz = 0.0;
        cnz = -4.0 / (dz * dz);
    } else if (j == nz + 1) {
        thzza = 8.0 * FX(th, i, j - 1, k) / (dz * dz);
        thz = 0.0;
        cnz = -4.0 / (dz * dz);
    } else {
        thzza = (FX(th, i, j - 1, k) + FX(th, i, j + 1, k)) / (dz * dz);
        thz = (FX(th, i, j + 1, k) - FX(th, i, j - 1, k)) * 0.5 / dz;
        const double Pe = fabs(w * dz / Ptl);
        if (Pe > 2.0) {
            if (w > 0.0) thz = (FX(th, i, j, k) - FX(th, i, j - 1, k)) / dz;
            else if (w < 0.0) thz = (FX(th, i, j + 1, k) - FX(th, i, j, k)) / dz;
        }
        cnz = -1.0 / (dz * dz);
    }
    const double thhha = (FX(th, i, j, ka) + FX(th, i, j, km)) / (dp * dp);
    double thh = (FX(th, i, j, ka) - FX(th, i, j, km)) * 0.5 / dp;
    {
        const double Pe = fabs(v * dp * r / Ptl);
        if (Pe > 2.0) {
            if (v > 0.0) thh = (FX(th, i, j, k) - FX(th, i, j, km)) / dp;
            else if (v < 0.0) thh = (FX(th, i, j, ka) - FX(th, i, j, k)) / dp;
        }
    }
    const double cnp = -1.0 / (dp * dp) / (r * r);
    const double RHS1 = thrra + thra / r + thhha / (r * r) + thzza + FX(th, i, j, k) / dt;
    const double ULT = u * thr + v * thh / r + w * thz;
    const double cf1 = 1.0 / dt - cnr - cnz - cnp;
    const double cf2 = cnr + cnz + cnp;
    FX(thn, i, j, k) = (cf2 * FX(thp, i, j, k) - ULT + RHS1) / cf1;
}

// heat (rot3dmg.f:882-909): one thread per k sums its z column in the
// reference's order; k_r3d_heat_sum adds the columns k = 1..np in order.
__global__ void k_r3d_heat_k(R3Dev d)
{
    if (*(volatile int *)d.abort) return;
    const int k = 1 + blockIdx.x * blockDim.x + threadIdx.x;
    if (k > d.np) return;
    const int ni = d.ni, nj = d.nj, nz = d.nz;
    const double dr = d.dr, dz = d.dz;
    const double *th = d.fld[GB_R_th];
#define HT(j, k) ((-184.0 * FX(th, 0, j, k) + 225.0 * FX(th, 1, j, k) - 50.0 * FX(th, 2, j, k) + 9.0 * FX(th, 3, j, k)))
    if (d.horizontal) {
        // rot3dmghor.f:913-945: both cylinders over j = nz/2-3 .. nz/2+3
        const int nr = d.nr, nza = nz / 2 - 3, nzb = nz / 2 + 3;
#define HB(j, k) ((184.0 * FX(th, nr + 1, j, k) - 225.0 * FX(th, nr, j, k) + 50.0 * FX(th, nr - 1, j, k) - \
                   9.0 * FX(th, nr - 2, j, k)))
        double ta = dz * HT(nza, k) / (120.0 * dr);
        double tb = dz * HB(nza, k) / (120.0 * dr);
        ta = ta + dz * HT(nzb, k) / (120.0 * dr);
        tb = tb + dz * HB(nzb, k) / (120.0 * dr);
        for (int j = nza + 1; j <= nzb - 1; ++j) {
            ta = ta + dz * HT(j, k) / (60.0 * dr);
            tb = tb + dz * HB(j, k) / (60.0 * dr);
        }
#undef HB
        d.trans[k] = ta;
        d.trans2[k] = tb;
        return;
    }
    double trans = dz * HT(0, k) / (240.0 * dr);
    trans = trans + dz * HT(1, k) / (80.0 * dr);
    trans = trans + dz * HT(nz, k) / (80.0 * dr);
    trans = trans + dz * HT(nz + 1, k) / (240.0 * dr);
    for (int j = 2; j <= nz - 1; ++j) trans = trans + dz * HT(j, k) / (60.0 * dr);
#undef HT
    d.trans[k] = trans;
}

__global__ void k_r3d_heat_sum(R3Dev d, int step)
{
    if (*(volatile int *)d.abort) return;
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    double trans1 = 0.0, trans2 = 0.0;
    for (int k = 1; k <= d.np; ++k) trans1 = trans1 + d.trans[k] * d.dp;
    if (d.horizontal)
        for (int k = 1; k <= d.np; ++k) trans2 = trans2 + d.trans2[k] * d.dp;
    d.trans[0] = trans1;
    d.trans2[0] = trans2;
    if (step >= 0) {
        d.hist_nu[step] = d.nu_num * trans1 / d.nu_den;
        d.hist_nu2[step] = d.horizontal ? d.nu2_num * trans2 / d.nu_den : 0.0;
    }
}

// rhsw / rhsv / rhsu (rot3dmg.f:1026-1150)
template <int COMP>
__global__ void k_r3d_rhs(R3Dev d)
{
    if (*(volatile int *)d.abort) return;
    const int nr = d.nr, nz = d.nz, np = d.np, ni = d.ni, nj = d.nj;
    const int I = COMP == 3 ? nr - 1 : nr, J = COMP == 1 ? nz - 1 : nz;
    const long long total = (long long)I * J * (np + 1);
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= total) return;
    const int i = 1 + (int)(t % I);
    const long long rest = t / I;
    const int j = 1 + (int)(rest % J);
    const int k = (int)(rest / J);
    const double dr = d.dr, dz = d.dz, dp = d.dp;
    const double *An = d.fld[GB_R_An], *Bn = d.fld[GB_R_Bn], *Cn = d.fld[GB_R_Cn], *wel = d.fld[GB_R_wel];
    const int km = k == 0 ? np - 1 : k - 1;
    if (COMP == 1) {
        const double r = d.r0 + ((double)i - 0.5) * dr;
        const double Ah = (FX(An, i, j, k) - FX(An, i, j, km)) / dp;
        double w;
        if (i == 1) w = Ah / r - FX(Bn, 1, j, k) / dr - 0.5 * FX(Bn, 1, j, k) / r;
        else if (i == nr) w = Ah / r + FX(Bn, nr - 1, j, k) / dr - 0.5 * FX(Bn, nr - 1, j, k) / r;
        else {
            const double Br = (FX(Bn, i, j, k) - FX(Bn, i - 1, j, k)) / dr;
            w = Ah / r - Br - 0.5 * (FX(Bn, i, j, k) + FX(Bn, i - 1, j, k)) / r;
        }
        FX(d.fld[GB_R_wrh], i, j, k) = w;
    } else if (COMP == 2) {
        const double r = d.r0 + ((double)i - 0.5) * dr;
        double v;
        if (i == 1) v = FX(Cn, 1, j, k) / dr + FX(Cn, 1, j, k) / r;
        else if (i == nr) v = -FX(Cn, nr - 1, j, k) / dr + FX(Cn, nr - 1, j, k) / r;
        else {
            const double Cr = (FX(Cn, i, j, k) - FX(Cn, i - 1, j, k)) / dr;
            v = Cr + (FX(Cn, i, j, k) + FX(Cn, i - 1, j, k)) / r;
        }
        if (j == 1) v = v - FX(An, i, 1, k) / dz;
        else if (j == nz) v = v + FX(An, i, nz - 1, k) / dz;
        else {
            const double Az = (FX(An, i, j, k) - FX(An, i, j - 1, k)) / dz;
            v = v - Az;
        }
        FX(d.fld[GB_R_vrh], i, j, k) = v;
    } else {
        const double r = d.r0 + (double)i * dr;
        const double welz =
            0.5 * (FX(wel, i, j, k) + FX(wel, i + 1, j, k) - FX(wel, i, j - 1, k) - FX(wel, i + 1, j - 1, k)) / dz;
        const double Ch = (FX(Cn, i, j, k) - FX(Cn, i, j, km)) / dp;
        double u;
        if (j == 1) u = FX(Bn, i, 1, k) / dz - Ch / r - 2.0 * welz / r;
        else if (j == nz) u = -FX(Bn, i, nz - 1, k) / dz - Ch / r - 2.0 * welz / r;
        else {
            const double Bz = (FX(Bn, i, j, k) - FX(Bn, i, j - 1, k)) / dz;
            u = Bz - Ch / r - 2.0 * welz / r;
        }
        FX(d.fld[GB_R_urh], i, j, k) = u;
    }
}

// update (rot3dmg.f:964-1023): each thread sets the wall values of its own
// point (they depend on the velocities only) and moves its time levels.
__global__ void k_r3d_update(R3Dev d, int step)
{
    if (*(volatile int *)d.abort) return;
    const int nr = d.nr, nz = d.nz, ni = d.ni, nj = d.nj;
    const long long total = (long long)ni * nj * d.nk;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t == 0 && step >= 0) atomicAdd(d.steps_done, 1);
    if (t >= total) return;
    const int i = (int)(t % ni);
    const long long rest = t / ni;
    const int j = (int)(rest % nj);
    const int k = (int)(rest / nj);
    const double dr = d.dr, dz = d.dz;
    const double *uel = d.fld[GB_R_uel], *vel = d.fld[GB_R_vel], *wel = d.fld[GB_R_wel];
    double *An = d.fld[GB_R_An], *Bn = d.fld[GB_R_Bn], *Cn = d.fld[GB_R_Cn], *thn = d.fld[GB_R_thn];
    if (i >= 1 && i <= nr) {
        if (j == 0) FX(An, i, 0, k) = -(3.0 * FX(vel, i, 1, k) - FX(vel, i, 2, k) / 3.0) / dz;
        else if (j == nz) FX(An, i, nz, k) = -(FX(vel, i, nz - 1, k) / 3.0 - 3.0 * FX(vel, i, nz, k)) / dz;
    }
    if (i >= 1 && i <= nr - 1) {
        if (j == 0) FX(Bn, i, 0, k) = (3.0 * FX(uel, i, 1, k) - FX(uel, i, 2, k) / 3.0) / dz;
        else if (j == nz) FX(Bn, i, nz, k) = (-3.0 * FX(uel, i, nz, k) + FX(uel, i, nz - 1, k) / 3.0) / dz;
    }
    if (j >= 1 && j <= nz - 1) {
        if (i == 0) FX(Bn, 0, j, k) = -(3.0 * FX(wel, 1, j, k) - FX(wel, 2, j, k) / 3.0) / dr;
        else if (i == nr) FX(Bn, nr, j, k) = -(FX(wel, nr - 1, j, k) / 3.0 - 3.0 * FX(wel, nr, j, k)) / dr;
    }
    if (j >= 1 && j <= nz) {
        if (i == 0) FX(Cn, 0, j, k) = (3.0 * FX(vel, 1, j, k) - FX(vel, 2, j, k) / 3.0) / dr;
        else if (i == nr) FX(Cn, nr, j, k) = (FX(vel, nr - 1, j, k) / 3.0 - 3.0 * FX(vel, nr, j, k)) / dr;
    }
    // wall temperatures: inner 0, outer 1 (the horizontal annulus: inner 1, outer 0)
    if (i == 0) FX(thn, 0, j, k) = d.horizontal ? 1.0 : 0.0;
    else if (i == nr + 1) FX(thn, nr + 1, j, k) = d.horizontal ? 0.0 : 1.0;
    const size_t p = (size_t)t;
    d.fld[GB_R_Ap][p] = d.fld[GB_R_A][p];
    d.fld[GB_R_A][p] = An[p];
    d.fld[GB_R_Bp][p] = d.fld[GB_R_B][p];
    d.fld[GB_R_B][p] = Bn[p];
    d.fld[GB_R_Cp][p] = d.fld[GB_R_C][p];
    d.fld[GB_R_C][p] = Cn[p];
    d.fld[GB_R_thp][p] = d.fld[GB_R_th][p];
    d.fld[GB_R_th][p] = thn[p];
}

// ---------------------------------------------------------------------------
// Multigrid line relaxation (rot3dmg.f:1543-2173)
// ---------------------------------------------------------------------------

// Solver of each (component, direction): 0 pdma, 1 tdma, 2 ptdma.
__host__ __device__ __forceinline__ int r3_kind(int comp, int dir)
{
    if (dir == 2) return 2;
    if (dir == 0) return comp == 3 ? 1 : 0;
    return comp == 1 ? 1 : 0;
}
__host__ __device__ __forceinline__ int r3_len(int comp, int dir, int n1, int n2, int n3)
{
    if (dir == 0) return comp == 3 ? n1 - 1 : n1;
    if (dir == 1) return comp == 1 ? n2 - 1 : n2;
    return n3;
}
__host__ __device__ __forceinline__ int r3_tabsize(int kind, int n)
{
    return kind == 0 ? (int)pdma_fac_len(n) : kind == 1 ? (int)tdma_fac_len(n) : 7 * n;
}
__host__ __device__ __forceinline__ int r3_tabsize32(int kind, int n)
{
    return kind == 0 ? (int)pdma32_len(n) : kind == 1 ? (int)tdma32_len(n) : 4;
}
__host__ __device__ __forceinline__ int r3_imax(int comp, int n1) { return comp == 3 ? n1 - 1 : n1; }
__host__ __device__ __forceinline__ int r3_jmax(int comp, int n2) { return comp == 1 ? n2 - 1 : n2; }

// Matrix row e (0-based) of a line of component comp in direction dir on
// level L (ti: the line's i for z- and phi-lines), as the reference builds
// it: relax1 :1576-1598, :1614-1643, :1652-1683; relax2 :1776-1799,
// :1830-1878, :1890-1926; relax3 :2022-2026, :2060-2081, :2094-2120.
__device__ void r3_coef(const R3Lev &L, int comp, int dir, int ti, int e, double &a, double &b, double &c, double &dd,
                        double &ee)
{
    const int n1 = L.n1, n2 = L.n2;
    const double hr = L.hr, hhr = L.hhr, hhz = L.hhz, hhp = L.hhp;
    dd = 0.0;
    ee = 0.0;
    if (dir == 0) {
        const int i = e + 1;
        if (comp == 1) {
            const double rval = L.rvc[i];
            if (i == 1) {
                a = 0.0;
                b = 0.0;
                c = -2.0 / hhr - 1.0 / hr / rval * 0.5 - 2.0 / hhz - 2.0 / hhp / (rval * rval);
                dd = 5.0 / hhr / 3.0 + 1.0 / hr / rval * 0.5;
                ee = -0.2 / hhr;
            } else if (i == n1) {
                a = -0.2 / hhr;
                b = 5.0 / hhr / 3.0 - 1.0 / hr / rval * 0.5;
                c = -2.0 / hhr + 1.0 / hr / rval * 0.5 - 2.0 / hhz - 2.0 / hhp / (rval * rval);
            } else {
                a = 0.0;
                b = 1.0 / hhr - 0.5 / hr / rval;
                c = -(2.0 / hhr + 2.0 / hhz + 2.0 / hhp / (rval * rval));
                dd = 1.0 / hhr + 0.5 / hr / rval;
            }
        } else if (comp == 2) {
            const double rval = L.rvc[i];
            const double rq = rval * rval;
            if (i == 1) {
                a = 0.0;
                b = 0.0;
                c = -2.0 / hhr - 2.0 / hhp / rq + 1.0 / rq;
                dd = 5.0 / 3.0 / hhr + 4.0 / 3.0 / hr / rval;
                ee = -0.2 / hhr;
            } else if (i == n1) {
                a = -0.2 / hhr;
                b = 5.0 / 3.0 / hhr - 4.0 / 3.0 / hr / rval;
                c = -2.0 / hhr - 2.0 / hhp / rq + 1.0 / rq;
            } else {
                a = 0.0;
                b = 1.0 / hhr - 1.5 / hr / rval;
                c = -(2.0 / hhr + 2.0 / hhp / rq) + 1.0 / rq;
                dd = 1.0 / hhr + 1.5 / hr / rval;
            }
            c = c - 2.0 / hhz;
        } else {
            const double rval = L.rvv[i];
            const double rq = rval * rval;
            a = 1.0 / hhr - 1.5 / hr / rval;
            b = -(2.0 / hhr - 1.0 / rq + 2.0 / hhp / rq);
            c = 1.0 / hhr + 1.5 / hr / rval;
            b = b - 2.0 / hhz;
        }
    } else if (dir == 1) {
        const int i = ti, j = e + 1;
        if (comp == 1) {
            const double rval = L.rvc[i];
            a = 1.0 / hhz;
            b = -(2.0 / hhz + 2.0 / hhp / (rval * rval));
            c = 1.0 / hhz;
            if (i == 1) b = b - 2.0 / hhr - 1.0 / hr / rval * 0.5;
            else if (i == n1) b = b - 2.0 / hhr + 1.0 / hr / rval * 0.5;
            else b = b - 2.0 / hhr;
        } else if (comp == 2) {
            const double rval = L.rvc[i];
            const double rq = rval * rval;
            if (j == 1) {
                a = 0.0;
                b = 0.0;
                c = -2.0 / hhz - 2.0 / hhp / rq + 1.0 / rq;
                dd = 5.0 / 3.0 / hhz;
                ee = -0.2 / hhz;
            } else if (j == n2) {
                a = -0.2 / hhz;
                b = 5.0 / 3.0 / hhz;
                c = -2.0 / hhz - 2.0 / hhp / rq + 1.0 / rq;
            } else {
                a = 0.0;
                b = 1.0 / hhz;
                c = -(2.0 / hhz + 2.0 / hhp / rq) + 1.0 / rq;
                dd = 1.0 / hhz;
            }
            c = c - 2.0 / hhr;
        } else {
            const double rval = L.rvv[i];
            const double rq = rval * rval;
            if (j == 1) {
                a = 0.0;
                b = 0.0;
                c = -2.0 / hhz - 2.0 / hhr + 1.0 / rq - 2.0 / hhp / rq;
                dd = 5.0 / hhz / 3.0;
                ee = -0.2 / hhz;
            } else if (j == n2) {
                a = -0.2 / hhz;
                b = 5.0 / hhz / 3.0;
                c = -2.0 / hhz - 2.0 / hhr + 1.0 / rq - 2.0 / hhp / rq;
            } else {
                a = 0.0;
                b = 1.0 / hhz;
                c = -(2.0 / hhz + 2.0 / hhr + 2.0 / hhp / rq) + 1.0 / rq;
                dd = 1.0 / hhz;
            }
        }
    } else {
        const int i = ti;
        if (comp == 1) {
            const double rval = L.rvc[i];
            a = 1.0 / hhp / (rval * rval);
            b = -(2.0 / hhz + 2.0 / hhp / (rval * rval));
            c = 1.0 / hhp / (rval * rval);
            if (i == 1) b = b - 2.0 / hhr - 1.0 / hr / rval * 0.5;
            else if (i == n1) b = b - 2.0 / hhr + 1.0 / hr / rval * 0.5;
            else b = b - 2.0 / hhr;
        } else if (comp == 2) {
            const double rval = L.rvc[i];
            const double rq = rval * rval;
            a = 1.0 / hhp / rq;
            c = 1.0 / hhp / rq;
            b = -(2.0 / hhp / rq) + 1.0 / rq;
            b = b - 2.0 / hhr;
            b = b - 2.0 / hhz;
        } else {
            const double rval = L.rvv[i];
            const double rq = rval * rval;
            a = 1.0 / hhp / rq;
            b = -(2.0 / hhr - 1.0 / rq + 2.0 / hhp / rq);
            c = 1.0 / hhp / rq;
            b = b - 2.0 / hhz;
        }
    }
}

struct FacJob {
    int lev, comp, dir, ti;
    double *tab;
};

// Runs the matrix half of the reference's eliminations once per line class
// and records what the right-hand-side half needs (one thread per class, seven
// rows of scratch each): pdma and tdma in banded.cuh's layouts,
//   ptdma [A | B | C | F1 | F2 | F3 | 1/B]: eliminated a (fill-in column), b,
//         c; multipliers of row j and of row n at step j; the last multiplier;
//         reciprocals of the pivots.
__global__ void k_r3d_factors(const __grid_constant__ R3Dev d, const FacJob *jobs, int njobs, double *work, int wstride)
{
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= njobs) return;
    const FacJob J = jobs[q];
    const R3Lev &L = d.lev[J.lev];
    const int kind = r3_kind(J.comp, J.dir);
    const int n = r3_len(J.comp, J.dir, L.n1, L.n2, L.n3);
    double *T = J.tab;
    if (kind <= 1) {
        double *w = work + (size_t)q * wstride;
        double *a = w, *b = w + n, *c = w + 2 * n, *dd = w + 3 * n, *ee = w + 4 * n;
        for (int e = 0; e < n; ++e) r3_coef(L, J.comp, J.dir, J.ti, e, a[e], b[e], c[e], dd[e], ee[e]);
        if (kind == 0) factor_pdma(a, b, c, dd, ee, n, T, w + 5 * n);
        else factor_tdma(a, b, c, n, T);
    } else {
        double *a = T, *b = T + n, *c = T + 2 * n, *F1 = T + 3 * n, *F2 = T + 4 * n, *F3 = T + 5 * n;
        double dummy_d, dummy_e;
        for (int e = 0; e < n; ++e) {
            r3_coef(L, J.comp, J.dir, J.ti, e, a[e], b[e], c[e], dummy_d, dummy_e);
            F1[e] = 0.0;
            F2[e] = 0.0;
        }
        const int N = n - 1;
        double fact;
        for (int j = 1; j <= n - 3; ++j) {
            fact = a[j] / b[j - 1];
            b[j] = b[j] - fact * c[j - 1];
            a[j] = -fact * a[j - 1];
            F1[j] = fact;
            fact = c[N] / b[j - 1];
            c[N] = -fact * c[j - 1];
            b[N] = b[N] - fact * a[j - 1];
            F2[j] = fact;
        }
        fact = a[n - 2] / b[n - 3];
        b[n - 2] = b[n - 2] - fact * c[n - 3];
        c[n - 2] = c[n - 2] - fact * a[n - 3];
        F1[n - 2] = fact;
        fact = c[N] / b[n - 3];
        a[N] = a[N] - fact * c[n - 3];
        b[N] = b[N] - fact * a[n - 3];
        F2[n - 2] = fact;
        fact = a[N] / b[n - 2];
        b[N] = b[N] - fact * c[n - 2];
        F3[0] = fact;
        for (int j = 0; j < n; ++j) T[6 * n + j] = 1.0 / b[j];
    }
}

static const double F02 = (double)0.2f;   // REAL*4 literal 0.2 (rot3dmg.f:1626, 1800, 2029, 2106 ...)

// Divisors with their stored reciprocals: x / d is the IEEE quotient (divrn.cuh)
// up to the sign of a zero, in 3 FP64 instructions where the hardware division
// takes 9 (562 cycles of an SM quarter's FP64 unit against 192).
struct Dv {
    double v, inv;
};
struct Rv {   // a radius, with the reciprocal of its square
    double v, inv, inv2;
};
__device__ __forceinline__ double operator/(double a, const Dv &d) { return div_by_rcp_neg(a, d.v, d.inv); }
__device__ __forceinline__ double operator/(double a, const Rv &r) { return div_by_rcp_neg(a, r.v, r.inv); }
__device__ __forceinline__ Dv operator*(const Rv &r, const Rv &) { return {r.v * r.v, r.inv2}; }
#define DV3 (Dv{3.0, 1.0 / 3.0})

#define PV(i, j, k) v[(size_t)(i) + (size_t)L1 * ((size_t)(j) + (size_t)L2 * (size_t)(k))]
#define RF(i, j, k) f[(size_t)(i) + (size_t)L1 * ((size_t)(j) + (size_t)L2 * (size_t)(k))]

// Right-hand side of row e of line (p, q): relax1 :1599-1601, :1616-1640,
// :1655-1681; relax2 :1798-1816, :1858-1876, :1891-1922; relax3 :2027-2041,
// :2082-2085, :2096-2118.
template <int COMP>
__device__ __forceinline__ double r3_rhs(const R3Lev &L, const R3Work &W, int dir, int p, int q, int e)
{
    const int n1 = L.n1, n2 = L.n2, n3 = L.n3, L1 = L.L1, L2 = L.L2;
    const Dv hr{L.hr, L.ihr}, hhr{L.hhr, L.ihhr}, hhz{L.hhz, L.ihhz}, hhp{L.hhp, L.ihhp};
    const double *v = W.v, *f = W.f;
    if (dir == 0) {
        const int i = e + 1, j = p, k = q;
        const int ka = k == n3 ? 1 : k + 1, km = k - 1;
        if (COMP == 1) {
            const Rv rval{L.rvc[i], L.dirc[i], L.diqc[i]};
            return -(PV(i, j + 1, k) + PV(i, j - 1, k)) / hhz - (PV(i, j, ka) + PV(i, j, km)) / hhp / (rval * rval) +
                   RF(i, j, k);
        } else if (COMP == 2) {
            const Rv rval{L.rvc[i], L.dirc[i], L.diqc[i]};
            const Dv rq = rval * rval;
            if (j == 1)
                return -(5.0 / 3.0 * PV(i, j + 1, k) - F02 * PV(i, j + 2, k)) / hhz -
                       (PV(i, j, ka) + PV(i, j, km)) / hhp / rq + RF(i, j, k);
            if (j == n2)
                return -(5.0 / 3.0 * PV(i, j - 1, k) - F02 * PV(i, j - 2, k)) / hhz -
                       (PV(i, j, ka) + PV(i, j, km)) / hhp / rq + RF(i, j, k);
            return -(PV(i, j - 1, k) + PV(i, j + 1, k)) / hhz - (PV(i, j, ka) + PV(i, j, km)) / hhp / rq + RF(i, j, k);
        } else {
            const Rv rval{L.rvv[i], L.dirv[i], L.diqv[i]};
            const Dv rq = rval * rval;
            if (j == 1)
                return -(5.0 * PV(i, j + 1, k) / DV3 - F02 * PV(i, j + 2, k)) / hhz -
                       (PV(i, j, ka) + PV(i, j, km)) / hhp / rq + RF(i, j, k);
            if (j == n2)
                return -(5.0 * PV(i, j - 1, k) / DV3 - F02 * PV(i, j - 2, k)) / hhz -
                       (PV(i, j, ka) + PV(i, j, km)) / hhp / rq + RF(i, j, k);
            return -(PV(i, j - 1, k) + PV(i, j + 1, k)) / hhz - (PV(i, j, ka) + PV(i, j, km)) / hhp / rq + RF(i, j, k);
        }
    } else if (dir == 1) {
        const int i = p, j = e + 1, k = q;
        const int ka = k == n3 ? 1 : k + 1, km = k - 1;
        if (COMP == 1) {
            const Rv rval{L.rvc[i], L.dirc[i], L.diqc[i]};
            if (i == 1)
                return -(5.0 * PV(i + 1, j, k) / DV3 - F02 * PV(i + 2, j, k)) / hhr - 1.0 * PV(i + 1, j, k) / hr / rval * 0.5 -
                       (PV(i, j, ka) + PV(i, j, km)) / hhp / (rval * rval) + RF(i, j, k);
            if (i == n1)
                return -(5.0 * PV(i - 1, j, k) / DV3 - F02 * PV(i - 2, j, k)) / hhr + 1.0 * PV(i - 1, j, k) / hr / rval * 0.5 -
                       (PV(i, j, ka) + PV(i, j, km)) / hhp / (rval * rval) + RF(i, j, k);
            return -(PV(i + 1, j, k) + PV(i - 1, j, k)) / hhr - 0.5 * (PV(i + 1, j, k) - PV(i - 1, j, k)) / hr / rval -
                   (PV(i, j, ka) + PV(i, j, km)) / hhp / (rval * rval) + RF(i, j, k);
        } else if (COMP == 2) {
            const Rv rval{L.rvc[i], L.dirc[i], L.diqc[i]};
            const Dv rq = rval * rval;
            if (i == 1)
                return -(5.0 / 3.0 * PV(i + 1, j, k) - 0.2 * PV(i + 2, j, k)) / hhr - 4.0 / 3.0 * PV(i + 1, j, k) / hr / rval -
                       (PV(i, j, ka) + PV(i, j, km)) / hhp / rq + RF(i, j, k);
            if (i == n1)
                return -(5.0 / 3.0 * PV(i - 1, j, k) - 0.2 * PV(i - 2, j, k)) / hhr + 4.0 / 3.0 * PV(i - 1, j, k) / hr / rval -
                       (PV(i, j, ka) + PV(i, j, km)) / hhp / rq + RF(i, j, k);
            return -(PV(i + 1, j, k) + PV(i - 1, j, k)) / hhr - 1.5 * (PV(i + 1, j, k) - PV(i - 1, j, k)) / hr / rval -
                   (PV(i, j, ka) + PV(i, j, km)) / hhp / rq + RF(i, j, k);
        } else {
            const Rv rval{L.rvv[i], L.dirv[i], L.diqv[i]};
            const Dv rq = rval * rval;
            return -(PV(i + 1, j, k) + PV(i - 1, j, k)) / hhr - 1.5 * (PV(i + 1, j, k) - PV(i - 1, j, k)) / hr / rval -
                   (PV(i, j, ka) + PV(i, j, km)) / hhp / rq + RF(i, j, k);
        }
    } else {
        const int i = p, j = q, k = e + 1;
        if (COMP == 1) {
            const Rv rval{L.rvc[i], L.dirc[i], L.diqc[i]};
            if (i == 1)
                return -(5.0 * PV(i + 1, j, k) / DV3 - F02 * PV(i + 2, j, k)) / hhr - PV(i + 1, j, k) / hr / rval * 0.5 -
                       (PV(i, j + 1, k) + PV(i, j - 1, k)) / hhz + RF(i, j, k);
            if (i == n1)
                return -(5.0 * PV(i - 1, j, k) / DV3 - F02 * PV(i - 2, j, k)) / hhr + PV(i - 1, j, k) / hr / rval * 0.5 -
                       (PV(i, j + 1, k) + PV(i, j - 1, k)) / hhz + RF(i, j, k);
            return -(PV(i + 1, j, k) + PV(i - 1, j, k)) / hhr - 0.5 * (PV(i + 1, j, k) - PV(i - 1, j, k)) / hr / rval -
                   (PV(i, j + 1, k) + PV(i, j - 1, k)) / hhz + RF(i, j, k);
        } else if (COMP == 2) {
            const Rv rval{L.rvc[i], L.dirc[i], L.diqc[i]};
            double rr;
            if (i == 1)
                rr = -(5.0 / 3.0 * PV(i + 1, j, k) - 0.2 * PV(i + 2, j, k)) / hhr - 4.0 / 3.0 * PV(i + 1, j, k) / hr / rval;
            else if (i == n1)
                rr = -(5.0 / 3.0 * PV(i - 1, j, k) - 0.2 * PV(i - 2, j, k)) / hhr + 4.0 / 3.0 * PV(i - 1, j, k) / hr / rval;
            else
                rr = -(PV(i + 1, j, k) + PV(i - 1, j, k)) / hhr - 1.5 * (PV(i + 1, j, k) - PV(i - 1, j, k)) / hr / rval;
            if (j == 1) return rr - (5.0 / 3.0 * PV(i, j + 1, k) - 0.2 * PV(i, j + 2, k)) / hhz + RF(i, j, k);
            if (j == n2) return rr - (5.0 / 3.0 * PV(i, j - 1, k) - 0.2 * PV(i, j - 2, k)) / hhz + RF(i, j, k);
            return rr - (PV(i, j - 1, k) + PV(i, j + 1, k)) / hhz + RF(i, j, k);
        } else {
            const Rv rval{L.rvv[i], L.dirv[i], L.diqv[i]};
            if (j == 1)
                return -(PV(i + 1, j, k) + PV(i - 1, j, k)) / hhr - 1.5 * (PV(i + 1, j, k) - PV(i - 1, j, k)) / hr / rval -
                       (5.0 * PV(i, j + 1, k) / DV3 - F02 * PV(i, j + 2, k)) / hhz + RF(i, j, k);
            if (j == n2)
                return -(PV(i + 1, j, k) + PV(i - 1, j, k)) / hhr - 1.5 * (PV(i + 1, j, k) - PV(i - 1, j, k)) / hr / rval -
                       (5.0 * PV(i, j - 1, k) / DV3 - F02 * PV(i, j - 2, k)) / hhz + RF(i, j, k);
            return -(PV(i + 1, j, k) + PV(i - 1, j, k)) / hhr - 1.5 * (PV(i + 1, j, k) - PV(i - 1, j, k)) / hr / rval -
                   (PV(i, j + 1, k) + PV(i, j - 1, k)) / hhz + RF(i, j, k);
        }
    }
}

// Periodic tridiagonal in place on a staged line: the reference's ptdma in its
// order, the factors of the next rows loaded while a row is eliminated (see
// banded.cuh).
template <int U = 2> __device__ __forceinline__ void ptdma_staged(const double *T, int n, double *x, int pitch)
{
    const double *Aa = T, *Bb = T + n, *Cc = T + 2 * n, *F1 = T + 3 * n, *F2 = T + 4 * n, *F3 = T + 5 * n, *iB = T + 6 * n;
    const int N = n - 1;
    double rN = x[N * pitch], prev = x[0];
    double f[U], g[U], r[U], b[U], ib[U];
    auto fetch = [&](int j0) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int j = min(j0 + u, n - 2);
            f[u] = F1[j];
            g[u] = F2[j];
            r[u] = x[j * pitch];
        }
    };
    fetch(1);
    for (int j0 = 1; j0 <= n - 2; j0 += U) {
        double f0[U], g0[U], r0[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            f0[u] = f[u];
            g0[u] = g[u];
            r0[u] = r[u];
        }
        if (j0 + U <= n - 2) fetch(j0 + U);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (j0 + u <= n - 2) {
                const double rj = r0[u] - f0[u] * prev;
                rN = rN - g0[u] * prev;
                x[(j0 + u) * pitch] = rj;
                prev = rj;
            }
        }
    }
    rN = rN - F3[0] * prev;
    const double yN = div_by_rcp_neg(rN, Bb[N], iB[N]);
    x[N * pitch] = yN;
    double y = div_by_rcp_neg(prev - Cc[n - 2] * yN, Bb[n - 2], iB[n - 2]);
    x[(n - 2) * pitch] = y;
    auto fetch_back = [&](int j0) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int j = max(j0 - u, 0);
            f[u] = Cc[j];
            g[u] = Aa[j];
            b[u] = Bb[j];
            ib[u] = iB[j];
            r[u] = x[j * pitch];
        }
    };
    fetch_back(n - 3);
    for (int j0 = n - 3; j0 >= 0; j0 -= U) {
        double f0[U], g0[U], b0[U], ib0[U], r0[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            f0[u] = f[u];
            g0[u] = g[u];
            b0[u] = b[u];
            ib0[u] = ib[u];
            r0[u] = r[u];
        }
        if (j0 - U >= 0) fetch_back(j0 - U);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (j0 - u >= 0) {
                y = div_by_rcp_neg(r0[u] - f0[u] * y - g0[u] * yN, b0[u], ib0[u]);
                x[(j0 - u) * pitch] = y;
            }
        }
    }
}

// A phi-line's matrix is the same in every row, a (x(k-1) + x(k+1)) + b x(k)
// = r(k) around the ring, and factors into two first-order recurrences with
// one coefficient: with rho + 1/rho = -b/a, 0 < rho < 1,
//   z(k) = r(k) / s + rho z(k-1),   x(k) = z(k) + rho x(k+1),   s = -a/rho,
// each around the ring: run from zero, its value after one turn, divided by
// 1 - rho^n, is the value it should have entered with.
struct R3Ring {
    float rho, scale, turn;   // rho, 1/s, 1/(1 - rho^n)
    int steps;                // scan steps; -1: a ring of the level is not diagonally dominant
};

// y(u) = t(u) + rho y(u-1) around the ring of n rows over W = 2^lw lanes (BACK:
// t(u) + rho y(u+1)), in place; rows past the end are left zero.
template <int M, bool BACK>
__device__ __forceinline__ void r3_ring(int lw, int n, const R3Ring &R, float (&t)[M])
{
    const unsigned full = 0xffffffffu;
    const int W = 1 << lw, lane = threadIdx.x & (W - 1), last = (n - 1) / M;   // the last lane with rows
    const int pos = BACK ? last - lane : lane;
    float w = 0.f, p = 1.f;
#pragma unroll
    for (int s = 0; s < M; ++s) {
        const int u = BACK ? M - 1 - s : s;
        if (lane * M + u < n) {
            w = __fmaf_rn(R.rho, w, t[u]);
            p *= R.rho;
        }
    }
#pragma unroll 1
    for (int d = 1; d < 1 << R.steps; d <<= 1) {
        const int src = BACK ? lane + d : lane - d;
        const float v = __shfl_sync(full, w, src, W), g = __shfl_sync(full, p, src, W);
        if (pos >= d) {
            w = __fmaf_rn(p, v, w);
            p *= g;
        }
    }
    const float c = __shfl_sync(full, w, BACK ? 0 : last, W) * R.turn;
    const float s = __fmaf_rn(p, c, w);
    float y = __shfl_sync(full, s, BACK ? lane + 1 : lane - 1, W);
    if (pos == 0) y = c;
#pragma unroll
    for (int q = 0; q < M; ++q) {
        const int u = BACK ? M - 1 - q : q;
        if (lane * M + u < n) {
            y = __fmaf_rn(R.rho, y, t[u]);
            t[u] = y;
        }
    }
}

// Rings of n rows, nl of them, in place in shared memory (x: [line][row], a
// lane's rows padded); rings longer than a warp's 512 rows by one thread each.
template <int M> __device__ __forceinline__ void r3_rings_m(const R3Ring *tab, const int *lines, int n, float *x, int xpitch, int nl)
{
    const int lw = wl_log2w(n), per = 32 >> lw;
    const int sub = (threadIdx.x & 31) >> lw, lane = threadIdx.x & ((1 << lw) - 1);
    const int slot = (threadIdx.x >> 5) * per + sub, nslots = ((int)blockDim.x >> 5) * per;
    for (int t0 = 0; t0 < nl; t0 += nslots) {
        if (t0 + slot - sub >= nl) continue;   // no line for this warp
        const bool live = t0 + slot < nl;
        const int l = live ? t0 + slot : t0 + slot - sub;   // idle groups repeat a line and store nothing
        const R3Ring R = tab[(lines[l] & 0xffff) - 1];
        float *xs = x + (size_t)l * xpitch + lane * (M + 1);
        float t[M];
#pragma unroll
        for (int u = 0; u < M; ++u) t[u] = lane * M + u < n ? xs[u] * R.scale : 0.f;
        r3_ring<M, false>(lw, n, R, t);
        r3_ring<M, true>(lw, n, R, t);
        if (live) {
#pragma unroll
            for (int u = 0; u < M; ++u) xs[u] = t[u];
        }
    }
}
// Levels with a ring that is not diagonally dominant (radii below the mesh
// size) take the FP64 factors, a thread per line.
__device__ __forceinline__ void r3_rings(const R3Ring *tab, const double *fac, const int *lines, int n, float *x, int xpitch, int nl)
{
    if (tab[0].steps < 0) {
        const int lg = wl_log2m(n), N = n - 1;
        for (int l = threadIdx.x; l < nl; l += blockDim.x) {
            const double *T = fac + (size_t)((lines[l] & 0xffff) - 1) * 7 * n;
            const double *Aa = T, *Bb = T + n, *Cc = T + 2 * n, *F1 = T + 3 * n, *F2 = T + 4 * n, *F3 = T + 5 * n;
            float *y = x + (size_t)l * xpitch;
            double rN = y[wl_slot(lg, N)], prev = y[wl_slot(lg, 0)];
            for (int k = 1; k <= n - 2; ++k) {
                const double r = y[wl_slot(lg, k)] - F1[k] * prev;
                rN -= F2[k] * prev;
                y[wl_slot(lg, k)] = (float)r;
                prev = r;
            }
            rN -= F3[0] * prev;
            const double yN = rN / Bb[N];
            double yk = (prev - Cc[n - 2] * yN) / Bb[n - 2];
            y[wl_slot(lg, N)] = (float)yN;
            y[wl_slot(lg, n - 2)] = (float)yk;
            for (int k = n - 3; k >= 0; --k) {
                yk = (y[wl_slot(lg, k)] - Cc[k] * yk - Aa[k] * yN) / Bb[k];
                y[wl_slot(lg, k)] = (float)yk;
            }
        }
    } else if (n <= 256) {
        r3_rings_m<8>(tab, lines, n, x, xpitch, nl);
    } else if (n <= 512) {
        r3_rings_m<16>(tab, lines, n, x, xpitch, nl);
    } else {
        for (int l = threadIdx.x; l < nl; l += blockDim.x) {
            const R3Ring R = tab[(lines[l] & 0xffff) - 1];
            float *y = x + (size_t)l * xpitch;
            const int lg = wl_log2m(n);
            float c = 0.f;
            for (int k = 0; k < n; ++k) c = __fmaf_rn(R.rho, c, y[wl_slot(lg, k)] * R.scale);
            c *= R.turn;
            for (int k = 0; k < n; ++k) y[wl_slot(lg, k)] = c = __fmaf_rn(R.rho, c, y[wl_slot(lg, k)] * R.scale);
            c = 0.f;
            for (int k = n - 1; k >= 0; --k) c = __fmaf_rn(R.rho, c, y[wl_slot(lg, k)]);
            c *= R.turn;
            for (int k = n - 1; k >= 0; --k) y[wl_slot(lg, k)] = c = __fmaf_rn(R.rho, c, y[wl_slot(lg, k)]);
        }
    }
}

// Dynamic shared memory of a solve block (two blocks an SM): the levels'
// descriptors, the staged lines' right-hand sides (R3_CHUNK_BYTES; a group of
// lines that must share a chunk fits them, r3_phases) and their factors.
// Behind the kernel's parameter each descriptor field would be a load of its
// own ahead of every pass's loads, and after each barrier again.
#define R3_LEVS 5   // levels 1 .. 4
#define R3_WEIGHTS 512   // float4: grids up to about 110 x 110 keep all levels' here
struct R3Shared {
    R3Lev lev[R3_LEVS];
    R3Work work[R3_LEVS];
    int my0, my1;           // the block's share of the phase at hand
    int p0, staged;         // its first chunk's factors: first radius, whether staged
    int n, len, chunk;      // rows of a line, elements of a table, lines of a chunk
    int lpitch, lg;         // FP32 lines' layout (warpline.cuh)
    int nl;                 // lines of the first chunk
    unsigned by_line, by_row;   // RowSplit of n and of nl
    int line[R3_THREADS];   // its first chunk's lines
    float4 weights[R3_WEIGHTS];   // the FP32 operator's, where they fit
};
#define R3_SMEM_BYTES (110 * 1024)
static_assert(sizeof(R3Shared) + R3_CHUNK_BYTES + R3_FAC_BYTES <= R3_SMEM_BYTES, "shared memory of a solve block");
__device__ __forceinline__ R3Shared &r3_shared()
{
    extern __shared__ __align__(16) unsigned char s_r3[];
    return *(R3Shared *)s_r3;
}
__device__ __forceinline__ void r3_descriptors(const R3Dev &d, int comp, bool mixed)
{
    R3Shared &S = r3_shared();
    for (int q = threadIdx.x; q < (int)(R3_LEVS * sizeof(R3Lev) / 4); q += R3_THREADS) ((unsigned *)S.lev)[q] = ((const unsigned *)d.lev)[q];
    for (int q = threadIdx.x; q < (int)(R3_LEVS * sizeof(R3Work) / 4); q += R3_THREADS)
        ((unsigned *)S.work)[q] = ((const unsigned *)d.work[comp])[q];
    __syncthreads();
    if (!mixed) return;
    int at = 0;
    for (int l = 1; l <= d.nlev; ++l) {
        const int n1 = S.lev[l].n1, n2 = S.lev[l].n2, need = (n1 + 1) + (n2 + 1) + (n1 + 4) / 4;
        if (at + need > R3_WEIGHTS) break;
        float4 *wi = S.weights + at, *wj = wi + n1 + 1;
        float *wp = (float *)(wj + n2 + 1);
        for (int i = threadIdx.x; i <= n1; i += R3_THREADS) {
            wi[i] = S.lev[l].wi[comp][i];
            wp[i] = S.lev[l].wp[comp][i];
        }
        for (int j = threadIdx.x; j <= n2; j += R3_THREADS) wj[j] = S.lev[l].wj[comp][j];
        __syncthreads();
        if (threadIdx.x == 0) {
            S.lev[l].wi[comp] = wi;
            S.lev[l].wj[comp] = wj;
            S.lev[l].wp[comp] = wp;
        }
        at += need;
    }
    __syncthreads();
}

// A block's share of a phase's entries [a, b) starts at x moved forward
// past the rest of a group that x would split (entries marked as continued
// belong with the next one); every block moves its two ends the same way,
// so the shares still partition [a, b).
__device__ __forceinline__ int r3_group_start(const int *lines, int a, int b, int x)
{
    if (x >= b) return b;
    while (x > a && (lines[x - 1] & 0x80000000)) ++x;
    return x;
}

// End of a chunk [c0, c1): moved back to the end of the last whole group
// (groups never exceed a chunk; the phase lists are built so).
__device__ __forceinline__ int r3_chunk_end(const int *lines, int c0, int c1)
{
    int e = c1;
    while (e > c0 + 1 && (lines[e - 1] & 0x80000000)) --e;
    return e;
}

template <int COMP> struct R3Point;
template <int COMP>
__device__ __forceinline__ void r3_rhs32_batch(const R3Lev &L, const R3Work &W, int dir, const int *s_line, int nl, int n, const RowSplit &split,
                               float *x, int lpitch, int lg);

// Starts the copy of the factors of nl lines: one table in direction 0, else
// one per radius p.  FP64 lists keep a radius's lines together, so the tables
// of a chunk's radii are few and lie in a row (p0 gets the first); FP32 ones
// take a table per line (a ring's is four words, read where it is used).
// Returns whether they fit.  line(t): the t-th line.
template <int COMP, class T, class Line>
__device__ __forceinline__ bool r3_fetch(const R3Lev &L, int dir, int n, int len, int nl, Line line, int tid, int nthr, int &p0)
{
    constexpr bool F64 = sizeof(T) == 8;
    extern __shared__ __align__(16) unsigned char s_r3[];
    T *sfac = (T *)(s_r3 + sizeof(R3Shared) + R3_CHUNK_BYTES);
    const T *fac = F64 ? (const T *)L.fac[COMP][dir] : (const T *)L.fac32[COMP][dir];
    const int room = (int)(R3_FAC_BYTES / sizeof(T));
    p0 = 1;
    if (dir == 0) {
        if (len > room) return false;
        async_copy(sfac, fac, len, tid, nthr);
    } else if constexpr (F64) {
        int a = line(0) & 0xffff, b = a;
        for (int t = threadIdx.x & 31; t < nl; t += 32) {
            a = min(a, line(t) & 0xffff);
            b = max(b, line(t) & 0xffff);
        }
        p0 = __reduce_min_sync(0xffffffffu, a);
        b = __reduce_max_sync(0xffffffffu, b);
        if ((b - p0 + 1) * len > room) return false;
        async_copy(sfac, fac + (size_t)(p0 - 1) * len, (b - p0 + 1) * len, tid, nthr);
    } else if (dir == 1) {
        if (nl * len > room) return false;
        for (int t = 0; t < nl; ++t) async_copy(sfac + t * len, fac + (size_t)((line(t) & 0xffff) - 1) * len, len, tid, nthr);
    }
    return true;
}

// What phase ph of direction dir on level lev reads besides the solution: the
// block's share of the lines, the first chunk's lines and factors, and what
// takes divisions to know (a thousand cycles of a phase of eight).  None of it
// changes during a solve, so it is fetched while the block waits at the
// barrier before the phase (threads 32 .. of the block).
template <int COMP, class T> __device__ __noinline__ void r3_prepare(int lev, int dir, int ph)
{
    R3Shared &S = r3_shared();
    const R3Lev &L = S.lev[lev];
    constexpr bool F64 = sizeof(T) == 8;
    const int tid = (int)threadIdx.x - 32, nthr = R3_THREADS - 32;
    const int *lines = L.lines[COMP][dir];
    const int a = L.poff[COMP][dir][ph], b = L.poff[COMP][dir][ph + 1];
    const int kind = r3_kind(COMP, dir), n = r3_len(COMP, dir, L.n1, L.n2, L.n3);
    const int len = F64 ? r3_tabsize(kind, n) : r3_tabsize32(kind, n);
    const int per = (b - a + (int)gridDim.x - 1) / (int)gridDim.x;
    const int my0 = r3_group_start(lines, a, b, a + (int)blockIdx.x * per);
    const int my1 = r3_group_start(lines, a, b, a + ((int)blockIdx.x + 1) * per);
    int p0 = 1;
    bool staged = false;
    int nl = 0, chunk = 1;
    if (my0 < my1) {
        chunk = r3_chunk(F64, dir, n, len);
        const int c1 = r3_chunk_end(lines, my0, min(my1, my0 + chunk));
        nl = c1 - my0;
        for (int t = tid; t < nl; t += nthr) S.line[t] = lines[my0 + t] & 0x7fffffff;
        staged = r3_fetch<COMP, T>(L, dir, n, len, c1 - my0, [&](int t) { return lines[my0 + t] & 0x7fffffff; }, tid, nthr, p0);
    }
    if (tid == 0) {
        S.my0 = my0;
        S.my1 = my1;
        S.p0 = p0;
        S.staged = staged;
        S.n = n;
        S.len = len;
        S.chunk = chunk;
        S.lpitch = F64 ? 0 : wl_pitch(n);
        S.lg = F64 ? 0 : wl_log2m(n);
        S.nl = nl;
        S.by_line = RowSplit(n).magic;
        S.by_row = RowSplit(max(nl, 1)).magic;
    }
}

// One phase of independent lines, prepared by r3_prepare: each block takes a
// contiguous share, in chunks that fit its shared memory.  All threads form a
// chunk's right-hand sides (along the line in direction 0, across the lines in
// the others, whichever runs with memory), the lines are eliminated (FP64: one
// thread per line in the reference's order; FP32: up to 32 lanes per line),
// the solutions go to the level's correction v.  Lines along r and z on plane
// k = n3 also write plane 0; phi-lines write plane 0 from plane n3.
template <int COMP, class T> __device__ __noinline__ void r3_phase(int lev, int dir)
{
    extern __shared__ __align__(16) unsigned char s_r3[];
    R3Shared &S = r3_shared();
    const R3Lev &L = S.lev[lev];
    const R3Work &W = S.work[lev];
    constexpr bool F64 = sizeof(T) == 8;
    const int my0 = S.my0, my1 = S.my1;
    if (my0 >= my1) return;
    const int n3 = L.n3, L1 = L.L1, L2 = L.L2;
    const int kind = r3_kind(COMP, dir), n = S.n, len = S.len, lpitch = S.lpitch, lg = S.lg, chunk = S.chunk;
    const int *lines = L.lines[COMP][dir];
    int *s_line = S.line;
    T *v = F64 ? (T *)W.v : (T *)W.v32;
    const T *fac = F64 ? (const T *)L.fac[COMP][dir] : (const T *)L.fac32[COMP][dir];
    T *x = (T *)(s_r3 + sizeof(R3Shared)), *sfac = (T *)(s_r3 + sizeof(R3Shared) + R3_CHUNK_BYTES);
    const RowSplit by_line(n, S.by_line);
    RowSplit by_row(S.nl, S.by_row);
    for (int c0 = my0; c0 < my1;) {
        int nl = S.nl;
        if (c0 != my0) {
            nl = r3_chunk_end(lines, c0, min(my1, c0 + chunk)) - c0;
            if (nl != by_row.n) by_row = RowSplit(nl);
        }
        const int c1 = c0 + nl, pitch = nl | 1;
        auto at = [&](int t, int e) -> T & { return F64 ? x[e * pitch + t] : x[t * lpitch + wl_slot(lg, e)]; };
        int p0 = S.p0;
        bool staged = S.staged;
        if (c0 != my0) {
            __syncthreads();   // the chunk before has left s_line, the factors and x
            for (int t = threadIdx.x; t < nl; t += R3_THREADS) s_line[t] = lines[c0 + t] & 0x7fffffff;
            __syncthreads();
            staged = r3_fetch<COMP, T>(L, dir, n, len, nl, [&](int t) { return s_line[t]; }, threadIdx.x, R3_THREADS, p0);
        }
        if constexpr (!F64) {
            r3_rhs32_batch<COMP>(L, W, dir, s_line, nl, n, dir == 0 ? by_line : by_row, x, lpitch, lg);
        } else if (dir == 0) {
            for (int idx = threadIdx.x; idx < nl * n; idx += R3_THREADS) {
                int t, e;
                by_line(idx, t, e);
                at(t, e) = r3_rhs<COMP>(L, W, 0, s_line[t] & 0xffff, s_line[t] >> 16, e);
            }
        } else {
            for (int idx = threadIdx.x; idx < nl * n; idx += R3_THREADS) {
                int e, t;
                by_row(idx, e, t);
                at(t, e) = r3_rhs<COMP>(L, W, dir, s_line[t] & 0xffff, s_line[t] >> 16, e);
            }
        }
        if constexpr (!F64) {   // rows past the line's end
            const int pad = wl_rows(n) - n, warp = threadIdx.x >> 5;
            for (int t = warp; t < nl; t += R3_THREADS / 32)
                for (int q = threadIdx.x & 31; q < pad; q += 32) at(t, n + q) = T(0);
        }
        async_copy_wait();
        __syncthreads();
        if constexpr (F64) {
            const int t = threadIdx.x;
            if (t < nl) {
                auto solve = [&](const double *tab) {
                    if (kind == 0) pdma_staged(tab, n, x + t, pitch);
                    else if (kind == 1) tdma_staged(tab, n, x + t, pitch);
                    else ptdma_staged(tab, n, x + t, pitch);
                };
                const int p = dir == 0 ? 1 : s_line[t] & 0xffff;
                if (staged) solve(sfac + (size_t)(p - p0) * len);
                else solve(fac + (size_t)(p - 1) * len);
            }
        } else if (kind == 2) {
            r3_rings((const R3Ring *)fac, L.fac[COMP][2], s_line, n, x, lpitch, nl);
        } else if (staged) {
            if (kind == 0) wl_lines<true, true>(sfac, dir == 0 ? 0 : len, n, x, lpitch, nl);
            else wl_lines<false, true>(sfac, dir == 0 ? 0 : len, n, x, lpitch, nl);
        } else {   // each line's table from global memory
            for (int t = 0; t < nl; ++t) {
                const T *tab = fac + (dir == 0 ? 0 : (size_t)((s_line[t] & 0xffff) - 1) * len);
                if (threadIdx.x < 32) {
                    if (kind == 0) wl_lines_m<16, true, true>(tab, 0, n, x + t * lpitch, lpitch, 1, 0, 1);
                    else wl_lines_m<16, false, true>(tab, 0, n, x + t * lpitch, lpitch, 1, 0, 1);
                }
            }
        }
        __syncthreads();
        if (dir == 0) {
            for (int idx = threadIdx.x; idx < nl * n; idx += R3_THREADS) {
                int t, e;
                by_line(idx, t, e);
                const int j = s_line[t] & 0xffff, k = s_line[t] >> 16;
                const T val = at(t, e);
                const int o = e + 1 + L1 * (j + L2 * k);
                v[o] = val;
                if (k == n3) v[o - L1 * L2 * n3] = val;
            }
        } else {
            for (int idx = threadIdx.x; idx < nl * n; idx += R3_THREADS) {
                int e, t;
                by_row(idx, e, t);
                const int i = s_line[t] & 0xffff, q = s_line[t] >> 16;
                const int j = dir == 1 ? e + 1 : q, k = dir == 1 ? q : e + 1;
                const T val = at(t, e);
                const int o = i + L1 * (j + L2 * k);
                v[o] = val;
                if (k == n3) v[o - L1 * L2 * n3] = val;
            }
        }
        c0 = c1;
    }
}

// Residual rc = rf - A psif at the level's unknowns (relax1 :1688-1720,
// relax2 :1935-1977, relax3 :2129-2160), one point per call.
template <int COMP>
__device__ __forceinline__ double r3_resid(const R3Lev &L, const R3Work &W, int i, int j, int k)
{
    const int n1 = L.n1, n2 = L.n2, n3 = L.n3, L1 = L.L1, L2 = L.L2;
    const Dv hr{L.hr, L.ihr}, hhr{L.hhr, L.ihhr}, hhz{L.hhz, L.ihhz}, hhp{L.hhp, L.ihhp};
    const double *v = W.v, *f = W.f;
    const int ka = k == n3 ? 1 : k + 1, km = k - 1;
    double temp;
    if (COMP == 1) {
        const Rv rval{L.rvc[i], L.dirc[i], L.diqc[i]};
        temp = (PV(i, j + 1, k) + PV(i, j - 1, k)) / hhz + (PV(i, j, ka) + PV(i, j, km)) / hhp / (rval * rval) -
               PV(i, j, k) * (2.0 / hhz + 2.0 / hhp / (rval * rval));
        if (i == 1)
            temp = temp + (-2.0 * PV(i, j, k) + 5.0 * PV(i + 1, j, k) / DV3 - 0.2 * PV(i + 2, j, k)) / hhr +
                   0.5 * (-PV(i, j, k) + PV(i + 1, j, k)) / hr / rval;
        else if (i == n1)
            temp = temp + (-2.0 * PV(i, j, k) + 5.0 * PV(i - 1, j, k) / DV3 - 0.2 * PV(i - 2, j, k)) / hhr +
                   0.5 * (PV(i, j, k) - PV(i - 1, j, k)) / hr / rval;
        else
            temp = temp + (PV(i - 1, j, k) - 2.0 * PV(i, j, k) + PV(i + 1, j, k)) / hhr +
                   0.5 * (PV(i + 1, j, k) - PV(i - 1, j, k)) / hr / rval;
    } else if (COMP == 2) {
        const Rv rval{L.rvc[i], L.dirc[i], L.diqc[i]};
        const Dv rq = rval * rval;
        temp = (PV(i, j, ka) - 2.0 * PV(i, j, k) + PV(i, j, km)) / hhp / rq + PV(i, j, k) / rq;
        if (i == 1)
            temp = temp + (-2.0 * PV(i, j, k) + 5.0 / 3.0 * PV(i + 1, j, k) - 0.2 * PV(i + 2, j, k)) / hhr +
                   4.0 / 3.0 * PV(i + 1, j, k) / hr / rval;
        else if (i == n1)
            temp = temp + (-2.0 * PV(i, j, k) + 5.0 / 3.0 * PV(i - 1, j, k) - 0.2 * PV(i - 2, j, k)) / hhr -
                   4.0 / 3.0 * PV(i - 1, j, k) / hr / rval;
        else
            temp = temp + (PV(i - 1, j, k) - 2.0 * PV(i, j, k) + PV(i + 1, j, k)) / hhr +
                   1.5 * (PV(i + 1, j, k) - PV(i - 1, j, k)) / hr / rval;
        if (j == 1)
            temp = temp + (-2.0 * PV(i, j, k) + 5.0 / 3.0 * PV(i, j + 1, k) - 0.2 * PV(i, j + 2, k)) / hhz;
        else if (j == n2)
            temp = temp + (-2.0 * PV(i, j, k) + 5.0 / 3.0 * PV(i, j - 1, k) - 0.2 * PV(i, j - 2, k)) / hhz;
        else
            temp = temp + (PV(i, j + 1, k) - 2.0 * PV(i, j, k) + PV(i, j - 1, k)) / hhz;
    } else {
        const Rv rval{L.rvv[i], L.dirv[i], L.diqv[i]};
        const Dv rq = rval * rval;
        temp = (PV(i + 1, j, k) + PV(i - 1, j, k)) / hhr + 1.5 * (PV(i + 1, j, k) - PV(i - 1, j, k)) / hr / rval +
               PV(i, j, k) / rq + (PV(i, j, ka) + PV(i, j, km)) / hhp / rq - PV(i, j, k) * (2.0 / hhr + 2.0 / hhp / rq);
        if (j == 1)
            temp = temp + (-2.0 * PV(i, j, k) + 5.0 * PV(i, j + 1, k) / DV3 - 0.2 * PV(i, j + 2, k)) / hhz;
        else if (j == n2)
            temp = temp + (-2.0 * PV(i, j, k) + 5.0 * PV(i, j - 1, k) / DV3 - 0.2 * PV(i, j - 2, k)) / hhz;
        else
            temp = temp + (PV(i, j + 1, k) - 2.0 * PV(i, j, k) + PV(i, j - 1, k)) / hhz;
    }
    return RF(i, j, k) - temp;
}

#undef PV
#undef RF

struct SolveCtx {
    int m;              // level-1 residual evaluations so far (selects the max slot)
};

// relax's line sweeps on level klev, whose first phase the barrier before has
// prepared; the barrier after each phase prepares the next.
template <int COMP, class T> __device__ __noinline__ bool r3_sweeps(const R3Dev &d, int klev)
{
    const R3Lev &L = r3_shared().lev[klev];
    const GridSync gs = d.gs[COMP];
    const int nrel = d.nrel;
    for (int irel = 1; irel <= nrel; ++irel)
        for (int dir = 0; dir < 3; ++dir) {
            const int nph = L.nphase[COMP][dir];
            for (int ph = 0; ph < nph; ++ph) {
                r3_phase<COMP, T>(klev, dir);
                const int nd = ph + 1 < nph ? dir : dir < 2 ? dir + 1 : 0, np = ph + 1 < nph ? ph + 1 : 0;
                const bool more = nd > dir || np > 0 || irel < nrel;
                if (!grid_sync(gs, [&] {
                        if (more) r3_prepare<COMP, T>(klev, nd, np);
                    })) {
                    async_copy_wait();
                    return false;
                }
            }
        }
    return true;
}

// One relaxation call relax<COMP>(nrel, klev); returns false when a grid
// barrier timed out.  The reference forms the residual after every sweep; it
// is read where a restriction follows (`residual`) and its norm on level 1.
template <int COMP>
__device__ bool r3_relax(const R3Dev &d, int klev, SolveCtx &cx, bool residual)
{
    if (!r3_sweeps<COMP, double>(d, klev)) return false;
    if (!residual && klev != 1) return true;
    const R3Lev &L = r3_shared().lev[klev];
    const R3Work &W = r3_shared().work[klev];
    const GridSync &gs = d.gs[COMP];
    unsigned long long *resmax = d.resmax + 2 * COMP;
    int *nanflag = d.nanflag + 2 * COMP;
    const int gt = blockIdx.x * blockDim.x + threadIdx.x, T = gridDim.x * blockDim.x;
    const int im = r3_imax(COMP, L.n1), jm = r3_jmax(COMP, L.n2), n3 = L.n3;
    // its max norm goes into slot m & 1; the other slot is cleared for the
    // next evaluation (nobody reads it before then)
    const int slot = cx.m & 1;
    if (klev == 1 && gt == 0) {
        resmax[slot ^ 1] = 0ull;
        nanflag[slot ^ 1] = 0;
    }
    const int npts = im * jm * n3;
    const RowSplit si(im), sj(jm);
    unsigned long long lmax = 0;   // bit patterns of non-negative doubles are ordered as they are
    int lnan = 0;
    for (int t = gt; t < npts; t += T) {
        int i, j, k, rest;
        si(t, rest, i);
        sj(rest, k, j);
        ++i;
        ++j;
        ++k;
        const double r = r3_resid<COMP>(L, W, i, j, k);
        W.res[(size_t)i + (size_t)L.L1 * ((size_t)j + (size_t)L.L2 * (size_t)k)] = r;
        const unsigned long long a = (unsigned long long)__double_as_longlong(r) & 0x7fffffffffffffffull;
        if (a > 0x7ff0000000000000ull) lnan = 1;
        else if (a > lmax) lmax = a;
    }
    if (klev == 1) {
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long v = __shfl_xor_sync(0xffffffffu, lmax, o);
            lmax = v > lmax ? v : lmax;
            lnan |= __shfl_xor_sync(0xffffffffu, lnan, o);
        }
        if ((threadIdx.x & 31) == 0) {
            if (lmax) atomicMax(&resmax[slot], lmax);
            if (lnan) atomicOr(&nanflag[slot], 1);
        }
        cx.m++;
    }
    return grid_sync(gs);
}

// corser (rot3dmg.f:2176-2265): coarse right-hand side and zero correction.
__device__ void r3_corser(const R3Dev &d, int comp, int klev)
{
    const R3Lev &F = r3_shared().lev[klev], &Cl = r3_shared().lev[klev + 1];
    const R3Work &FW = r3_shared().work[klev], &CW = r3_shared().work[klev + 1];
    const int n1c = Cl.n1, n2c = Cl.n2, n3c = Cl.n3;
    const int gt = blockIdx.x * blockDim.x + threadIdx.x;
    const int T = gridDim.x * blockDim.x;
    const int npts = Cl.L1 * Cl.L2 * (n3c + 1);
    const RowSplit si(Cl.L1), sj(Cl.L2);
    const double *rf = FW.res;
    const size_t F1 = (size_t)F.L1, F2 = (size_t)F.L2;
#define R(i, j, k) rf[(size_t)(i) + F1 * ((size_t)(j) + F2 * (size_t)(k))]
    for (int t = gt; t < npts; t += T) {
        int i, j, k, rest;
        si(t, rest, i);
        sj(rest, k, j);
        double val;
        if (i == 0 || i == n1c || j == 0 || j == n2c) {
            val = 0.0;
        } else if (k == 0 || k == n3c) {
            val = R(i, j, k);
        } else {
            const int ii = i + i, jj = j + j, kk = k + k;
            const int iip = ii + 1, iim = ii - 1, jjp = jj + 1, jjm = jj - 1, kkp = kk + 1, kkm = kk - 1;
            double temp = R(ii, jj, kk);
            temp = temp + temp + R(iip, jj, kk) + R(iim, jj, kk) + R(ii, jjp, kk) + R(ii, jjm, kk) + R(ii, jj, kkp) +
                   R(ii, jj, kkm);
            temp = temp + temp + R(iip, jjp, kk) + R(iip, jjm, kk) + R(iim, jjp, kk) + R(iim, jjm, kk) + R(iip, jj, kkp) +
                   R(iip, jj, kkm) + R(iim, jj, kkp) + R(iim, jj, kkm) + R(ii, jjp, kkp) + R(ii, jjp, kkm) +
                   R(ii, jjm, kkp) + R(ii, jjm, kkm);
            temp = temp + temp + R(iip, jjp, kkp) + R(iip, jjp, kkm) + R(iip, jjm, kkp) + R(iip, jjm, kkm) +
                   R(iim, jjm, kkp) + R(iim, jjm, kkm) + R(iim, jjp, kkp) + R(iim, jjp, kkm);
            val = temp * 0.015625;
        }
        CW.f[t] = val;
        CW.v[t] = 0.0;
    }
#undef R
}

// finer (rot3dmg.f:2268-2344): trilinear prolongation added to the fine
// level.  The coarse correction is cleared by the next corser.
__device__ void r3_finer(const R3Dev &d, int comp, int klev)
{
    const R3Lev &Cl = r3_shared().lev[klev], &F = r3_shared().lev[klev - 1];
    const R3Work &CW = r3_shared().work[klev], &FW = r3_shared().work[klev - 1];
    const int gt = blockIdx.x * blockDim.x + threadIdx.x;
    const int T = gridDim.x * blockDim.x;
    const int npts = F.L1 * F.L2 * (F.n3 + 1);
    const RowSplit si(F.L1), sj(F.L2);
    const double *pc = CW.v;
    const size_t C1 = (size_t)Cl.L1, C2 = (size_t)Cl.L2;
#define PC(i, j, k) pc[(size_t)(i) + C1 * ((size_t)(j) + C2 * (size_t)(k))]
    for (int t = gt; t < npts; t += T) {
        int i, j, k, rest;
        si(t, rest, i);
        sj(rest, k, j);
        const int i1 = i / 2, j1 = j / 2, k1 = k / 2;
        const bool ie = i1 * 2 == i, je = j1 * 2 == j, ke = k1 * 2 == k;
        double p;
        if (ie) {
            if (je) {
                if (ke) p = PC(i1, j1, k1);
                else p = (PC(i1, j1, k1) + PC(i1, j1, k1 + 1)) * 0.5;
            } else {
                if (ke) p = (PC(i1, j1, k1) + PC(i1, j1 + 1, k1)) * 0.5;
                else p = (PC(i1, j1, k1) + PC(i1, j1 + 1, k1) + PC(i1, j1, k1 + 1) + PC(i1, j1 + 1, k1 + 1)) * 0.25;
            }
        } else {
            if (je) {
                if (ke) p = (PC(i1, j1, k1) + PC(i1 + 1, j1, k1)) * 0.5;
                else p = (PC(i1, j1, k1) + PC(i1 + 1, j1, k1) + PC(i1, j1, k1 + 1) + PC(i1 + 1, j1, k1 + 1)) * 0.25;
            } else {
                if (ke)
                    p = (PC(i1, j1, k1) + PC(i1 + 1, j1, k1) + PC(i1, j1 + 1, k1) + PC(i1 + 1, j1 + 1, k1)) * 0.25;
                else
                    p = (PC(i1, j1, k1) + PC(i1 + 1, j1, k1) + PC(i1, j1 + 1, k1) + PC(i1 + 1, j1 + 1, k1) +
                         PC(i1, j1, k1 + 1) + PC(i1 + 1, j1, k1 + 1) + PC(i1, j1 + 1, k1 + 1) +
                         PC(i1 + 1, j1 + 1, k1 + 1)) *
                        0.125;
            }
        }
        FW.v[t] = p + FW.v[t];
    }
#undef PC
}

// poisson1/2/3 (rot3dmg.f:1216-1540) in one cooperative launch.
template <int COMP>
__global__ void __launch_bounds__(R3_THREADS, 2) k_r3d_solve(const __grid_constant__ R3Dev d, int step)
{
    if (*(volatile int *)d.abort) return;
    const int ni = d.ni, nj = d.nj;
    const int gt = blockIdx.x * blockDim.x + threadIdx.x, T = gridDim.x * blockDim.x;
    r3_descriptors(d, COMP, false);
    double *psi = d.fld[COMP == 1 ? GB_R_wel : COMP == 2 ? GB_R_vel : GB_R_uel];
    double *psip = d.fld[COMP == 1 ? GB_R_welp : COMP == 2 ? GB_R_velp : GB_R_uelp];
    const double *rhs = d.fld[COMP == 1 ? GB_R_wrh : COMP == 2 ? GB_R_vrh : GB_R_urh];
    const R3Lev &L = r3_shared().lev[1];
    const R3Work W = r3_shared().work[1];
    const GridSync gs = d.gs[COMP];
    const int n1p = L.L1, n2p = L.L2;
    const int nlvl = n1p * n2p * (L.n3 + 1);
    const RowSplit si(n1p), sj(n2p);
    // a barrier that prepares the first line phase of level l
    auto sync_before = [&](int l) {
        const bool ok = grid_sync(gs, [&] { r3_prepare<COMP, double>(l, 0, 0); });
        if (!ok) async_copy_wait();   // no copy in flight outlives the block
        return ok;
    };
    for (int t = gt; t < nlvl; t += T) {
        int i, j, k, rest;
        si(t, rest, i);
        sj(rest, k, j);
        W.f[t] = FX(rhs, i, j, k);
        W.v[t] = 2.0 * FX(psi, i, j, k) - FX(psip, i, j, k);
    }
    if (!sync_before(1)) return;
    SolveCtx cx;
    cx.m = 0;
    int status = GB_MAXSWEEPS, sweeps = d.maxsweeps;
    const int nlev = d.nlev;
    for (int sweep = 1; sweep <= d.maxsweeps; ++sweep) {
        if (sweep != 1 && !d.horizontal) {
            for (int t = gt; t < nlvl; t += T) {
                int i, j, k, rest;
                si(t, rest, i);
                sj(rest, k, j);
                const double pp = FX(psip, i, j, k);
                const double nv = pp + d.sor * (W.v[t] - pp);
                W.v[t] = nv;
                FX(psip, i, j, k) = nv;
            }
            // with one level a relaxation of level 1 follows, else a restriction
            if (!(nlev == 1 ? sync_before(1) : grid_sync(gs))) return;
        } else if (sweep != 1 && nlev == 1) {
            if (!sync_before(1)) return;
        }
        if (sweep == 1 || nlev == 1) {
            if (!r3_relax<COMP>(d, 1, cx, true)) return;
            if (!d.horizontal) {
                for (int t = gt; t < nlvl; t += T) {
                    int i, j, k, rest;
                    si(t, rest, i);
                    sj(rest, k, j);
                    FX(psip, i, j, k) = W.v[t];
                }
                if (!grid_sync(gs)) return;
            }
        }
        if (nlev > 1) {
            for (int l = 1; l <= nlev - 1; ++l) {
                r3_corser(d, COMP, l);
                if (!sync_before(l + 1)) return;
                if (!r3_relax<COMP>(d, l + 1, cx, l + 1 < nlev)) return;
            }
            for (int l = nlev; l >= 2; --l) {
                r3_finer(d, COMP, l);
                if (!sync_before(l - 1)) return;
                if (!r3_relax<COMP>(d, l - 1, cx, false)) return;
            }
        }
        const int slot = (cx.m - 1) & 1;
        const double resmax =
            __longlong_as_double((long long)*(volatile unsigned long long *)&d.resmax[2 * COMP + slot]);
        if (*(volatile int *)&d.nanflag[2 * COMP + slot]) {
            status = GB_NAN;
            sweeps = sweep;
            break;
        }
        if (resmax < d.tolcon) {
            status = GB_OK;
            sweeps = sweep;
            break;
        }
    }
    if (status == GB_OK) {
        const int imax = COMP == 3 ? d.nr : d.nr + 1;
        const int jmax = COMP == 1 ? d.nz : d.nz + 1;
        const int ii1 = COMP == 3 ? d.nr - 1 : d.nr;
        const int jj1 = COMP == 1 ? d.nz - 1 : d.nz;
        const int npts = (imax + 1) * (jmax + 1) * (d.np + 1);
        const RowSplit ti(imax + 1), tj(jmax + 1);
        for (int t = gt; t < npts; t += T) {
            int i, j, k, rest;
            ti(t, rest, i);
            tj(rest, k, j);
            const double old = FX(psi, i, j, k);
            FX(psip, i, j, k) = old;
            const bool inner = i >= 1 && i <= ii1 && j >= 1 && j <= jj1;
            FX(psi, i, j, k) = inner ? W.v[(size_t)i + (size_t)n1p * ((size_t)j + (size_t)n2p * (size_t)k)] : 0.0;
        }
    }
    if (gt == 0) {
        d.solve_status[COMP] = status;
        d.solve_sweeps[COMP] = sweeps;
        if (step >= 0) d.hist_sw[3 * step + COMP - 1] = sweeps;
        if (status != GB_OK) atomicExch(d.abort, status);
    }
}

// ---------------------------------------------------------------------------
// Mixed precision (GB_PRB_MIXED): FP32 V-cycles on the residual equation
// inside an FP64 defect correction.  The FP32 operator is the reference's
// operator with every division by a level constant or a radius replaced by
// a multiplication with its reciprocal; pivots of the factor tables are
// stored as reciprocals.
// ---------------------------------------------------------------------------

// FP32 fused tables (one thread per line class).
__global__ void k_r3d_factors32(const __grid_constant__ R3Dev d, const FacJob *jobs, int njobs)
{
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= njobs) return;
    const FacJob J = jobs[q];
    const R3Lev &L = d.lev[J.lev];
    const int kind = r3_kind(J.comp, J.dir);
    const int n = r3_len(J.comp, J.dir, L.n1, L.n2, L.n3);
    float *o = L.fac32[J.comp][J.dir] + (size_t)(J.dir == 0 ? 0 : J.ti - 1) * r3_tabsize32(kind, n);
    if (kind == 0) {
        pdma32_fold<true>(J.tab, n, o);
    } else if (kind == 1) {
        tdma32_fold<true>(J.tab, n, o);
    } else {
        double a, b, c, dd, ee;
        r3_coef(L, J.comp, J.dir, J.ti, 0, a, b, c, dd, ee);
        const double h = -b / (2.0 * a);
        if (!(h > 1.0 + 1e-9)) {
            *(R3Ring *)o = R3Ring{0.f, 0.f, 0.f, 0};
            return;
        }
        const double rho = 1.0 / (h + sqrt(h * h - 1.0)), turn = pow(rho, (double)n);
        int steps = 0;
        const int lw = wl_log2w(n), M = 1 << wl_log2m(n);
        while (steps < lw && pow(rho, (double)(M << steps)) > 9.313226e-10) ++steps;
        *(R3Ring *)o = R3Ring{(float)rho, (float)(-rho / a), (float)(1.0 / (1.0 - turn)), steps};
    }
}

// One scan-step count per level, component and ring direction (block x:
// level, y: component, z: direction 1 or 2): a warp's rings scan together, and
// the result must not depend on which rings share a warp.
__global__ void k_r3d_steps32(const __grid_constant__ R3Dev d)
{
    const R3Lev &L = d.lev[1 + blockIdx.x];
    const int comp = 1 + blockIdx.y, dir = 1 + blockIdx.z;
    if (r3_kind(comp, dir) != 2) return;
    const int inst = r3_imax(comp, L.n1);
    R3Ring *ring = (R3Ring *)L.fac32[comp][dir];
    __shared__ int most, weak;
    if (threadIdx.x == 0) most = weak = 0;
    __syncthreads();
    for (int q = threadIdx.x; q < inst; q += blockDim.x) {
        atomicMax(&most, ring[q].steps);
        if (ring[q].scale == 0.f) weak = 1;
    }
    __syncthreads();
    for (int q = threadIdx.x; q < inst; q += blockDim.x) ring[q].steps = weak ? -1 : most;
}

// Matrix weights of row i in r and of row j in z, from relax's operator: the
// references are those of r3_coef and r3_resid.
__global__ void k_r3d_weights32(const __grid_constant__ R3Dev d)
{
    const R3Lev &L = d.lev[1 + blockIdx.x];
    const int comp = 1 + blockIdx.y;
    const double ihr = 1.0 / L.hr, ihhr = 1.0 / L.hhr, ihhz = 1.0 / L.hhz, ihhp = 1.0 / L.hhp;
    for (int i = 1 + threadIdx.x; i <= L.n1; i += blockDim.x) {
        const double r = comp == 3 ? L.rvv[i] : L.rvc[i], ir = 1.0 / r, iq = 1.0 / (r * r);
        const double g = comp == 1 ? 0.5 : 1.5;
        double m = ihhr - g * ihr * ir, p = ihhr + g * ihr * ir, f = 0.0, c = -2.0 * ihhr;
        if (comp != 3 && (i == 1 || i == L.n1)) {
            const double e = (comp == 1 ? 0.5 : 4.0 / 3.0) * ihr * ir, s = i == 1 ? 1.0 : -1.0;
            m = i == 1 ? 0.0 : 5.0 / 3.0 * ihhr - e;
            p = i == 1 ? 5.0 / 3.0 * ihhr + e : 0.0;
            f = -0.2 * ihhr;
            if (comp == 1) c -= s * e;
        }
        c -= 2.0 * ihhp * iq;
        if (comp != 1) c += iq;
        L.wi[comp][i] = make_float4((float)m, (float)p, (float)f, (float)c);
        L.wp[comp][i] = (float)(ihhp * iq);
    }
    for (int j = 1 + threadIdx.x; j <= L.n2; j += blockDim.x) {
        double m = ihhz, p = ihhz, f = 0.0;
        if (comp != 1 && (j == 1 || j == L.n2)) {
            m = j == 1 ? 0.0 : 5.0 / 3.0 * ihhz;
            p = j == 1 ? 5.0 / 3.0 * ihhz : 0.0;
            f = -0.2 * ihhz;
        }
        L.wj[comp][j] = make_float4((float)m, (float)p, (float)f, (float)(-2.0 * ihhz));
    }
}

// A point's neighbours in FP32: right-hand side of its line in direction dir,
// or the residual (dir 3).  Loads first, arithmetic after, so that a thread
// has several points' loads in flight (r3_rhs32_batch).
template <int COMP> struct R3Point {
    float f, im, ip, ifar, jm, jp, jfar, ka, km, c;
    float4 wi, wj;
    float wp;
    __device__ __forceinline__ void load(const R3Lev &L, const R3Work &W, int dir, int i, int j, int k)
    {
        const int L1 = L.L1, P = L1 * L.L2, n1 = L.n1, n2 = L.n2, n3 = L.n3;
        const int o = i + L1 * j + P * k;
        const float *v = W.v32 + o;
        f = W.f32[o];
        if (dir != 0) {
            im = v[-1];
            ip = v[1];
            ifar = COMP != 3 ? v[i == 1 ? 2 : i == n1 ? -2 : 0] : 0.f;
        }
        if (dir != 1) {
            jm = v[-L1];
            jp = v[L1];
            jfar = COMP != 1 ? v[j == 1 ? 2 * L1 : j == n2 ? -2 * L1 : 0] : 0.f;
        }
        if (dir != 2) {
            km = v[-P];
            ka = v[k == n3 ? P * (1 - n3) : P];
        }
        if (dir == 3) c = v[0];
        wi = L.wi[COMP][i];
        wj = L.wj[COMP][j];
        wp = L.wp[COMP][i];
    }
    __device__ __forceinline__ float value(int dir) const
    {
        float r = f;
        if (dir != 0) {
            r = __fmaf_rn(-wi.x, im, __fmaf_rn(-wi.y, ip, r));
            if (COMP != 3) r = __fmaf_rn(-wi.z, ifar, r);
        }
        if (dir != 1) {
            r = __fmaf_rn(-wj.x, jm, __fmaf_rn(-wj.y, jp, r));
            if (COMP != 1) r = __fmaf_rn(-wj.z, jfar, r);
        }
        if (dir != 2) r = __fmaf_rn(-wp, ka + km, r);
        if (dir == 3) r = __fmaf_rn(-(wi.w + wj.w), c, r);
        return r;
    }
};


// The right-hand sides of a chunk's lines, four points per thread in flight.
template <int COMP>
__device__ __forceinline__ void r3_rhs32_batch(const R3Lev &L, const R3Work &W, int dir, const int *s_line, int nl, int n,
                                               const RowSplit &split, float *x, int lpitch, int lg)
{
    constexpr int U = 4;
    auto run = [&](auto d) {
        constexpr int DIR = decltype(d)::value;
        for (int base = threadIdx.x; base < nl * n; base += U * R3_THREADS) {
            R3Point<COMP> pt[U];
            int slot[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int idx = min(base + u * R3_THREADS, nl * n - 1);   // a repeated point is not stored
                int t, e;
                if (DIR == 0) split(idx, t, e);
                else split(idx, e, t);
                const int p = s_line[t] & 0xffff, q = s_line[t] >> 16;
                slot[u] = t * lpitch + wl_slot(lg, e);
                pt[u].load(L, W, DIR, DIR == 0 ? e + 1 : p, DIR == 0 ? p : DIR == 1 ? e + 1 : q, DIR == 2 ? e + 1 : q);
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (base + u * R3_THREADS < nl * n) x[slot[u]] = pt[u].value(DIR);
        }
    };
    if (dir == 0) run(std::integral_constant<int, 0>());
    else if (dir == 1) run(std::integral_constant<int, 1>());
    else run(std::integral_constant<int, 2>());
}

// relax in FP32; the residual only when a restriction follows.
template <int COMP>
__device__ bool r3_relax32(const R3Dev &d, int klev, bool residual)
{
    if (!r3_sweeps<COMP, float>(d, klev)) return false;
    if (!residual) return true;
    const R3Lev &L = r3_shared().lev[klev];
    const R3Work &W = r3_shared().work[klev];
    const int im = r3_imax(COMP, L.n1), jm = r3_jmax(COMP, L.n2), npts = im * jm * L.n3;
    const RowSplit si(im), sj(jm);
    const int T = gridDim.x * blockDim.x;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < npts; t += 2 * T) {
        R3Point<COMP> pt[2];
        int o[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            int i, j, k, rest;
            si(min(t + u * T, npts - 1), rest, i);
            sj(rest, k, j);
            o[u] = i + 1 + L.L1 * (j + 1 + L.L2 * (k + 1));
            pt[u].load(L, W, 3, i + 1, j + 1, k + 1);
        }
#pragma unroll
        for (int u = 0; u < 2; ++u)
            if (t + u * T < npts) W.res32[o[u]] = pt[u].value(3);
    }
    return grid_sync(d.gs[COMP]);
}

__device__ void r3_corser32(const R3Dev &d, int comp, int klev)
{
    const R3Lev &F = r3_shared().lev[klev], &Cl = r3_shared().lev[klev + 1];
    const R3Work &WF = r3_shared().work[klev], &WC = r3_shared().work[klev + 1];
    const int n1c = Cl.n1, n2c = Cl.n2, n3c = Cl.n3;
    const int gt = blockIdx.x * blockDim.x + threadIdx.x;
    const int T = gridDim.x * blockDim.x;
    const int npts = Cl.L1 * Cl.L2 * (n3c + 1);
    const RowSplit si(Cl.L1), sj(Cl.L2);
    const float *rf = WF.res32;
    const size_t F1 = (size_t)F.L1, F2 = (size_t)F.L2;
#define R(i, j, k) rf[(size_t)(i) + F1 * ((size_t)(j) + F2 * (size_t)(k))]
    for (int t = gt; t < npts; t += T) {
        int i, j, k, rest;
        si(t, rest, i);
        sj(rest, k, j);
        float val;
        if (i == 0 || i == n1c || j == 0 || j == n2c) {
            val = 0.f;
        } else if (k == 0 || k == n3c) {
            val = k == 0 ? 0.f : R(i, j, k);
        } else {
            const int ii = i + i, jj = j + j, kk = k + k;
            float c = 0.f;
#pragma unroll
            for (int dk = -1; dk <= 1; ++dk)
#pragma unroll
                for (int dj = -1; dj <= 1; ++dj)
#pragma unroll
                    for (int di = -1; di <= 1; ++di) {
                        const float w = (di ? 0.5f : 1.f) * (dj ? 0.5f : 1.f) * (dk ? 0.5f : 1.f);
                        c = __fmaf_rn(w, R(ii + di, jj + dj, kk + dk), c);
                    }
            val = c * 0.125f;
        }
        WC.f32[t] = val;
        WC.v32[t] = 0.f;
    }
#undef R
}

__device__ void r3_finer32(const R3Dev &d, int comp, int klev)
{
    const R3Lev &Cl = r3_shared().lev[klev], &F = r3_shared().lev[klev - 1];
    const R3Work &WC = r3_shared().work[klev], &WF = r3_shared().work[klev - 1];
    const int gt = blockIdx.x * blockDim.x + threadIdx.x;
    const int T = gridDim.x * blockDim.x;
    const int npts = F.L1 * F.L2 * (F.n3 + 1);
    const RowSplit si(F.L1), sj(F.L2);
    const float *pc = WC.v32;
    const size_t C1 = (size_t)Cl.L1, C2 = (size_t)Cl.L2;
#define PC(i, j, k) pc[(size_t)(i) + C1 * ((size_t)(j) + C2 * (size_t)(k))]
    for (int t = gt; t < npts; t += T) {
        int i, j, k, rest;
        si(t, rest, i);
        sj(rest, k, j);
        const int i1 = i >> 1, j1 = j >> 1, k1 = k >> 1;
        const int i2 = i1 + (i & 1), j2 = j1 + (j & 1), k2 = k1 + (k & 1);
        const float p = 0.125f * (PC(i1, j1, k1) + PC(i2, j1, k1) + PC(i1, j2, k1) + PC(i2, j2, k1) + PC(i1, j1, k2) +
                                  PC(i2, j1, k2) + PC(i1, j2, k2) + PC(i2, j2, k2));
        WF.v32[t] += p;
    }
#undef PC
}

// poisson1/2/3 in mixed precision: the FP64 iterate lives in level 1's v,
// the FP64 right-hand side in level 1's f.
template <int COMP>
__global__ void __launch_bounds__(R3_THREADS, 2) k_r3d_solve_mixed(const __grid_constant__ R3Dev d, int step)
{
    if (*(volatile int *)d.abort) return;
    const int ni = d.ni, nj = d.nj;
    const int gt = blockIdx.x * blockDim.x + threadIdx.x, T = gridDim.x * blockDim.x;
    r3_descriptors(d, COMP, true);
    double *psi = d.fld[COMP == 1 ? GB_R_wel : COMP == 2 ? GB_R_vel : GB_R_uel];
    double *psip = d.fld[COMP == 1 ? GB_R_welp : COMP == 2 ? GB_R_velp : GB_R_uelp];
    const double *rhs = d.fld[COMP == 1 ? GB_R_wrh : COMP == 2 ? GB_R_vrh : GB_R_urh];
    const R3Lev &L = r3_shared().lev[1];
    const R3Work W = r3_shared().work[1];
    const GridSync gs = d.gs[COMP];
    const int n1p = L.L1, n2p = L.L2;
    const int nlvl = n1p * n2p * (L.n3 + 1);
    const RowSplit si(n1p), sj(n2p);
    // a barrier that prepares the first line phase of level l
    auto sync_before = [&](int l) {
        const bool ok = grid_sync(gs, [&] { r3_prepare<COMP, float>(l, 0, 0); });
        if (!ok) async_copy_wait();   // no copy in flight outlives the block
        return ok;
    };
    for (int t = gt; t < nlvl; t += T) {
        int i, j, k, rest;
        si(t, rest, i);
        sj(rest, k, j);
        W.f[t] = FX(rhs, i, j, k);
        W.v[t] = 2.0 * FX(psi, i, j, k) - FX(psip, i, j, k);
        W.f32[t] = 0.f;
        W.v32[t] = 0.f;
    }
    if (!grid_sync(gs)) return;
    const int im = r3_imax(COMP, L.n1), jm = r3_jmax(COMP, L.n2), n3 = L.n3;
    const int nunk = im * jm * n3;
    const RowSplit ui(im), uj(jm);
    int status = GB_MAXSWEEPS, cycles = d.maxsweeps, m = 0;
    const int nlev = d.nlev;
    for (int it = 0;; ++it) {
        // FP64 residual of the iterate, its FP32 copy the cycle's right-hand side
        const int slot = m & 1;
        if (gt == 0) {
            d.resmax[2 * COMP + (slot ^ 1)] = 0ull;
            d.nanflag[2 * COMP + (slot ^ 1)] = 0;
        }
        unsigned long long lmax = 0;   // bit patterns of non-negative doubles are ordered as they are
        int lnan = 0;
        for (int t = gt; t < nunk; t += T) {
            int i, j, k, rest;
            ui(t, rest, i);
            uj(rest, k, j);
            ++i;
            ++j;
            ++k;
            const double r = r3_resid<COMP>(L, W, i, j, k);
            W.f32[(size_t)i + (size_t)L.L1 * ((size_t)j + (size_t)L.L2 * (size_t)k)] = d2f_rn(r);
            const unsigned long long a = (unsigned long long)__double_as_longlong(r) & 0x7fffffffffffffffull;
            if (a > 0x7ff0000000000000ull) lnan = 1;
            else if (a > lmax) lmax = a;
        }
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long v = __shfl_xor_sync(0xffffffffu, lmax, o);
            lmax = v > lmax ? v : lmax;
            lnan |= __shfl_xor_sync(0xffffffffu, lnan, o);
        }
        if ((threadIdx.x & 31) == 0) {
            if (lmax) atomicMax(&d.resmax[2 * COMP + slot], lmax);
            if (lnan) atomicOr(&d.nanflag[2 * COMP + slot], 1);
        }
        ++m;
        if (!sync_before(1)) return;
        const double res = __longlong_as_double((long long)*(volatile unsigned long long *)&d.resmax[2 * COMP + slot]);
        if (*(volatile int *)&d.nanflag[2 * COMP + slot]) {
            status = GB_NAN;
            cycles = it;
            break;
        }
        if (res < d.tolcon) {
            status = GB_OK;
            cycles = it;
            break;
        }
        if (it == d.maxsweeps) break;
        // one FP32 cycle from e = 0: relax on level 1, descent, ascent
        if (!r3_relax32<COMP>(d, 1, nlev > 1)) return;
        for (int l = 1; l <= nlev - 1; ++l) {
            r3_corser32(d, COMP, l);
            if (!sync_before(l + 1)) return;
            if (!r3_relax32<COMP>(d, l + 1, l + 1 < nlev)) return;
        }
        for (int l = nlev; l >= 2; --l) {
            r3_finer32(d, COMP, l);
            if (!sync_before(l - 1)) return;
            if (!r3_relax32<COMP>(d, l - 1, false)) return;
        }
        const double w = (it == 0 || d.horizontal) ? 1.0 : d.sor;
        for (int t = gt; t < nlvl; t += T) {
            W.v[t] += w * f2d(W.v32[t]);
            W.v32[t] = 0.f;
        }
        if (!grid_sync(gs)) return;
    }
    async_copy_wait();   // the copies prepared for a cycle that is not run
    if (status == GB_OK) {
        const int imax = COMP == 3 ? d.nr : d.nr + 1;
        const int jmax = COMP == 1 ? d.nz : d.nz + 1;
        const int ii1 = COMP == 3 ? d.nr - 1 : d.nr;
        const int jj1 = COMP == 1 ? d.nz - 1 : d.nz;
        const int npts = (imax + 1) * (jmax + 1) * (d.np + 1);
        const RowSplit ti(imax + 1), tj(jmax + 1);
        for (int t = gt; t < npts; t += T) {
            int i, j, k, rest;
            ti(t, rest, i);
            tj(rest, k, j);
            const double old = FX(psi, i, j, k);
            FX(psip, i, j, k) = old;
            const bool inner = i >= 1 && i <= ii1 && j >= 1 && j <= jj1;
            FX(psi, i, j, k) = inner ? W.v[(size_t)i + (size_t)n1p * ((size_t)j + (size_t)n2p * (size_t)k)] : 0.0;
        }
    }
    if (gt == 0) {
        d.solve_status[COMP] = status;
        d.solve_sweeps[COMP] = cycles;
        if (step >= 0) d.hist_sw[3 * step + COMP - 1] = cycles;
        if (status != GB_OK) atomicExch(d.abort, status);
    }
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
struct gb_r3d {
    gb_r3d_params p;
    R3Dev dev;
    double *fields = nullptr, *pool = nullptr, *work = nullptr, *tables = nullptr;
    int *itab = nullptr;
    void *small = nullptr;
    double *hist_nu = nullptr;
    int *hist_sw = nullptr;
    int hist_cap = 0;
    unsigned *sync = nullptr;
    int grid = 0;
    cudaStream_t stream = nullptr, side = nullptr;   // side: the v solve, beside the w solve
    cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
};

static int r3_levels(int nr, int nz)
{
    int nlev = 0, itest = nr, itest2 = nr, jtest = nz, jtest2 = nz;
    for (int i = 2; i <= 8; ++i) {
        itest /= 2;
        jtest /= 2;
        if (itest * 2 - itest2 == 0 && jtest * 2 - jtest2 == 0) {
            if (itest2 >= 4 && jtest2 >= 4) nlev++;
            itest2 = itest;
            jtest2 = jtest;
        } else {
            break;
        }
    }
    if (nlev > 4) nlev = 4;
    return nlev < 1 ? 1 : nlev;
}

extern "C" void gb_r3d_default_params(gb_r3d_params *p, int nr, int nz, int np)
{
    if (!p) return;
    memset(p, 0, sizeof(*p));
    p->nr = nr;
    p->nz = nz;
    p->np = np;
    p->dt = 1e-5;
    p->r0 = 0.5;
    p->rmax = 1.0;
    p->zmax = 0.5;
    p->Ra = 1e6;
    p->Re = 500.0;
    p->Gr = 0.0;
    p->Pr = 7.0;
    p->tolcon = 1e-5;
    p->sor = 1.2;
    p->maxsweeps = 500;
    p->nrel = 2;
    p->smoother = GB_SMOOTHER_LEX;
    p->precision = GB_PRB_FP64;
}

extern "C" int gb_r3d_destroy(gb_r3d *h)
{
    if (!h) return GB_OK;
    cudaFree(h->fields);
    cudaFree(h->pool);
    cudaFree(h->work);
    cudaFree(h->tables);
    cudaFree(h->itab);
    cudaFree(h->small);
    cudaFree(h->hist_nu);
    cudaFree(h->hist_sw);
    if (h->stream) cudaStreamDestroy(h->stream);
    if (h->side) cudaStreamDestroy(h->side);
    if (h->ev_fork) cudaEventDestroy(h->ev_fork);
    if (h->ev_join) cudaEventDestroy(h->ev_join);
    delete h;
    return GB_OK;
}

// Phase lists of one (level, component, direction), as packed (p, q);
// R3_CONT marks an entry whose line must be solved in the same chunk as the
// next entry's.
//
// LEX: the anti-diagonals p + q, in the reference's order.
//
// ZEBRA: lines with even p + q, then odd.  A line on a one-sided row (p = 1
// or P where p is one-sided, likewise q) also reads the line two over, of
// its own colour; within a colour such lines are solved before the lines
// they read (corners, then the other one-sided lines, then the rest), so
// every read two lines over sees the value from before the colour's pass.
// On the device a colour is one phase: a line and the lines that read it
// two over form a group of consecutive entries that one block solves in
// one chunk, whose right-hand sides are all formed before any of its
// eliminations writes.  A group larger than a chunk (only on grids far from
// the sizes the solver is built for) makes the classes separate phases in
// the same order.
#define R3_CONT 0x80000000u

// Lines that any chunk of n-row lines holds: the least of both types.
static int r3_chunk_lines(int comp, int dir, int n)
{
    const int kind = r3_kind(comp, dir);
    return std::min(r3_chunk(true, dir, n, r3_tabsize(kind, n)), r3_chunk(false, dir, n, r3_tabsize32(kind, n)));
}

static void r3_phases(int mode, int pslow, int comp, int dir, int n1, int n2, int n3, std::vector<int> &lines,
                      std::vector<int> &off)
{
    const int im = r3_imax(comp, n1), jm = r3_jmax(comp, n2);
    int P, Q, p_os, q_os;
    if (dir == 0) {
        P = jm;
        Q = n3;
        p_os = comp != 1;
        q_os = 0;
    } else if (dir == 1) {
        P = im;
        Q = n3;
        p_os = comp != 3;
        q_os = 0;
    } else {
        P = im;
        Q = jm;
        p_os = comp != 3;
        q_os = comp != 1;
    }
    off.clear();
    lines.clear();
    off.push_back(0);
    if (mode == GB_SMOOTHER_LEX) {
        for (int dsum = 2; dsum <= P + Q; ++dsum) {
            for (int p = std::max(1, dsum - Q); p <= std::min(P, dsum - 1); ++p) lines.push_back(p | ((dsum - p) << 16));
            off.push_back((int)lines.size());
        }
        return;
    }
    const int chunk = r3_chunk_lines(comp, dir, r3_len(comp, dir, n1, n2, n3));
    auto cls_of = [&](int p, int q) { return (p_os && (p == 1 || p == P)) + (q_os && (q == 1 || q == Q)); };
    auto id = [&](int p, int q) { return (q - 1) * P + (p - 1); };
    for (int colour = 0; colour < 2; ++colour) {
        // groups: union of each one-sided line with the line it reads two over
        std::vector<int> parent((size_t)P * Q);
        for (size_t t = 0; t < parent.size(); ++t) parent[t] = (int)t;
        std::function<int(int)> root = [&](int x) { return parent[x] == x ? x : (parent[x] = root(parent[x])); };
        auto join = [&](int a, int b) { parent[root(a)] = root(b); };
        for (int q = 1; q <= Q; ++q)
            for (int p = 1; p <= P; ++p) {
                if (((p + q) & 1) != colour) continue;
                if (p_os && p == 1 && P >= 3) join(id(p, q), id(3, q));
                if (p_os && p == P && P >= 3) join(id(p, q), id(P - 2, q));
                if (q_os && q == 1 && Q >= 3) join(id(p, q), id(p, 3));
                if (q_os && q == Q && Q >= 3) join(id(p, q), id(p, Q - 2));
            }
        // members of each group, the group ordered by class (highest first)
        std::vector<std::vector<int>> groups((size_t)P * Q);
        for (int cls = 2; cls >= 0; --cls)
            for (int q = 1; q <= Q; ++q)
                for (int p = 1; p <= P; ++p)
                    if (((p + q) & 1) == colour && cls_of(p, q) == cls) groups[root(id(p, q))].push_back(p | (q << 16));
        // FP64 lines share a radius's factors: its lines in a row (p slow, a
        // group where its least p belongs); FP32 ones take what runs with memory
        // (p fast)
        std::vector<std::vector<int>> at(pslow ? (size_t)P + 1 : 1);
        for (int g = 0; g < (int)groups.size(); ++g) {
            if (groups[g].empty()) continue;
            int least = pslow ? P : 0;
            if (pslow)
                for (int e : groups[g]) least = std::min(least, e & 0xffff);
            at[least].push_back(g);
        }
        size_t biggest = 0;
        for (const auto &g : groups) biggest = std::max(biggest, g.size());
        if ((int)biggest <= chunk) {
            const size_t before = lines.size();
            for (int multi = 1; multi >= 0; --multi)   // groups of several lines first, then single lines
                for (const auto &some : at)
                    for (int which : some) {
                        const auto &g = groups[which];
                        if ((g.size() > 1) != (multi == 1)) continue;
                        for (size_t t = 0; t < g.size(); ++t)
                            lines.push_back((int)((unsigned)g[t] | (t + 1 < g.size() ? R3_CONT : 0u)));
                    }
            if (lines.size() != before) off.push_back((int)lines.size());
        } else {
            for (int cls = 2; cls >= 0; --cls) {
                const size_t before = lines.size();
                for (int q = 1; q <= Q; ++q)
                    for (int p = 1; p <= P; ++p)
                        if (((p + q) & 1) == colour && cls_of(p, q) == cls) lines.push_back(p | (q << 16));
                if (lines.size() != before) off.push_back((int)lines.size());
            }
        }
    }
}

static int r3_create(const gb_r3d_params *p, const double *spacing, gb_r3d **out, int *nlev_out);

extern "C" int gb_r3d_create(const gb_r3d_params *p, gb_r3d **out, int *nlev_out)
{
    return r3_create(p, nullptr, out, nlev_out);
}

extern "C" int gb_r3d_create_spacing(const gb_r3d_params *p, double dr, double dz, double dp, gb_r3d **out,
                                     int *nlev_out)
{
    if (!(dr > 0.0 && dz > 0.0 && dp > 0.0)) {
        gb_set_error("gb_r3d_create_spacing: spacings must be positive");
        return GB_ERR_INVALID;
    }
    const double sp[3] = {dr, dz, dp};
    return r3_create(p, sp, out, nlev_out);
}

static int r3_create(const gb_r3d_params *p, const double *spacing, gb_r3d **out, int *nlev_out)
{
    if (!p || !out) { gb_set_error("gb_r3d_create: null argument"); return GB_ERR_INVALID; }
    *out = nullptr;
    const int nr = p->nr, nz = p->nz, np = p->np;
    const int nlev = r3_levels(nr, nz);
    if (nlev_out) *nlev_out = nlev;
    if (nr < 4 || nz < 4 || np < 4 || nr > 4096 || nz > 4096 || np > 16384 || np % (1 << nlev) != 0 ||
        np / (1 << (nlev - 1)) < 4 || !(p->r0 > 0.0 && p->rmax > p->r0) || !(p->zmax > 0.0) || !(p->dt > 0.0) ||
        p->Pr == 0.0 || (p->Re == 0.0 && p->variant != GB_R3D_HORIZONTAL) || p->nrel < 1 || p->maxsweeps < 1) {
        gb_set_error("gb_r3d_create: unsupported parameters (nr=%d nz=%d np=%d: nr, nz >= 4, np a multiple of 2^%d "
                     "with >= 4 phi intervals on the coarsest level; 0 < r0 < rmax, zmax, dt > 0, Pr != 0, Re != 0 "
                     "unless horizontal)",
                     nr, nz, np, nlev);
        return GB_ERR_INVALID;
    }
    if (p->smoother != GB_SMOOTHER_LEX && p->smoother != GB_SMOOTHER_ZEBRA) {
        gb_set_error("gb_r3d_create: unknown smoother %d", p->smoother);
        return GB_ERR_INVALID;
    }
    if (p->precision != GB_PRB_FP64 && p->precision != GB_PRB_MIXED) {
        gb_set_error("gb_r3d_create: unknown precision %d", p->precision);
        return GB_ERR_INVALID;
    }
    if (p->variant != GB_R3D_VERTICAL && p->variant != GB_R3D_HORIZONTAL) {
        gb_set_error("gb_r3d_create: unknown variant %d", p->variant);
        return GB_ERR_INVALID;
    }
    if (p->precision == GB_PRB_FP64 && np > R3_MAX_ROWS) {
        gb_set_error("gb_r3d_create: np=%d: an FP64 phi-line of more than %d rows does not fit a block's shared memory", np, R3_MAX_ROWS);
        return GB_ERR_INVALID;
    }
    if (p->variant == GB_R3D_HORIZONTAL && nz < 6) {
        gb_set_error("gb_r3d_create: the horizontal annulus's heat band j = nz/2-3..nz/2+3 needs nz >= 6 (nz=%d)", nz);
        return GB_ERR_INVALID;
    }
    gb_r3d *h = new gb_r3d();
    h->p = *p;
    R3Dev &d = h->dev;
    memset(&d, 0, sizeof(d));
    d.nr = nr;
    d.nz = nz;
    d.np = np;
    d.ni = nr + 2;
    d.nj = nz + 2;
    d.nk = np + 1;
    d.nlev = nlev;
    d.dt = p->dt;
    d.r0 = p->r0;
    d.rmax = p->rmax;
    d.zmax = p->zmax;
    d.Ra = p->Ra;
    d.Re = p->Re;
    d.Gr = p->Gr;
    d.Ptl = p->Pr;
    const double pi = acos(-1.0);
    d.dr = spacing ? spacing[0] : (p->rmax - p->r0) / (double)nr;
    d.dz = spacing ? spacing[1] : p->zmax / (double)nz;
    d.dp = spacing ? spacing[2] : 2.0 * pi / (double)np;
    d.nu_num = -p->r0 * log(p->r0 / p->rmax);
    d.nu_den = p->zmax * 2.0 * pi;
    d.horizontal = p->variant == GB_R3D_HORIZONTAL;
    if (d.horizontal) {
        // httrans1, httrans2 of rot3dmghor.f:264-267, host libm as the Fortran runtime
        d.nu_num = (double)nz / 6.0 * p->r0 * log(p->r0 / p->rmax);
        d.nu2_num = (double)nz / 6.0 * p->rmax * log(p->r0 / p->rmax);
    }
    d.tolcon = p->tolcon;
    d.sor = p->sor;
    d.nrel = p->nrel;
    d.maxsweeps = p->maxsweeps;
    const size_t fsz = (size_t)d.ni * d.nj * d.nk;
    cudaError_t e = cudaMalloc(&h->fields, sizeof(double) * fsz * GB_R_COUNT);
    if (e != cudaSuccess) { gb_set_error("gb_r3d_create: fields: %s", cudaGetErrorString(e)); delete h; return GB_ERR_ALLOC; }
    cudaMemset(h->fields, 0, sizeof(double) * fsz * GB_R_COUNT);
    for (int q = 0; q < GB_R_COUNT; ++q) d.fld[q] = h->fields + (size_t)q * fsz;

    // multigrid pool: per level rvc, rvv and the factor tables (shared by the
    // components); the work pool: per component and level v, f, res and their
    // FP32 twins
    std::vector<FacJob> jobs;
    size_t need = 0, wneed = 0;
    for (int l = 1; l <= nlev; ++l) {
        const int n1 = nr >> (l - 1), n2 = nz >> (l - 1), n3 = np >> (l - 1);
        const size_t sz = (size_t)(n1 + 1) * (n2 + 1) * (n3 + 1);
        wneed += 3 * (3 * sz + (3 * sz + 1) / 2 + 2);
        need += 6 * (size_t)(n1 + 2);
        size_t f32 = 3 * (4 * (size_t)(n1 + 1) + 4 * (size_t)(n2 + 1) + (size_t)(n1 + 4)) + 4;
        for (int comp = 1; comp <= 3; ++comp)
            for (int dir = 0; dir < 3; ++dir) {
                const int n = r3_len(comp, dir, n1, n2, n3);
                const int inst = dir == 0 ? 1 : r3_imax(comp, n1);
                need += (size_t)inst * r3_tabsize(r3_kind(comp, dir), n);
                f32 += (size_t)inst * r3_tabsize32(r3_kind(comp, dir), n) + 4;
            }
        need += (f32 + 1) / 2 + 2;
    }
    e = cudaMalloc(&h->pool, sizeof(double) * need);
    if (e != cudaSuccess) { gb_r3d_destroy(h); gb_set_error("gb_r3d_create: multigrid pool"); return GB_ERR_ALLOC; }
    cudaMemset(h->pool, 0, sizeof(double) * need);
    e = cudaMalloc(&h->work, sizeof(double) * wneed);
    if (e != cudaSuccess) { gb_r3d_destroy(h); gb_set_error("gb_r3d_create: multigrid work arrays"); return GB_ERR_ALLOC; }
    cudaMemset(h->work, 0, sizeof(double) * wneed);
    double *b = h->pool, *wb = h->work;
    std::vector<int> itab;
    struct TabRef { int l, comp, dir; size_t lines, off; int nphase; };
    std::vector<TabRef> refs;
    std::vector<double> rv_host;
    for (int l = 1; l <= nlev; ++l) {
        R3Lev &L = d.lev[l];
        L.n1 = nr >> (l - 1);
        L.n2 = nz >> (l - 1);
        L.n3 = np >> (l - 1);
        L.L1 = L.n1 + 1;
        L.L2 = L.n2 + 1;
        const int p2 = 1 << l;
        L.hr = d.dr * (double)p2 * 0.5;
        L.hz = d.dz * (double)p2 * 0.5;
        L.hp = d.dp * (double)p2 * 0.5;
        L.hhr = L.hr * L.hr;
        L.hhz = L.hz * L.hz;
        L.hhp = L.hp * L.hp;
        L.ihr = 1.0 / L.hr;
        L.ihhr = 1.0 / L.hhr;
        L.ihhz = 1.0 / L.hhz;
        L.ihhp = 1.0 / L.hhp;
        const size_t sz = (size_t)L.L1 * L.L2 * (L.n3 + 1);
        for (int comp = 1; comp <= 3; ++comp) {
            R3Work &W = d.work[comp][l];
            W.v = wb; wb += sz;
            W.f = wb; wb += sz;
            W.res = wb; wb += sz;
            float *fw = (float *)wb;
            W.v32 = fw; fw += sz;
            W.f32 = fw; fw += sz;
            W.res32 = fw; fw += sz;
            wb = (double *)(((uintptr_t)fw + 15) & ~(uintptr_t)15);
        }
        L.rvc = b; b += L.n1 + 2;
        L.rvv = b; b += L.n1 + 2;
        L.dirc = b; b += L.n1 + 2;
        L.dirv = b; b += L.n1 + 2;
        L.diqc = b; b += L.n1 + 2;
        L.diqv = b; b += L.n1 + 2;
        const size_t m = (size_t)L.n1 + 2;
        rv_host.assign(6 * m, 0.0);
        for (int i = 0; i <= L.n1 + 1; ++i) {
            const double rc = d.r0 + ((double)i - 0.5) * L.hr, rv = (double)i * L.hr + d.r0;
            rv_host[i] = rc;
            rv_host[m + i] = rv;
            rv_host[2 * m + i] = 1.0 / rc;
            rv_host[3 * m + i] = 1.0 / rv;
            rv_host[4 * m + i] = 1.0 / (rc * rc);
            rv_host[5 * m + i] = 1.0 / (rv * rv);
        }
        cudaMemcpy(L.rvc, rv_host.data(), sizeof(double) * rv_host.size(), cudaMemcpyHostToDevice);
        for (int comp = 1; comp <= 3; ++comp)
            for (int dir = 0; dir < 3; ++dir) {
                const int kind = r3_kind(comp, dir);
                const int n = r3_len(comp, dir, L.n1, L.n2, L.n3);
                const int inst = dir == 0 ? 1 : r3_imax(comp, L.n1);
                L.fac[comp][dir] = b;
                for (int q = 0; q < inst; ++q) jobs.push_back({l, comp, dir, dir == 0 ? 0 : q + 1, b + (size_t)q * r3_tabsize(kind, n)});
                b += (size_t)inst * r3_tabsize(kind, n);
                std::vector<int> lines, off;
                r3_phases(p->smoother, p->precision == GB_PRB_FP64, comp, dir, L.n1, L.n2, L.n3, lines, off);
                TabRef tr;
                tr.l = l;
                tr.comp = comp;
                tr.dir = dir;
                tr.lines = itab.size();
                itab.insert(itab.end(), lines.begin(), lines.end());
                tr.off = itab.size();
                itab.insert(itab.end(), off.begin(), off.end());
                tr.nphase = (int)off.size() - 1;
                refs.push_back(tr);
            }
        // FP32 storage of the level
        {
            float *fb = (float *)b;
            fb = (float *)(((uintptr_t)fb + 15) & ~(uintptr_t)15);
            for (int comp = 1; comp <= 3; ++comp) {
                L.wi[comp] = (float4 *)fb; fb += 4 * (L.n1 + 1);
                L.wj[comp] = (float4 *)fb; fb += 4 * (L.n2 + 1);
                L.wp[comp] = fb; fb += (L.n1 + 4) & ~3;
            }
            for (int comp = 1; comp <= 3; ++comp)
                for (int dir = 0; dir < 3; ++dir) {
                    const int n = r3_len(comp, dir, L.n1, L.n2, L.n3);
                    const int inst = dir == 0 ? 1 : r3_imax(comp, L.n1);
                    fb = (float *)(((uintptr_t)fb + 15) & ~(uintptr_t)15);   // copied 16 bytes at a time
                    L.fac32[comp][dir] = fb;
                    fb += (size_t)inst * r3_tabsize32(r3_kind(comp, dir), n);
                }
            b = (double *)(((uintptr_t)fb + 15) & ~(uintptr_t)15);
        }
    }
    if ((size_t)(b - h->pool) > need || (size_t)(wb - h->work) > wneed) {
        gb_r3d_destroy(h);
        gb_set_error("gb_r3d_create: multigrid pool layout mismatch");
        return GB_ERR_CUDA;
    }
    e = cudaMalloc(&h->itab, sizeof(int) * itab.size());
    if (e != cudaSuccess) { gb_r3d_destroy(h); gb_set_error("gb_r3d_create: phase tables"); return GB_ERR_ALLOC; }
    cudaMemcpy(h->itab, itab.data(), sizeof(int) * itab.size(), cudaMemcpyHostToDevice);
    for (const TabRef &tr : refs) {
        R3Lev &L = d.lev[tr.l];
        L.lines[tr.comp][tr.dir] = h->itab + tr.lines;
        L.poff[tr.comp][tr.dir] = h->itab + tr.off;
        L.nphase[tr.comp][tr.dir] = tr.nphase;
    }
    // sin and cos of theta = 6.283185307/np k (rot3dmghor.f:373-378), host libm
    {
        std::vector<double> tab(2 * (size_t)(np + 1), 0.0);
        if (d.horizontal)
            for (int k = 0; k <= np; ++k) {
                const double theta = 6.283185307 / (double)np * (double)k;
                tab[k] = sin(theta);
                tab[np + 1 + k] = cos(theta);
            }
        e = cudaMalloc(&h->tables, sizeof(double) * tab.size());
        if (e != cudaSuccess) { gb_r3d_destroy(h); gb_set_error("gb_r3d_create: tables"); return GB_ERR_ALLOC; }
        cudaMemcpy(h->tables, tab.data(), sizeof(double) * tab.size(), cudaMemcpyHostToDevice);
        d.sinth = h->tables;
        d.costh = h->tables + np + 1;
    }
    // small state
    e = cudaMalloc(&h->small, 4096 + 2 * sizeof(double) * (size_t)(np + 2));
    if (e != cudaSuccess) { gb_r3d_destroy(h); gb_set_error("gb_r3d_create: state"); return GB_ERR_ALLOC; }
    cudaMemset(h->small, 0, 4096 + 2 * sizeof(double) * (size_t)(np + 2));
    char *sm = (char *)h->small;
    d.resmax = (unsigned long long *)(sm + 0);    // 8 slots
    d.nanflag = (int *)(sm + 64);                 // 8 slots
    d.abort = (int *)(sm + 128);
    d.steps_done = (int *)(sm + 192);
    d.solve_status = (int *)(sm + 256);           // 4 slots
    d.solve_sweeps = (int *)(sm + 320);           // 4 slots
    h->sync = (unsigned *)(sm + 512);             // 4 barriers, 128 bytes apart
    d.trans = (double *)(sm + 4096);
    d.trans2 = d.trans + (np + 2);
    for (int c = 0; c < 4; ++c) {
        d.gs[c].count = (unsigned long long *)(h->sync + R3_SYNC_STRIDE * c);
        d.gs[c].err = (int *)(h->sync + R3_SYNC_STRIDE * c + 2);
        d.gs[c].limit = GB_GRID_WAIT_LIMIT_DEFAULT;
        d.gs[c].tally = (unsigned long long *)(sm + 448) + c;   // 4 counters, one per component
    }
    // factor tables
    FacJob *djobs = nullptr;
    e = cudaMalloc(&djobs, sizeof(FacJob) * jobs.size());
    if (e != cudaSuccess) { gb_r3d_destroy(h); gb_set_error("gb_r3d_create: factor jobs"); return GB_ERR_ALLOC; }
    cudaMemcpy(djobs, jobs.data(), sizeof(FacJob) * jobs.size(), cudaMemcpyHostToDevice);
    {
        const int wstride = 7 * std::max(nr, std::max(nz, np));
        double *work = nullptr;
        e = cudaMalloc(&work, sizeof(double) * (size_t)wstride * jobs.size());
        if (e != cudaSuccess) { cudaFree(djobs); gb_r3d_destroy(h); gb_set_error("gb_r3d_create: factor scratch"); return GB_ERR_ALLOC; }
        k_r3d_factors<<<gb_ceil_div(jobs.size(), 64), 64>>>(d, djobs, (int)jobs.size(), work, wstride);
        if (p->precision == GB_PRB_MIXED) {
            k_r3d_factors32<<<gb_ceil_div(jobs.size(), 64), 64>>>(d, djobs, (int)jobs.size());
            k_r3d_steps32<<<dim3(nlev, 3, 2), 128>>>(d);
            k_r3d_weights32<<<dim3(nlev, 3), 128>>>(d);
        }
        cudaDeviceSynchronize();
        cudaFree(work);
    }
    e = cudaDeviceSynchronize();
    cudaFree(djobs);
    if (e != cudaSuccess) { gb_set_error("gb_r3d_create: factors: %s", cudaGetErrorString(e)); gb_r3d_destroy(h); return GB_ERR_CUDA; }
    // cooperative grid: every block resident
    int dev = 0, sms = 0, coop = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    int worst = 1 << 30;
    const void *kerns[6] = {(const void *)k_r3d_solve<1>, (const void *)k_r3d_solve<2>, (const void *)k_r3d_solve<3>,
                            (const void *)k_r3d_solve_mixed<1>, (const void *)k_r3d_solve_mixed<2>,
                            (const void *)k_r3d_solve_mixed<3>};
    for (int q = 0; q < 6; ++q) {
        cudaFuncSetAttribute(kerns[q], cudaFuncAttributeMaxDynamicSharedMemorySize, R3_SMEM_BYTES);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kerns[q], R3_THREADS, R3_SMEM_BYTES);
        worst = std::min(worst, per_sm);
    }
    if (!coop || worst < 1) {
        gb_r3d_destroy(h);
        gb_set_error("gb_r3d_create: cooperative launch unavailable (coop=%d, blocks/SM=%d)", coop, worst);
        return GB_ERR_CUDA;
    }
    h->grid = sms * std::min(worst, 2);
    e = cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&h->side, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&h->ev_fork, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&h->ev_join, cudaEventDisableTiming);
    if (e != cudaSuccess) { gb_r3d_destroy(h); gb_set_error("gb_r3d_create: streams"); return GB_ERR_CUDA; }
    *out = h;
    return GB_OK;
}

extern "C" void *gb_r3d_stream(gb_r3d *h) { return h ? (void *)h->stream : nullptr; }

extern "C" int gb_r3d_barrier_counts(gb_r3d *h, unsigned long long *counts, int *blocks, int reset)
{
    if (!h) { gb_set_error("gb_r3d_barrier_counts: null context"); return GB_ERR_INVALID; }
    GB_CUDA_TRY(cudaStreamSynchronize(h->side));
    GB_CUDA_TRY(cudaStreamSynchronize(h->stream));
    unsigned long long c[4] = {0, 0, 0, 0};
    GB_CUDA_TRY(cudaMemcpy(c, h->dev.gs[0].tally, sizeof(c), cudaMemcpyDeviceToHost));
    if (counts)
        for (int i = 0; i < 3; ++i) counts[i] = c[i + 1];
    if (blocks) *blocks = h->grid;
    if (reset) GB_CUDA_TRY(cudaMemset(h->dev.gs[0].tally, 0, sizeof(c)));
    return GB_OK;
}

extern "C" int gb_r3d_set_wait_limit(gb_r3d *h, long long polls)
{
    if (!h || polls < 0) {
        gb_set_error("gb_r3d_set_wait_limit: need a context and polls >= 0");
        return GB_ERR_INVALID;
    }
    for (int c = 0; c < 4; ++c) h->dev.gs[c].limit = polls;
    return GB_OK;
}

static int r3_io(gb_r3d *h, int field, double *host, int ld1, int ld2, bool to_dev)
{
    if (!h || !host || field < 0 || field >= GB_R_COUNT || ld1 < h->dev.ni || ld2 < h->dev.nj) {
        gb_set_error("gb_r3d_%s_field: invalid argument", to_dev ? "set" : "get");
        return GB_ERR_INVALID;
    }
    const R3Dev &d = h->dev;
    cudaMemcpy3DParms m;
    memset(&m, 0, sizeof(m));
    cudaPitchedPtr hp = make_cudaPitchedPtr(host, sizeof(double) * (size_t)ld1, (size_t)d.ni, (size_t)ld2);
    cudaPitchedPtr dp = make_cudaPitchedPtr(d.fld[field], sizeof(double) * (size_t)d.ni, (size_t)d.ni, (size_t)d.nj);
    m.srcPtr = to_dev ? hp : dp;
    m.dstPtr = to_dev ? dp : hp;
    m.extent = make_cudaExtent(sizeof(double) * (size_t)d.ni, (size_t)d.nj, (size_t)d.nk);
    m.kind = to_dev ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost;
    GB_CUDA_TRY(cudaMemcpy3DAsync(&m, h->stream));
    GB_CUDA_TRY(cudaStreamSynchronize(h->stream));
    return GB_OK;
}

extern "C" int gb_r3d_set_field(gb_r3d *h, int field, const double *host, int ld1, int ld2)
{
    return r3_io(h, field, (double *)host, ld1, ld2, true);
}

extern "C" int gb_r3d_get_field(gb_r3d *h, int field, double *host, int ld1, int ld2)
{
    return r3_io(h, field, host, ld1, ld2, false);
}

static const int R3_TPB = 256;

static void r3_launch_transport(gb_r3d *h, int what, int step, cudaStream_t s)
{
    const R3Dev &d = h->dev;
    const long long nr = d.nr, nz = d.nz, npp = d.np + 1;
    switch (what) {
    case 0: k_r3d_avort<<<gb_ceil_div(nr * (nz - 1) * npp, R3_TPB), R3_TPB, 0, s>>>(d); break;
    case 1: k_r3d_bvort<<<gb_ceil_div((nr - 1) * (nz - 1) * npp, R3_TPB), R3_TPB, 0, s>>>(d); break;
    case 2: k_r3d_cvort<<<gb_ceil_div((nr - 1) * nz * npp, R3_TPB), R3_TPB, 0, s>>>(d); break;
    case 3: k_r3d_temp<<<gb_ceil_div(nr * (nz + 2) * npp, R3_TPB), R3_TPB, 0, s>>>(d); break;
    case 4:
        k_r3d_heat_k<<<gb_ceil_div(d.np, 128), 128, 0, s>>>(d);
        k_r3d_heat_sum<<<1, 32, 0, s>>>(d, step);
        break;
    case 5: k_r3d_rhs<1><<<gb_ceil_div(nr * (nz - 1) * npp, R3_TPB), R3_TPB, 0, s>>>(d); break;
    case 6: k_r3d_rhs<2><<<gb_ceil_div(nr * nz * npp, R3_TPB), R3_TPB, 0, s>>>(d); break;
    case 7: k_r3d_rhs<3><<<gb_ceil_div((nr - 1) * nz * npp, R3_TPB), R3_TPB, 0, s>>>(d); break;
    case 8: k_r3d_update<<<gb_ceil_div((long long)d.ni * d.nj * d.nk, R3_TPB), R3_TPB, 0, s>>>(d, step); break;
    }
}

// One component's solve on `grid` blocks (at most h->grid, all resident).
// The w and v solves of a step run side by side on half the blocks each:
// their blocks together never exceed the resident capacity, and each waits
// only at its own barrier.
static int r3_launch_solve(gb_r3d *h, int comp, int step, cudaStream_t s, int grid)
{
    GB_CUDA_TRY(cudaMemsetAsync(h->sync + R3_SYNC_STRIDE * comp, 0, sizeof(unsigned) * 4, s));
    GB_CUDA_TRY(cudaMemsetAsync(h->dev.resmax + 2 * comp, 0, sizeof(unsigned long long) * 2, s));
    GB_CUDA_TRY(cudaMemsetAsync(h->dev.nanflag + 2 * comp, 0, sizeof(int) * 2, s));
    R3Dev D = h->dev;
    void *args[] = {&D, &step};
    const bool mixed = h->p.precision == GB_PRB_MIXED;
    const void *k = comp == 1   ? (mixed ? (const void *)k_r3d_solve_mixed<1> : (const void *)k_r3d_solve<1>)
                    : comp == 2 ? (mixed ? (const void *)k_r3d_solve_mixed<2> : (const void *)k_r3d_solve<2>)
                                : (mixed ? (const void *)k_r3d_solve_mixed<3> : (const void *)k_r3d_solve<3>);
    cudaError_t e = cudaLaunchCooperativeKernel(k, grid, R3_THREADS, args, R3_SMEM_BYTES, s);
    if (e != cudaSuccess) {
        gb_set_error("gb_r3d: cooperative solve launch (%d blocks): %s", grid, cudaGetErrorString(e));
        return GB_ERR_CUDA;
    }
    return GB_OK;
}

static int r3_sync(gb_r3d *h, const char *what)
{
    cudaError_t e = cudaStreamSynchronize(h->side);
    if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
    if (e != cudaSuccess) { gb_set_error("%s: %s", what, cudaGetErrorString(e)); return GB_ERR_CUDA; }
    unsigned sy[4 * R3_SYNC_STRIDE];
    GB_CUDA_TRY(cudaMemcpy(sy, h->sync, sizeof(sy), cudaMemcpyDeviceToHost));
    for (int c = 1; c <= 3; ++c)
        if (sy[R3_SYNC_STRIDE * c + 2]) {
            gb_set_error("%s: a grid barrier wait timed out (component %d)", what, c);
            return GB_TIMEOUT;
        }
    return GB_OK;
}

static void r3_clear_abort(gb_r3d *h) { cudaMemsetAsync(h->dev.abort, 0, sizeof(int), h->stream); }

#define R3_ROUTINE(name, what)                                  \
    extern "C" int gb_r3d_##name(gb_r3d *h)                     \
    {                                                           \
        if (!h) return GB_ERR_INVALID;                          \
        r3_clear_abort(h);                                      \
        r3_launch_transport(h, what, -1, h->stream);            \
        return r3_sync(h, "gb_r3d_" #name);                     \
    }
R3_ROUTINE(avorticity, 0)
R3_ROUTINE(bvorticity, 1)
R3_ROUTINE(cvorticity, 2)
R3_ROUTINE(temperature, 3)
R3_ROUTINE(rhsw, 5)
R3_ROUTINE(rhsv, 6)
R3_ROUTINE(rhsu, 7)
R3_ROUTINE(update, 8)
#undef R3_ROUTINE

extern "C" int gb_r3d_heat(gb_r3d *h, double *trans1)
{
    if (!h) return GB_ERR_INVALID;
    r3_clear_abort(h);
    r3_launch_transport(h, 4, -1, h->stream);
    int st = r3_sync(h, "gb_r3d_heat");
    if (st != GB_OK) return st;
    if (trans1) GB_CUDA_TRY(cudaMemcpy(trans1, h->dev.trans, sizeof(double), cudaMemcpyDeviceToHost));
    return GB_OK;
}

extern "C" int gb_r3d_heat2(gb_r3d *h, double *trans1, double *trans2)
{
    if (!h) return GB_ERR_INVALID;
    r3_clear_abort(h);
    r3_launch_transport(h, 4, -1, h->stream);
    int st = r3_sync(h, "gb_r3d_heat2");
    if (st != GB_OK) return st;
    if (trans1) GB_CUDA_TRY(cudaMemcpy(trans1, h->dev.trans, sizeof(double), cudaMemcpyDeviceToHost));
    if (trans2) GB_CUDA_TRY(cudaMemcpy(trans2, h->dev.trans2, sizeof(double), cudaMemcpyDeviceToHost));
    return GB_OK;
}

extern "C" int gb_r3d_nu2(gb_r3d *h, int nsteps, double *nu2)
{
    if (!h || nsteps < 0 || nsteps > h->hist_cap || (nsteps > 0 && !nu2)) {
        gb_set_error("gb_r3d_nu2: invalid argument");
        return GB_ERR_INVALID;
    }
    if (nsteps > 0)
        GB_CUDA_TRY(cudaMemcpy(nu2, h->hist_nu + h->hist_cap, sizeof(double) * (size_t)nsteps, cudaMemcpyDeviceToHost));
    return GB_OK;
}

extern "C" int gb_r3d_poisson(gb_r3d *h, int which, int *sweeps)
{
    if (!h || which < 1 || which > 3) { gb_set_error("gb_r3d_poisson: invalid argument"); return GB_ERR_INVALID; }
    r3_clear_abort(h);
    int st = r3_launch_solve(h, which, -1, h->stream, h->grid);
    if (st != GB_OK) return st;
    st = r3_sync(h, "gb_r3d_poisson");
    if (st != GB_OK) return st;
    int out[2] = {0, 0};
    GB_CUDA_TRY(cudaMemcpy(&out[0], h->dev.solve_status + which, sizeof(int), cudaMemcpyDeviceToHost));
    GB_CUDA_TRY(cudaMemcpy(&out[1], h->dev.solve_sweeps + which, sizeof(int), cudaMemcpyDeviceToHost));
    if (sweeps) *sweeps = out[1];
    return out[0];
}

extern "C" int gb_r3d_step(gb_r3d *h, int nsteps, double *nu, int *sweeps, int *steps_done)
{
    if (!h || nsteps < 0) { gb_set_error("gb_r3d_step: invalid argument"); return GB_ERR_INVALID; }
    if (steps_done) *steps_done = 0;
    if (nsteps == 0) return GB_OK;
    if (nsteps > h->hist_cap) {
        cudaFree(h->hist_nu);
        cudaFree(h->hist_sw);
        h->hist_nu = nullptr;
        h->hist_sw = nullptr;
        h->hist_cap = 0;
        GB_CUDA_TRY(cudaMalloc(&h->hist_nu, 2 * sizeof(double) * (size_t)nsteps));
        GB_CUDA_TRY(cudaMalloc(&h->hist_sw, sizeof(int) * 3 * (size_t)nsteps));
        h->hist_cap = nsteps;
    }
    h->dev.hist_nu = h->hist_nu;
    h->dev.hist_nu2 = h->hist_nu + h->hist_cap;
    h->dev.hist_sw = h->hist_sw;
    cudaStream_t s = h->stream;
    GB_CUDA_TRY(cudaMemsetAsync(h->hist_sw, 0, sizeof(int) * 3 * (size_t)nsteps, s));
    GB_CUDA_TRY(cudaMemsetAsync(h->hist_nu, 0, 2 * sizeof(double) * (size_t)h->hist_cap, s));
    GB_CUDA_TRY(cudaMemsetAsync(h->dev.steps_done, 0, sizeof(int), s));
    GB_CUDA_TRY(cudaMemsetAsync(h->dev.abort, 0, sizeof(int), s));
    for (int step = 0; step < nsteps; ++step) {
        r3_launch_transport(h, 0, step, s);
        r3_launch_transport(h, 1, step, s);
        r3_launch_transport(h, 2, step, s);
        r3_launch_transport(h, 3, step, s);
        r3_launch_transport(h, 4, step, s);
        r3_launch_transport(h, 5, step, s);
        // rhsv reads An and Cn only, and the w and v solves touch disjoint
        // fields: the v solve runs beside the w solve, on the side stream
        GB_CUDA_TRY(cudaEventRecord(h->ev_fork, s));
        GB_CUDA_TRY(cudaStreamWaitEvent(h->side, h->ev_fork, 0));
        const int half = std::max(1, h->grid / 2);
        int st = r3_launch_solve(h, 1, step, s, half);
        if (st == GB_OK) {
            r3_launch_transport(h, 6, step, h->side);
            st = r3_launch_solve(h, 2, step, h->side, h->grid - half);
        }
        if (st == GB_OK) {
            GB_CUDA_TRY(cudaEventRecord(h->ev_join, h->side));
            GB_CUDA_TRY(cudaStreamWaitEvent(s, h->ev_join, 0));
            r3_launch_transport(h, 7, step, s);
            st = r3_launch_solve(h, 3, step, s, h->grid);
        }
        if (st != GB_OK) return st;
        r3_launch_transport(h, 8, step, s);
    }
    int st = r3_sync(h, "gb_r3d_step");
    if (st != GB_OK) return st;
    int done = 0, ab = 0;
    GB_CUDA_TRY(cudaMemcpy(&done, h->dev.steps_done, sizeof(int), cudaMemcpyDeviceToHost));
    GB_CUDA_TRY(cudaMemcpy(&ab, h->dev.abort, sizeof(int), cudaMemcpyDeviceToHost));
    if (steps_done) *steps_done = done;
    if (nu && done > 0) GB_CUDA_TRY(cudaMemcpy(nu, h->hist_nu, sizeof(double) * (size_t)done, cudaMemcpyDeviceToHost));
    if (sweeps) {
        const int n = std::min(nsteps, done + 1);
        GB_CUDA_TRY(cudaMemcpy(sweeps, h->hist_sw, sizeof(int) * 3 * (size_t)n, cudaMemcpyDeviceToHost));
    }
    return ab ? ab : GB_OK;
}
