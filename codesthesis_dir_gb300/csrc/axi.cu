// Axisymmetric rotating annulus in the (r, z) meridional plane (rotann2.f,
// "AXI") on the device: Dufort-Frankel vorticity, swirl-velocity and
// temperature updates with the Arakawa Jacobian, Thom wall vorticity, the
// inner-wall heat flux, and the streamfunction multigrid.
//
// Numerics: every expression keeps the reference's operation order and the
// translation unit is compiled with -fmad=false, so the FP64 path is
// bit-identical to the reference algorithm (and to the C oracle).
//
// Layout: each field is a column-major (0:ld-1, 0:nz) array with ld = nr+1,
// the ten fields of an instance in one allocation.  The multigrid keeps the
// packed v / f slots per level, one residual array, the factored r-line
// matrix (one per level: its coefficients vary with r only) and one factored
// z-line matrix per r-row (its diagonal holds -1/r^2).
//
// The multigrid solve is one launch of one cluster of CTAs (cluster.cuh): the
// sweep loop, every level and the convergence test run in it.  LEX orders the
// lines as the reference does (rows j = 1..n2-1, then columns i = 1..n1-1,
// rotann2.f:698-725), one line after the other; ZEBRA solves odd lines, then
// even lines.  Mixed precision runs its FP32 cycles in the cluster's shared
// memory where they fit (meridian.cu).
#include <math.h>
#include <stdint.h>
#include <string.h>

#include <vector>

#include <algorithm>

#include "banded.cuh"
#include "cluster.cuh"
#include "gbcommon.cuh"
#include "meridian.cuh"
#include "str_internal.cuh"
#include "warpline.cuh"

#define AXI_THREADS 256
#define AXI_MAXLEV 8
#define AX(i, j) ((size_t)(i) + (size_t)ld * (size_t)(j))

struct AxiLevel {
    int n1, n2, lf;           // sizes; lf = 2^l / 2 scales i into rval
    double hr, hz, hhr, hhz;
    double ihr, ihhr, ihhz;   // their reciprocals (IEEE)
    double *v, *f;            // packed (n1+1)*(n2+1)
    double *fac_r;            // r-line factors, tdma_fac_len(n1-1)
    double *fac_z;            // z-line factors, tdma_fac_len(n2-1) for each i = 1..n1-1
    // mixed precision: FP32 correction cycle (line tables, warpline.cuh)
    float *v32, *f32, *fac_r32, *fac_z32;
};

// Stretched grid (gb_axi_create_stretched): level-1 positions, grid.f's
// finite-difference weights and the inner-wall d/dr weights of the heat flux.
struct AxsTab {
    const double *r, *z;      // r(0..nr), z(0..nz)
    const double *cr, *crr;   // rows i = 1..nr-1: [3(i-1) + k], [4(i-1) + k]
    const double *cz, *czz;   // rows j = 1..nz-1: [3(j-1) + k], [4(j-1) + k]
    double hw[5];             // d/dr at r(0) on r(0..4)
};

struct AxiDev {
    int nr, nz, ld, nlev, mode, maxsweeps, nrel;
    int stretched;            // 1: the transport uses st (and the stretched multigrid)
    AxsTab st;
    double dt, dr, dz, r0, rmax, zmax, Ra, Re, Ptl;
    double cf1, cf2, cf3, cf4, tolcon;
    double *f[GB_A_COUNT];
    double *rval;             // rotann2.f:626: rval(i) = i hr(1) + r0
    double *irv, *irq;        // 1/rval and 1/(rval rval) (IEEE)
    double *rc;               // the residual of the level it was last formed on, pitch n1 + 1
    float *rc32, *rval32;
    AxiLevel lev[AXI_MAXLEV];
    double *heat;
    unsigned long long *errmax;   // bit patterns of the step's max |x - x_p|, x = omega, v, T
    int *abort;               // 1: a solve failed; 2: the run reached the steady state
    int *status;              // [0] poisson status, [1] sweeps
    int *step_index;
    double *nu_hist;
    int *sweep_hist;
    int hist_cap;
    double nu_c, nu_d;        // httrans = trans * nu_c / nu_d
};

// ---------------------------------------------------------------------------
// Transport
// ---------------------------------------------------------------------------

// arakawa, rotann2.f:432-459, at one interior point.
__device__ __forceinline__ double arakawa_at(const double *psi, const double *th, int ld, int i, int j, double hx,
                                             double hy)
{
    const int ip = i + 1, im = i - 1;
    const double a = (psi[AX(ip, j)] - psi[AX(im, j)]) * (th[AX(i, j + 1)] - th[AX(i, j - 1)]) -
                     (psi[AX(i, j + 1)] - psi[AX(i, j - 1)]) * (th[AX(ip, j)] - th[AX(im, j)]) +
                     psi[AX(ip, j)] * (th[AX(ip, j + 1)] - th[AX(ip, j - 1)]) -
                     psi[AX(im, j)] * (th[AX(im, j + 1)] - th[AX(im, j - 1)]) -
                     psi[AX(i, j + 1)] * (th[AX(ip, j + 1)] - th[AX(im, j + 1)]) +
                     psi[AX(i, j - 1)] * (th[AX(ip, j - 1)] - th[AX(im, j - 1)]) +
                     th[AX(i, j + 1)] * (psi[AX(ip, j + 1)] - psi[AX(im, j + 1)]) -
                     th[AX(i, j - 1)] * (psi[AX(ip, j - 1)] - psi[AX(im, j - 1)]) -
                     th[AX(ip, j)] * (psi[AX(ip, j + 1)] - psi[AX(ip, j - 1)]) +
                     th[AX(im, j)] * (psi[AX(im, j + 1)] - psi[AX(im, j - 1)]);
    return a / (12.0 * hx * hy);
}

// ---------------------------------------------------------------------------
// Stretched-grid forms: every derivative of rotann2.f's transport taken with
// grid.f's weights, each sum in the order written here (the oracle's
// orc_axi_set_stretched states them and performs the same operations).
// ---------------------------------------------------------------------------
#define SCR(i, k) T.cr[3 * ((i) - 1) + (k) - 1]
#define SCRR(i, k) T.crr[4 * ((i) - 1) + (k) - 1]
#define SCZ(j, k) T.cz[3 * ((j) - 1) + (k) - 1]
#define SCZZ(j, k) T.czz[4 * ((j) - 1) + (k) - 1]

__device__ __forceinline__ double axs_dr_off(const AxsTab &T, const double *x, int ld, int i, int j)
{
    return SCR(i, 1) * x[AX(i - 1, j)] + SCR(i, 3) * x[AX(i + 1, j)];
}
__device__ __forceinline__ double axs_drr_off(const AxsTab &T, const double *x, int ld, int i, int j, int nr)
{
    if (i <= nr / 2) return SCRR(i, 1) * x[AX(i - 1, j)] + SCRR(i, 3) * x[AX(i + 1, j)] + SCRR(i, 4) * x[AX(i + 2, j)];
    return SCRR(i, 1) * x[AX(i - 2, j)] + SCRR(i, 2) * x[AX(i - 1, j)] + SCRR(i, 4) * x[AX(i + 1, j)];
}
__device__ __forceinline__ double axs_crrc(const AxsTab &T, int i, int nr) { return i <= nr / 2 ? SCRR(i, 2) : SCRR(i, 3); }
__device__ __forceinline__ double axs_dz(const AxsTab &T, const double *x, int ld, int i, int j)
{
    return SCZ(j, 1) * x[AX(i, j - 1)] + SCZ(j, 2) * x[AX(i, j)] + SCZ(j, 3) * x[AX(i, j + 1)];
}
__device__ __forceinline__ double axs_dzz_off(const AxsTab &T, const double *x, int ld, int i, int j, int nz)
{
    if (j <= nz / 2) return SCZZ(j, 1) * x[AX(i, j - 1)] + SCZZ(j, 3) * x[AX(i, j + 1)] + SCZZ(j, 4) * x[AX(i, j + 2)];
    return SCZZ(j, 1) * x[AX(i, j - 2)] + SCZZ(j, 2) * x[AX(i, j - 1)] + SCZZ(j, 4) * x[AX(i, j + 1)];
}
__device__ __forceinline__ double axs_czzc(const AxsTab &T, int j, int nz) { return j <= nz / 2 ? SCZZ(j, 2) : SCZZ(j, 3); }

// the Arakawa sum over the local metric 3 (r(i+1) - r(i-1)) (z(j+1) - z(j-1))
__device__ __forceinline__ double axs_arakawa(const AxsTab &T, const double *psi, const double *th, int ld, int i, int j)
{
    const int ip = i + 1, im = i - 1;
    const double a = (psi[AX(ip, j)] - psi[AX(im, j)]) * (th[AX(i, j + 1)] - th[AX(i, j - 1)]) -
                     (psi[AX(i, j + 1)] - psi[AX(i, j - 1)]) * (th[AX(ip, j)] - th[AX(im, j)]) +
                     psi[AX(ip, j)] * (th[AX(ip, j + 1)] - th[AX(ip, j - 1)]) -
                     psi[AX(im, j)] * (th[AX(im, j + 1)] - th[AX(im, j - 1)]) -
                     psi[AX(i, j + 1)] * (th[AX(ip, j + 1)] - th[AX(im, j + 1)]) +
                     psi[AX(i, j - 1)] * (th[AX(ip, j - 1)] - th[AX(im, j - 1)]) +
                     th[AX(i, j + 1)] * (psi[AX(ip, j + 1)] - psi[AX(im, j + 1)]) -
                     th[AX(i, j - 1)] * (psi[AX(ip, j - 1)] - psi[AX(im, j - 1)]) -
                     th[AX(ip, j)] * (psi[AX(ip, j + 1)] - psi[AX(ip, j - 1)]) +
                     th[AX(im, j)] * (psi[AX(im, j + 1)] - psi[AX(im, j - 1)]);
    return a / (3.0 * (T.r[ip] - T.r[im]) * (T.z[j + 1] - T.z[j - 1]));
}

// vorticity and velocity of the stretched state at interior point (i, j)
__device__ __forceinline__ void axs_vort_vel_at(const AxiDev &d, int what, int i, int j)
{
    const AxsTab &T = d.st;
    const int ld = d.ld, nr = d.nr, nz = d.nz;
    const double Ptl = d.Ptl, Ra = d.Ra, Re = d.Re, dt = d.dt;
    const double *phi = d.f[GB_A_phi], *omeg = d.f[GB_A_omeg], *vel = d.f[GB_A_vel], *theta = d.f[GB_A_theta];
    const double RRP = Ra / Re / Ptl;
    const double r = T.r[i];
    const double sigma = axs_crrc(T, i, nr) + SCR(i, 2) / r + axs_czzc(T, j, nz);
    const double A = 1.0 / (2.0 * Ptl * dt) - sigma / 2.0 + 1.0 / (2.0 * (r * r));
    const double AA = 1.0 / (2.0 * Ptl * dt) + sigma / 2.0 - 1.0 / (2.0 * (r * r));
    const double dz_phi = axs_dz(T, phi, ld, i, j), dz_v = axs_dz(T, vel, ld, i, j);
    if (what & 1) {
        const double arak = axs_arakawa(T, phi, omeg, ld, i, j);
        const double dz_om = axs_dz(T, omeg, ld, i, j), dz_th = axs_dz(T, theta, ld, i, j);
        const double B = (phi[AX(i, j)] * dz_om + omeg[AX(i, j)] * dz_phi) / (Ptl * r);
        const double C = 2.0 * vel[AX(i, j)] * dz_v / (Ptl * r);
        const double D = 2.0 * Re * dz_v;
        const double E = r * Ra * dz_th;
        const double EE = 2.0 * RRP * vel[AX(i, j)] * dz_th + 2.0 * RRP * theta[AX(i, j)] * dz_v;
        const double F = axs_drr_off(T, omeg, ld, i, j, nr);
        const double G = axs_dr_off(T, omeg, ld, i, j) / r;
        const double H = axs_dzz_off(T, omeg, ld, i, j, nz);
        d.f[GB_A_omegn][AX(i, j)] = (AA * d.f[GB_A_omegp][AX(i, j)] + arak / Ptl + B + C + D - E - EE + F + G + H) / A;
    }
    if (what & 2) {
        const double arak = axs_arakawa(T, phi, vel, ld, i, j);
        const double B = (vel[AX(i, j)] * dz_phi - phi[AX(i, j)] * dz_v) / (Ptl * r);
        const double C = 2.0 * Re * dz_phi;
        const double CC = -2.0 * RRP * theta[AX(i, j)] * dz_phi;
        const double D = axs_drr_off(T, vel, ld, i, j, nr);
        const double E = axs_dr_off(T, vel, ld, i, j) / r;
        const double F = axs_dzz_off(T, vel, ld, i, j, nz);
        d.f[GB_A_veln][AX(i, j)] = (AA * d.f[GB_A_velp][AX(i, j)] + arak / Ptl - B - C - CC + D + E + F) / A;
    }
}

// temperature of the stretched state at (i, j), j = 0..nz (rows 0 and nz
// mirrored: d/dz = 0, d2/dz2 from the wall spacing)
__device__ __forceinline__ void axs_temperature_at(const AxiDev &d, int i, int j)
{
    const AxsTab &T = d.st;
    const int ld = d.ld, nr = d.nr, nz = d.nz;
    const double dt = d.dt;
    const double *phi = d.f[GB_A_phi], *theta = d.f[GB_A_theta];
    const double r = T.r[i];
    double arak, B, E, czzc;
    if (j == 0) {
        const double h1 = T.z[1] - T.z[0];
        arak = 0.0;
        B = 0.0;
        E = 2.0 * theta[AX(i, 1)] / (h1 * h1);
        czzc = -2.0 / (h1 * h1);
    } else if (j == nz) {
        const double hn = T.z[nz] - T.z[nz - 1];
        arak = 0.0;
        B = 0.0;
        E = 2.0 * theta[AX(i, nz - 1)] / (hn * hn);
        czzc = -2.0 / (hn * hn);
    } else {
        arak = axs_arakawa(T, phi, theta, ld, i, j);
        B = phi[AX(i, j)] * axs_dz(T, theta, ld, i, j) / r;
        E = axs_dzz_off(T, theta, ld, i, j, nz);
        czzc = axs_czzc(T, j, nz);
    }
    const double sigma = axs_crrc(T, i, nr) + SCR(i, 2) / r + czzc;
    const double cf3 = 1.0 / (2.0 * dt) - sigma / 2.0;
    const double cf4 = 1.0 / (2.0 * dt) + sigma / 2.0;
    const double C = axs_drr_off(T, theta, ld, i, j, nr);
    const double D = axs_dr_off(T, theta, ld, i, j) / r;
    d.f[GB_A_thetan][AX(i, j)] = (cf4 * d.f[GB_A_thetap][AX(i, j)] + arak + B + C + D + E) / cf3;
}

#undef SCR
#undef SCRR
#undef SCZ
#undef SCZZ

// vorticity (rotann2.f:268-316, what & 1) and velocity (rotann2.f:324-370,
// what & 2) on the interior, one thread per point (S: the stretched forms).
template <bool S>
__device__ __forceinline__ void k_axi_vort_vel_body(const AxiDev &d, int what, int bidx)
{
    const int t = bidx * blockDim.x + threadIdx.x;
    const int ni = d.nr - 1, nj = d.nz - 1;
    if (t >= ni * nj || *d.abort) return;
    const int i = t % ni + 1, j = t / ni + 1;
    if constexpr (S) {
        axs_vort_vel_at(d, what, i, j);
        return;
    }
    const int ld = d.ld;
    const int ip = i + 1, im = i - 1, jp = j + 1, jm = j - 1;
    const double dr = d.dr, dz = d.dz, Ptl = d.Ptl;
    const double *phi = d.f[GB_A_phi], *omeg = d.f[GB_A_omeg], *vel = d.f[GB_A_vel], *theta = d.f[GB_A_theta];
    const double RRP = d.Ra / d.Re / Ptl;
    const double r = d.r0 + (double)i * dr;
    const double A = d.cf1 + 1.0 / (2.0 * (r * r));
    const double AA = d.cf2 - 1.0 / (2.0 * (r * r));
    if (what & 1) {
        const double arak = arakawa_at(phi, omeg, ld, i, j, dr, dz);
        const double B = (1.0 / (2.0 * Ptl * r * dz)) *
                         (phi[AX(i, j)] * (omeg[AX(i, jp)] - omeg[AX(i, jm)]) +
                          omeg[AX(i, j)] * (phi[AX(i, jp)] - phi[AX(i, jm)]));
        const double C = (1.0 / (Ptl * r * dz)) * vel[AX(i, j)] * (vel[AX(i, jp)] - vel[AX(i, jm)]);
        const double D = d.Re * (vel[AX(i, jp)] - vel[AX(i, jm)]) / dz;
        const double E = r * d.Ra * (theta[AX(i, jp)] - theta[AX(i, jm)]) / (2.0 * dz);
        const double EE = RRP * vel[AX(i, j)] * (theta[AX(i, jp)] - theta[AX(i, jm)]) / dz +
                          RRP * theta[AX(i, j)] * (vel[AX(i, jp)] - vel[AX(i, jm)]) / dz;
        const double F = (omeg[AX(ip, j)] + omeg[AX(im, j)]) / (dr * dr);
        const double G = (1.0 / (2.0 * r * dr)) * (omeg[AX(ip, j)] - omeg[AX(im, j)]);
        const double H = (omeg[AX(i, jp)] + omeg[AX(i, jm)]) / (dz * dz);
        d.f[GB_A_omegn][AX(i, j)] =
            (AA * d.f[GB_A_omegp][AX(i, j)] + arak / Ptl + B + C + D - E - EE + F + G + H) / A;
    }
    if (what & 2) {
        const double arak = arakawa_at(phi, vel, ld, i, j, dr, dz);
        const double B = (1.0 / (2.0 * Ptl * r * dz)) *
                         (vel[AX(i, j)] * (phi[AX(i, jp)] - phi[AX(i, jm)]) -
                          phi[AX(i, j)] * (vel[AX(i, jp)] - vel[AX(i, jm)]));
        const double C = d.Re * (phi[AX(i, jp)] - phi[AX(i, jm)]) / dz;
        const double CC = -RRP * theta[AX(i, j)] * (phi[AX(i, jp)] - phi[AX(i, jm)]) / dz;
        const double D = (vel[AX(ip, j)] + vel[AX(im, j)]) / (dr * dr);
        const double E = (1.0 / (2.0 * r * dr)) * (vel[AX(ip, j)] - vel[AX(im, j)]);
        const double F = (vel[AX(i, jp)] + vel[AX(i, jm)]) / (dz * dz);
        d.f[GB_A_veln][AX(i, j)] = (AA * d.f[GB_A_velp][AX(i, j)] + arak / Ptl - B - C - CC + D + E + F) / A;
    }
}

template <bool S>
__global__ void k_axi_vort_vel(AxiDev d, int what) { k_axi_vort_vel_body<S>(d, what, blockIdx.x); }

// temperature, rotann2.f:379-424: rows j = 0 and nz mirror their neighbour
// and take no Jacobian.
template <bool S>
__device__ __forceinline__ void k_axi_temperature_body(const AxiDev &d, int bidx)
{
    const int t = bidx * blockDim.x + threadIdx.x;
    const int ni = d.nr - 1, nj = d.nz + 1;
    if (t >= ni * nj || *d.abort) return;
    const int i = t % ni + 1, j = t / ni;
    if constexpr (S) {
        axs_temperature_at(d, i, j);
        return;
    }
    const int ld = d.ld, nz = d.nz;
    const double dr = d.dr, dz = d.dz;
    const double *phi = d.f[GB_A_phi], *theta = d.f[GB_A_theta];
    const int ip = i + 1, im = i - 1;
    int jp = j + 1, jm = j - 1;
    double arak;
    if (j == 0) {
        jm = jp;
        arak = 0.0;
    } else if (j == nz) {
        jp = jm;
        arak = 0.0;
    } else {
        arak = arakawa_at(phi, theta, ld, i, j, dr, dz);
    }
    const double r = d.r0 + (double)i * dr;
    const double B = (1.0 / (2.0 * r * dz)) * phi[AX(i, j)] * (theta[AX(i, jp)] - theta[AX(i, jm)]);
    const double C = (theta[AX(ip, j)] + theta[AX(im, j)]) / (dr * dr);
    const double D = (1.0 / (2.0 * r * dr)) * (theta[AX(ip, j)] - theta[AX(im, j)]);
    const double E = (theta[AX(i, jp)] + theta[AX(i, jm)]) / (dz * dz);
    d.f[GB_A_thetan][AX(i, j)] = (d.cf4 * d.f[GB_A_thetap][AX(i, j)] + arak + B + C + D + E) / d.cf3;
}

template <bool S>
__global__ void k_axi_temperature(AxiDev d) { k_axi_temperature_body<S>(d, blockIdx.x); }

// update, rotann2.f:497-539, one thread per point: Thom wall vorticity (the
// r-walls written last own the corners), v = 0 on the walls, T = 0 / 1 on
// the inner / outer wall, then the time levels rotate.  The steady-state
// test's maxima of |x - x_p| (rotann2.f:162-180) are gathered here.
// S: the stretched grid's wall spacings in the Thom wall vorticity (rcsc.f
// update, :706-751).
template <bool S>
__device__ __forceinline__ void k_axi_update_body(const AxiDev &d, int bidx)
{
    const int t = bidx * blockDim.x + threadIdx.x;
    const int nr = d.nr, nz = d.nz, ld = d.ld;
    if (*d.abort) return;   // uniform over the grid
    const bool live = t < (nr + 1) * (nz + 1);
    double e[3] = {0.0, 0.0, 0.0};
    if (live) {
        const int i = t % (nr + 1), j = t / (nr + 1);
        const size_t c = AX(i, j);
        double *const *f = d.f;
        const double *phi = f[GB_A_phi];
        double hr0 = d.dr, hrn = d.dr, hz0 = d.dz, hzn = d.dz;
        if constexpr (S) {
            hr0 = d.st.r[1] - d.st.r[0];
            hrn = d.st.r[nr] - d.st.r[nr - 1];
            hz0 = d.st.z[1] - d.st.z[0];
            hzn = d.st.z[nz] - d.st.z[nz - 1];
        }
        double on = f[GB_A_omegn][c], vn = f[GB_A_veln][c], tn = f[GB_A_thetan][c];
        if (i == 0) {
            on = 2.0 * phi[AX(1, j)] / (hr0 * hr0);
            vn = 0.0;
            tn = 0.0;
        } else if (i == nr) {
            on = 2.0 * phi[AX(nr - 1, j)] / (hrn * hrn);
            vn = 0.0;
            tn = 1.0;
        } else if (j == 0) {
            on = 2.0 * phi[AX(i, 1)] / (hz0 * hz0);
            vn = 0.0;
        } else if (j == nz) {
            on = 2.0 * phi[AX(i, nz - 1)] / (hzn * hzn);
            vn = 0.0;
        }
        f[GB_A_omegn][c] = on;
        f[GB_A_veln][c] = vn;
        f[GB_A_thetan][c] = tn;
        const double o = f[GB_A_omeg][c], v = f[GB_A_vel][c], th = f[GB_A_theta][c];
        f[GB_A_omegp][c] = o;
        f[GB_A_omeg][c] = on;
        f[GB_A_velp][c] = v;
        f[GB_A_vel][c] = vn;
        f[GB_A_thetap][c] = th;
        f[GB_A_theta][c] = tn;
        e[0] = fabs(on - o);
        e[1] = fabs(vn - v);
        e[2] = fabs(tn - th);
    }
    // non-negative doubles order like their bit patterns: warp maximum, then
    // one atomic per warp
    for (int q = 0; q < 3; ++q) {
        unsigned long long m = (unsigned long long)__double_as_longlong(e[q]);
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long w = __shfl_down_sync(0xffffffffu, m, o);
            m = w > m ? w : m;
        }
        if ((threadIdx.x & 31) == 0) atomicMax(&d.errmax[q], m);
    }
}

template <bool S>
__global__ void k_axi_update(AxiDev d) { k_axi_update_body<S>(d, blockIdx.x); }

// heat, rotann2.f:468-487: the per-row terms in parallel, summed by one
// thread in the reference's order.
// S: the five-point one-sided weights of the stretched grid and the
// trapezoid rule on its z positions.
template <bool S>
__device__ __forceinline__ void k_axi_heat_body(const AxiDev &d, int bidx)
{
    extern __shared__ double sh[];
    if (*d.abort == 1) return;
    const int ld = d.ld, nz = d.nz;
    const double dr = d.dr, dz = d.dz;
    const double *th = d.f[GB_A_theta];
    for (int j = threadIdx.x; j <= nz; j += blockDim.x) {
        if constexpr (S) {
            const AxsTab &T = d.st;
            const double *w = T.hw;
            const double wz = j == 0 ? (T.z[1] - T.z[0]) / 2.0
                                     : (j == nz ? (T.z[nz] - T.z[nz - 1]) / 2.0 : (T.z[j + 1] - T.z[j - 1]) / 2.0);
            sh[j] = wz * (w[0] * th[AX(0, j)] + w[1] * th[AX(1, j)] + w[2] * th[AX(2, j)] + w[3] * th[AX(3, j)] +
                          w[4] * th[AX(4, j)]);
        } else {
            const double div = (j == 0 || j == nz) ? 24.0 * dr : 12.0 * dr;
            sh[j] = dz * (-25.0 * th[AX(0, j)] + 48.0 * th[AX(1, j)] - 36.0 * th[AX(2, j)] + 16.0 * th[AX(3, j)] -
                          3.0 * th[AX(4, j)]) / div;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double trans = sh[0];
        trans = trans + sh[nz];
        for (int j = 1; j <= nz - 1; ++j) trans = trans + sh[j];
        d.heat[0] = trans;
    }
}

template <bool S>
__global__ void k_axi_heat(AxiDev d) { k_axi_heat_body<S>(d, blockIdx.x); }

// Per-step bookkeeping: Nu and sweeps into the history, the steady-state
// test (REAL*4 threshold 1e-6, rotann2.f:191) and its reset.
__device__ __forceinline__ void k_axi_record_body(const AxiDev &d, int bidx)
{
    if (threadIdx.x != 0 || bidx != 0) return;
    if (*d.abort) return;
    const int s = *d.step_index;
    if (s < d.hist_cap) {
        d.nu_hist[s] = d.heat[0] * d.nu_c / d.nu_d;
        d.sweep_hist[s] = d.status[1];
    }
    *d.step_index = s + 1;
    const double tol = (double)1e-6f;
    const double e1 = __longlong_as_double((long long)d.errmax[0]), e2 = __longlong_as_double((long long)d.errmax[1]),
                 e3 = __longlong_as_double((long long)d.errmax[2]);
    if (e1 < tol && e2 < tol && e3 < tol) *d.abort = 2;
    d.errmax[0] = d.errmax[1] = d.errmax[2] = 0ull;
}

__global__ void k_axi_record(AxiDev d) { k_axi_record_body(d, blockIdx.x); }

// ---------------------------------------------------------------------------
// Streamfunction multigrid (rotann2.f:543-854)
// ---------------------------------------------------------------------------
template <class T> struct AxiView {
    int n1, n2, ld, lf;
    T *v;
    const T *f;
    T hr, hhr, hhz, ihr, ihhr, ihhz;
    const T *rval, *irv, *irq;   // float: rval only
    const T *fac[2];             // r-lines (one table), z-lines
};
__device__ __forceinline__ AxiView<double> axi_view(const AxiDev &d, int l, double)
{
    const AxiLevel &L = d.lev[l];
    return {L.n1, L.n2, L.n1 + 1, L.lf, L.v, L.f, L.hr, L.hhr, L.hhz, L.ihr, L.ihhr, L.ihhz, d.rval, d.irv, d.irq, {L.fac_r, L.fac_z}};
}
__device__ __forceinline__ AxiView<float> axi_view(const AxiDev &d, int l, float)
{
    const AxiLevel &L = d.lev[l];
    return {L.n1, L.n2, L.n1 + 1, L.lf, L.v32, L.f32, (float)L.hr, (float)L.hhr, (float)L.hhz, (float)L.ihr, (float)L.ihhr,
            (float)L.ihhz, d.rval32, nullptr, nullptr, {L.fac_r32, L.fac_z32}};
}
#define V(i, j) L.v[(i) + L.ld * (j)]
#define F(i, j) L.f[(i) + L.ld * (j)]

// x / h: the IEEE quotient (FP64: from the stored reciprocal)
__device__ __forceinline__ double axi_over(double x, double h, double ih) { return div_by_rcp(x, h, ih); }
__device__ __forceinline__ float axi_over(float x, float h, float) { return x / h; }

// Right-hand sides of r-line j at row i (rotann2.f:698-710) and of z-line i
// at row j (rotann2.f:712-725).
template <class T> __device__ __forceinline__ T axi_rhs(const AxiView<T> &L, int dir, int i, int j)
{
    if (dir == 0) return axi_over(-(V(i, j + 1) + V(i, j - 1)), L.hhz, L.ihhz) + F(i, j);
    const T rv = L.rval[i * L.lf];
    T irv;
    if constexpr (sizeof(T) == 8) irv = L.irv[i * L.lf];
    else irv = 1.0f / rv;
    const T vp = V(i + 1, j), vm = V(i - 1, j);
    return axi_over(-(vp + vm), L.hhr, L.ihhr) + F(i, j) - axi_over(axi_over((vp - vm) * T(0.5), rv, irv), L.hr, L.ihr);
}

// f - A v at (i, j) (relax's residual, rotann2.f:727-741)
template <class T> __device__ __forceinline__ T axi_resid(const AxiView<T> &L, T drdz, int i, int j)
{
    const T rv = L.rval[i * L.lf];
    T irv, irq;
    if constexpr (sizeof(T) == 8) {
        irv = L.irv[i * L.lf];
        irq = L.irq[i * L.lf];
    } else {
        irv = 1.0f / rv;
        irq = irv * irv;
    }
    const T vp = V(i + 1, j), vm = V(i - 1, j), vc = V(i, j);
    const T a = axi_over(vp + vm, L.hhr, L.ihhr) + axi_over(axi_over((vp - vm) * T(0.5), L.hr, L.ihr), rv, irv) -
                axi_over(vc, rv * rv, irq) + axi_over(V(i, j + 1) + V(i, j - 1), L.hhz, L.ihhz) - vc * drdz;
    return F(i, j) - a;
}

// Dynamic shared memory of a solve: per staged line its right-hand sides and
// its factors.
#define AXI_SMEM_BYTES (160 * 1024)

// The nl lines first, first + step, ... of one direction (DIR 0: r-lines j,
// DIR 1: z-lines i), which read none of one another: a colour, or one line of
// the reference's order.  Each CTA takes a contiguous share, in batches that
// fit its shared memory: the lines' factors are copied there while all
// threads form the right-hand sides, the lines are eliminated (FP64: one
// thread per line in the reference's order; FP32: up to 32 lanes per line),
// the solutions go back.  FRESH: the r-lines' table is not staged yet (the
// reference's order comes here line by line).
template <class T, int DIR, bool FRESH = true>
__device__ __noinline__ void axi_lines(const AxiDev &d, int l, int first, int step, int nl)
{
    extern __shared__ __align__(16) unsigned char s_axi[];
    constexpr bool F64 = sizeof(T) == 8;
    T *smem = (T *)s_axi;
    const Cluster cl = Cluster::self();
    const AxiView<T> L = axi_view(d, l, T(0));
    const int n = DIR == 0 ? L.n1 - 1 : L.n2 - 1;
    const int flen = (int)(F64 ? tdma_fac_len(n) : tdma32_len(n));
    const int fpitch = DIR == 0 ? 0 : F64 ? flen | 1 : flen;   // r-lines share one table
    const int lpitch = F64 ? 0 : wl_pitch(n), lg = F64 ? 0 : wl_log2m(n);
    const int share = (nl + cl.size - 1) / cl.size;
    const int t0 = cl.rank * share, t1 = min(nl, t0 + share);
    const int words = (int)(AXI_SMEM_BYTES / sizeof(T)) - (DIR == 0 ? (flen + 3) & ~3 : 0);
    int B = F64 ? (words - n) / (n + fpitch) : words / (lpitch + fpitch);
    const bool staged = B >= 1;       // a line with its factors fits (n up to 4000 in FP64)
    if (!staged) B = 1;
    B = min(B, min(share, (int)blockDim.x));
    T *sfac = smem, *x = !staged ? smem : smem + (DIR == 0 ? (flen + 3) & ~3 : B * fpitch);
    auto table = [&](int line) { return L.fac[DIR] + (DIR == 0 ? 0 : (size_t)(line - 1) * flen); };
    for (int b0 = t0; b0 < t1; b0 += B) {
        const int nb = min(B, t1 - b0), pitch = nb | 1;
        // FP64: [row][line], odd pitch; FP32: [line][row], padded per lane
        auto at = [&](int t, int q) -> T & { return F64 ? x[q * pitch + t] : x[t * lpitch + wl_slot(lg, q)]; };
        if (staged && FRESH)
            for (int t = 0; t < (DIR == 0 ? 1 : nb); ++t)
                async_copy(sfac + t * fpitch, table(first + step * (b0 + t)), flen, threadIdx.x, blockDim.x);
        if (DIR == 0) {
            const RowSplit split(n);
            for (int idx = threadIdx.x; idx < nb * n; idx += blockDim.x) {
                int t, q;
                split(idx, t, q);
                at(t, q) = axi_rhs<T>(L, 0, q + 1, first + step * (b0 + t));
            }
        } else {
            const RowSplit split(nb);
            for (int idx = threadIdx.x; idx < nb * n; idx += blockDim.x) {
                int q, t;
                split(idx, q, t);
                at(t, q) = axi_rhs<T>(L, 1, first + step * (b0 + t), q + 1);
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
                if (staged) tdma_staged(sfac + t * fpitch, n, x + t, pitch);
                else tdma_staged(table(first + step * (b0 + t)), n, x + t, pitch);
            }
        } else {
            if (staged) wl_lines<false, false, true>(sfac, fpitch, n, x, lpitch, nb);
            else wl_lines<false, false, true>(table(first + step * b0), DIR == 0 ? 0 : (size_t)step * flen, n, x, lpitch, nb);
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

// relax's line sweeps (rotann2.f:668-725), nrel of them, in place on v.  The
// reference also forms the residual after every sweep; only the last one is
// ever read, and the caller forms that.
template <class T> __device__ __forceinline__ void axi_sweeps(const AxiDev &d, int l)
{
    const int nj = d.lev[l].n2 - 1, ni = d.lev[l].n1 - 1;
    for (int irel = 0; irel < d.nrel; ++irel) {
        if (d.mode == GB_SMOOTHER_LEX) {
            for (int j = 1; j <= nj; ++j) {
                if (j == 1) axi_lines<T, 0>(d, l, j, 1, 1);
                else axi_lines<T, 0, false>(d, l, j, 1, 1);
            }
            for (int i = 1; i <= ni; ++i) axi_lines<T, 1>(d, l, i, 1, 1);
        } else {
            for (int c = 1; c <= 2; ++c)
                if (c <= nj) axi_lines<T, 0>(d, l, c, 2, (nj - c) / 2 + 1);
            for (int c = 1; c <= 2; ++c)
                if (c <= ni) axi_lines<T, 1>(d, l, c, 2, (ni - c) / 2 + 1);
        }
    }
}

// The residual of level l into rc (not followed by a barrier): its largest
// magnitude and whether one is a NaN over the calling thread's points.
template <class T, class R> __device__ __noinline__ T axi_residual(const AxiDev &d, int l, R *rc, int *nan_out)
{
    const Cluster cl = Cluster::self();
    const AxiView<T> L = axi_view(d, l, T(0));
    const T drdz = T(2.0) * (T(1.0) / L.hhr + T(1.0) / L.hhz);
    const int ni = L.n1 - 1, tot = ni * (L.n2 - 1);
    const RowSplit split(ni);
    T m = T(0);
    int nan = 0;
    for (int idx = cl.tid(); idx < tot; idx += cl.nthr()) {
        int j, i;
        split(idx, j, i);
        ++i;
        ++j;
        const T r = axi_resid<T>(L, drdz, i, j);
        rc[i + L.ld * j] = (R)r;
        const T a = fabs(r);
        if (a != a) nan = 1;
        if (a > m) m = a;
    }
    *nan_out = nan;
    return m;
}

// corser (rotann2.f:755-801): the nine-point restriction of rc into the
// packed coarse right-hand side; the rows and columns the reference clears
// (i = 0, n1c and j = 0, n1c: n1 of the coarse level in both directions)
// are zero, and the coarse solution slot is cleared.
template <class T> __device__ __noinline__ void axi_corser(const AxiDev &d, int l, const T *rc)
{
    const Cluster cl = Cluster::self();
    const AxiView<T> L = axi_view(d, l + 1, T(0));
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
            if constexpr (sizeof(T) == 8) {
                temp = q[0];
                temp = temp * T(2) + q[1] + q[-1];
                temp = temp + q[ld] + q[-ld];
                temp = temp * T(2) + q[1 + ld] + q[-1 - ld];
                temp = temp + q[1 - ld] + q[-1 + ld];
                temp = temp * T(0.0625);   // / 16, exactly
            } else {
                temp = 0.25f * q[0] + 0.125f * (q[1] + q[-1] + q[ld] + q[-ld]) + 0.0625f * (q[1 + ld] + q[-1 - ld] + q[1 - ld] + q[-1 + ld]);
            }
        }
        fc[idx] = temp;
        L.v[idx] = T(0);
    }
    cl.sync();
}

// finer (rotann2.f:803-854): bilinear prolongation added to the fine level.
// The coarse solution slot is cleared by the next corser.
template <class T> __device__ __noinline__ void axi_finer(const AxiDev &d, int l)
{
    const Cluster cl = Cluster::self();
    const AxiView<T> Cc = axi_view(d, l, T(0)), L = axi_view(d, l - 1, T(0));
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

// poisson (rotann2.f:598-666): phi from omegn.
__device__ __forceinline__ void k_axi_mg_solve_body(const AxiDev &d)
{
    __shared__ ClMaxState s_max;
    const Cluster cl = Cluster::self();
    if (*d.abort) return;   // the same for every CTA: nothing sets it while the solve runs
    int turn = 0;
    const int nlev = d.nlev;
    const AxiView<double> L = axi_view(d, 1, 0.0);
    const int tp = L.ld * (L.n2 + 1);
    double *psi = d.f[GB_A_phi];
    const double *rhs = d.f[GB_A_omegn];
    for (int idx = cl.tid(); idx < tp; idx += cl.nthr()) {
        const_cast<double *>(L.f)[idx] = rhs[idx];
        L.v[idx] = psi[idx];
    }
    cl.sync();
    double res1 = 0.0;
    int status = GB_MAXSWEEPS, sweeps = d.maxsweeps, nan1 = 0;
    // relax on level l and the residual for the restriction or the test that
    // follows; the norm matters on level 1 only
    auto relax = [&](int l, bool restricted) {
        axi_sweeps<double>(d, l);
        if (l != 1 && !restricted) return;
        int nan;
        const double m = axi_residual<double>(d, l, d.rc, &nan);
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
            axi_corser<double>(d, l, d.rc);
            relax(l + 1, l + 1 < nlev);
        }
        for (int l = nlev; l >= 2; --l) {
            axi_finer<double>(d, l);
            relax(l - 1, false);
        }
        if (nan1) { status = GB_NAN; sweeps = sweep; break; }
        if (res1 < d.tolcon) {
            for (int idx = cl.tid(); idx < tp; idx += cl.nthr()) psi[idx] = L.v[idx];
            status = GB_OK;
            sweeps = sweep;
            break;
        }
    }
    if (cl.tid() == 0) {
        d.status[0] = status;
        d.status[1] = sweeps;
        if (status == GB_NAN) *d.abort = 1;
    }
    cl.sync();   // no CTA leaves while another may still read its reduction slot
}

__global__ void __maxnreg__(255) k_axi_mg_solve(const __grid_constant__ AxiDev d) { k_axi_mg_solve_body(d); }

// ---------------------------------------------------------------------------
// Mixed precision: FP64 defect correction around one FP32 V-cycle of the
// reference's schedule (relax on the finest level, down, up) on A e = r from
// e = 0; psi += e in FP64 (AXI has no over-relaxation).  This form, on global
// memory, serves the reference's line order and grids whose cycles do not fit
// a cluster's shared memory; meridian.cu has the other.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void k_axi_mg_solve_mixed_body(const AxiDev &d)
{
    __shared__ ClMaxState s_max;
    const Cluster cl = Cluster::self();
    if (*d.abort) return;
    int turn = 0;
    const int nlev = d.nlev;
    const AxiView<double> L = axi_view(d, 1, 0.0);
    const AxiView<float> L32 = axi_view(d, 1, 0.f);
    const int tp = L.ld * (L.n2 + 1);
    double *psi = d.f[GB_A_phi];
    const double *rhs = d.f[GB_A_omegn];
    for (int idx = cl.tid(); idx < tp; idx += cl.nthr()) {
        const_cast<double *>(L.f)[idx] = rhs[idx];
        L.v[idx] = psi[idx];
        L32.v[idx] = 0.f;
    }
    cl.sync();
    auto relax = [&](int l, bool restricted) {
        axi_sweeps<float>(d, l);
        if (!restricted) return;
        int nan;
        axi_residual<float>(d, l, d.rc32, &nan);
        cl.sync();
    };
    int status = GB_MAXSWEEPS, cycles = 0;
    for (int it = 0;; ++it) {
        int nan;
        const double m = axi_residual<double>(d, 1, const_cast<float *>(L32.f), &nan);
        const double res = cl_max(cl, s_max, turn, m, nan);
        if (nan) { status = GB_NAN; break; }
        if (res < d.tolcon) { status = GB_OK; break; }
        if (it == d.maxsweeps) break;
        relax(1, nlev > 1);
        for (int l = 1; l <= nlev - 1; ++l) {
            axi_corser<float>(d, l, d.rc32);
            relax(l + 1, l + 1 < nlev);
        }
        for (int l = nlev; l >= 2; --l) {
            axi_finer<float>(d, l);
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
        for (int idx = cl.tid(); idx < tp; idx += cl.nthr()) psi[idx] = L.v[idx];
    if (cl.tid() == 0) {
        d.status[0] = status;
        d.status[1] = cycles;
        if (status == GB_NAN) *d.abort = 1;
    }
    cl.sync();
}
#undef V
#undef F

__global__ void __maxnreg__(255) k_axi_mg_solve_mixed(const __grid_constant__ AxiDev d) { k_axi_mg_solve_mixed_body(d); }

// FP32 copies of rval and the line tables: block l - 1 takes level l, its
// threads the level's lines (thread 0 also the r-line table).
__global__ void k_axi_factors32(AxiDev d)
{
    const int l = 1 + blockIdx.x;
    if (l == 1)
        for (int i = threadIdx.x; i <= d.lev[1].n1; i += blockDim.x) d.rval32[i] = (float)d.rval[i];
    const AxiLevel &L = d.lev[l];
    if (threadIdx.x == 0 && L.n1 - 1 >= 1) tdma32_fold(L.fac_r, L.n1 - 1, L.fac_r32);
    if (L.n2 - 1 >= 1) {
        const int n = L.n2 - 1;
        for (int i = 1 + threadIdx.x; i <= L.n1 - 1; i += blockDim.x)
            tdma32_fold(L.fac_z + (size_t)(i - 1) * tdma_fac_len(n), n, L.fac_z32 + (size_t)(i - 1) * tdma32_len(n));
    }
}

// The resident solve's weights (meridian.cu) from relax's operator.
__global__ void k_axi_weights(const __grid_constant__ AxiDev d, const __grid_constant__ MerDev m)
{
    const int l = 1 + blockIdx.y, t = blockIdx.x * blockDim.x + threadIdx.x;
    const AxiLevel &L = d.lev[l];
    if (t >= 1 && t < L.n1) {
        const float r = d.rval32[t * L.lf];
        const_cast<float4 *>(m.lev[l].ci)[t] = make_float4(r, r * r, 1.0f / r, 1.0f / (r * r));
        if (l == 1) {
            const double rv = d.rval[t];
            MerRow &q = const_cast<MerRow *>(m.d_i)[t];
            q.r = rv;
            q.ir = d.irv[t];
            q.rr = rv * rv;
            q.irr = d.irq[t];
        }
    }
}

__global__ void k_axi_rval(AxiDev d)
{
    for (int i = threadIdx.x; i <= d.lev[1].n1; i += blockDim.x) {
        const double rv = (double)i * d.lev[1].hr + d.r0;
        d.rval[i] = rv;
        d.irv[i] = 1.0 / rv;
        d.irq[i] = 1.0 / (rv * rv);
    }
}

// The factored line matrices of every level, with the coefficients relax
// forms for each line (rotann2.f:698-721): block l - 1 takes level l; its
// thread 0 the r-line matrix (work: three arrays per level), every thread
// the z-line matrices of its rows, whose coefficients are constant along the
// line (the tdma factorization with scalar a, b, c, the same operations).
__global__ void k_axi_factors(AxiDev d, double *work)
{
    const int l = 1 + blockIdx.x;
    const AxiLevel &L = d.lev[l];
    const int n1 = L.n1, n2 = L.n2;
    const double hhr = L.hhr, hhz = L.hhz, hr = L.hr;
    const int nmax = (d.lev[1].n1 > d.lev[1].n2 ? d.lev[1].n1 : d.lev[1].n2) + 2;
    if (threadIdx.x == 0 && n1 - 1 >= 1) {
        double *a = work + (size_t)blockIdx.x * 3 * nmax, *b = a + nmax, *c = b + nmax;
        for (int i = 1; i <= n1 - 1; ++i) {
            const double rv = d.rval[i * L.lf];
            a[i - 1] = 1.0 / hhr - 0.5 / hr / rv;
            c[i - 1] = 1.0 / hhr + 0.5 / hr / rv;
            b[i - 1] = -2.0 / hhr - 2.0 / hhz - 1.0 / (rv * rv);
        }
        factor_tdma(a, b, c, n1 - 1, L.fac_r);
    }
    const int n = n2 - 1;
    if (n < 1) return;
    for (int i = 1 + threadIdx.x; i <= n1 - 1; i += blockDim.x) {
        const double rv = d.rval[i * L.lf];
        const double av = 1.0 / hhz, cv = 1.0 / hhz;
        const double bv = -2.0 / hhr - 2.0 / hhz - 1.0 / (rv * rv);
        double *fac = L.fac_z + (size_t)(i - 1) * tdma_fac_len(n);
        double *fact = fac, *bp = fac + n, *cc = fac + 2 * n, *ibp = fac + 3 * n;
        bp[0] = bv;
        fact[0] = 0.0;
        for (int j = 0; j < n; ++j) cc[j] = cv;
        for (int j = 1; j < n; ++j) {
            fact[j] = av / bp[j - 1];
            bp[j] = bv - fact[j] * cv;
        }
        for (int j = 0; j < n; ++j) ibp[j] = 1.0 / bp[j];
    }
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
struct gb_axi {
    gb_axi_params p;
    AxiDev dev;
    gb_str *str = nullptr;              // stretched grid: rcsc.f's multigrid for the streamfunction
    double *stab = nullptr;             // stretched grid: the transport's tables (AxsTab)
    double *fields = nullptr, *pool = nullptr;
    void *small = nullptr, *hist = nullptr;
    int hist_cap = 0;
    cudaStream_t stream = nullptr;
    cudaGraphExec_t graph = nullptr;
    gb_axi_params graph_params;
    double dr_set = 0.0, dz_set = 0.0;   // a Fortran caller's /num/ spacings, 0 = derived
    int ctas = 1;                        // CTAs per ZEBRA solve on global memory
    MerDev mer;                          // the resident mixed solve, where its plan fits
    int mer_most = 0;                    // the largest cluster it can have; 0: k_axi_mg_solve_mixed
    int mer_ctas = 0;                    // its CTAs
    void *mer_mem = nullptr;
};

static int axi_levels(int nr, int nz)
{
    int nlev = 0, it = nr, it2 = nr, jt = nz, jt2 = nz;
    for (int i = 2; i <= 8; ++i) {
        it = it / 2;
        jt = jt / 2;
        if (it * 2 - it2 == 0 && jt * 2 - jt2 == 0) {
            nlev = nlev + 1;
            it2 = it;
            jt2 = jt;
        } else {
            break;
        }
    }
    if (nlev > 6) nlev = 6;
    return nlev;
}

extern "C" void gb_axi_default_params(gb_axi_params *p, int nr, int nz)
{
    memset(p, 0, sizeof(*p));
    p->nr = nr;
    p->nz = nz;
    p->dt = 1e-5;
    p->r0 = 0.5;
    p->rmax = 1.0;
    p->zmax = 0.5;
    p->Ra = 1e5;
    p->Re = 1e2;
    p->Pr = 1.0;
    p->tolcon = 1.0e-6;
    p->maxsweeps = 10000;
    p->nrel = 2;
    p->smoother = GB_SMOOTHER_LEX;
    p->precision = GB_PRB_FP64;
}

static void axi_scalars(gb_axi *h)
{
    AxiDev &d = h->dev;
    const gb_axi_params &p = h->p;
    d.dt = p.dt;
    d.r0 = p.r0;
    d.rmax = p.rmax;
    d.zmax = p.zmax;
    d.Ra = p.Ra;
    d.Re = p.Re;
    d.Ptl = p.Pr;
    d.dr = h->dr_set != 0.0 ? h->dr_set : (p.rmax - p.r0) / (double)p.nr;
    d.dz = h->dz_set != 0.0 ? h->dz_set : p.zmax / (double)p.nz;
    const double dr = d.dr, dz = d.dz, Ptl = p.Pr, dt = p.dt;
    d.cf1 = 1.0 / (2.0 * Ptl * dt) + 1.0 / (dr * dr) + 1.0 / (dz * dz);
    d.cf2 = 1.0 / (2.0 * Ptl * dt) - 1.0 / (dr * dr) - 1.0 / (dz * dz);
    d.cf3 = 1.0 / (2.0 * dt) + 1.0 / (dr * dr) + 1.0 / (dz * dz);
    d.cf4 = 1.0 / (2.0 * dt) - 1.0 / (dr * dr) - 1.0 / (dz * dz);
    d.tolcon = p.tolcon;
    d.maxsweeps = p.maxsweeps;
    d.nrel = p.nrel;
    d.mode = p.smoother;
    d.nu_c = -p.r0 * log(p.r0 / p.rmax);
    d.nu_d = p.zmax * p.rmax;
}

extern "C" int gb_axi_destroy(gb_axi *h)
{
    if (!h) return GB_OK;
    if (h->graph) cudaGraphExecDestroy(h->graph);
    if (h->str) gb_str_destroy(h->str);
    cudaFree(h->stab);
    cudaFree(h->fields);
    cudaFree(h->pool);
    cudaFree(h->small);
    cudaFree(h->hist);
    cudaFree(h->mer_mem);
    if (h->stream) cudaStreamDestroy(h->stream);
    delete h;
    return GB_OK;
}

// Prepares the resident mixed solve; a grid it cannot hold leaves mer_most 0.
static cudaError_t axi_mer_create(gb_axi *h)
{
    const AxiDev &d = h->dev;
    MerDev &m = h->mer;
    memset(&m, 0, sizeof(m));
    m.nlev = d.nlev;
    for (int l = 1; l <= d.nlev; ++l) {
        MerLevel &L = m.lev[l];
        L.n1 = d.lev[l].n1;
        L.n2 = d.lev[l].n2;
        L.fac_r = d.lev[l].fac_r32;
        L.fac_z = d.lev[l].fac_z32;
        L.fac_r_step = 0;
        L.hr = (float)d.lev[l].hr;
        L.hhr = (float)d.lev[l].hhr;
        L.hhz = (float)d.lev[l].hhz;
        L.drdz = 2.0f * (1.0f / L.hhr + 1.0f / L.hhz);
        L.ihr = 1.0f / L.hr;
        L.ihhr = 1.0f / L.hhr;
        L.ihhz = 1.0f / L.hhz;
        const float r0 = (float)(d.r0 * d.r0 < 1.0 ? d.r0 * d.r0 : 1.0), r1 = (float)std::max(1.0, h->p.rmax * h->p.rmax);
        L.quick = 1;
        for (float v : {L.hr, L.hhr, L.hhz, r0, r1})
            if (!(v >= 0x1p-24f && v <= 0x1p24f)) L.quick = 0;
        L.fac_z_step = (int)tdma32_len(L.n2 - 1);
    }
    const AxiLevel &L1 = d.lev[1];
    m.hr = MerOver{L1.hr, L1.ihr};
    m.hhr = MerOver{L1.hhr, L1.ihhr};
    m.hhz = MerOver{L1.hhz, L1.ihhz};
    m.drdz = 2.0 * (1.0 / L1.hhr + 1.0 / L1.hhz);
    m.v = d.lev[1].v;
    m.psi = d.f[GB_A_phi];
    m.rhs = d.f[GB_A_omegn];
    m.status = d.status;
    m.abort = d.abort;
    h->mer_most = mer_fit(m, CL_MAX_CTAS);
    if (!h->mer_most) return cudaSuccess;
    h->mer_ctas = mer_alone(m, h->mer_most);
    cudaError_t e = cudaMalloc(&h->mer_mem, mer_weight_bytes(m));
    if (e != cudaSuccess) return e;
    mer_weight_layout(m, h->mer_mem);
    k_axi_weights<<<dim3(gb_ceil_div((size_t)std::max(m.lev[1].n1, m.lev[1].n2), 128), m.nlev), 128>>>(d, m);
    return cudaGetLastError();
}

static int axi_create(const gb_axi_params *p, double dr, double dz, gb_axi **out, int *nlev_out);

extern "C" int gb_axi_create(const gb_axi_params *p, gb_axi **out, int *nlev_out)
{
    return axi_create(p, 0.0, 0.0, out, nlev_out);
}

extern "C" int gb_axi_create_spacing(const gb_axi_params *p, double dr, double dz, gb_axi **out, int *nlev_out)
{
    if (!(dr > 0.0 && dz > 0.0)) {
        gb_set_error("gb_axi_create_spacing: spacings must be positive");
        return GB_ERR_INVALID;
    }
    return axi_create(p, dr, dz, out, nlev_out);
}

static int axi_create(const gb_axi_params *p, double dr, double dz, gb_axi **out, int *nlev_out)
{
    if (!p || !out) { gb_set_error("gb_axi_create: null argument"); return GB_ERR_INVALID; }
    *out = nullptr;
    const int nr = p->nr, nz = p->nz;
    const int nlev = axi_levels(nr, nz);
    if (nlev_out) *nlev_out = nlev;
    if (nr < 4 || nz < 4 || nlev < 1 || nr > 8192 || nz > 8192 || !(p->r0 > 0.0 && p->rmax > p->r0) ||
        !(p->zmax > 0.0) || p->nrel < 1 || p->maxsweeps < 1 || p->Re == 0.0) {
        gb_set_error("gb_axi_create: unsupported parameters (nr=%d nz=%d need both even with >= 1 multigrid level; "
                     "0 < r0 < rmax, zmax > 0, Re != 0)", nr, nz);
        return GB_ERR_INVALID;
    }
    if (p->precision != GB_PRB_FP64 && p->precision != GB_PRB_MIXED) {
        gb_set_error("gb_axi_create: unknown precision %d", p->precision);
        return GB_ERR_INVALID;
    }
    gb_axi *h = new gb_axi();
    h->p = *p;
    h->dr_set = dr;
    h->dz_set = dz;
    AxiDev &d = h->dev;
    memset(&d, 0, sizeof(d));
    d.nr = nr;
    d.nz = nz;
    d.ld = nr + 1;
    d.nlev = nlev;
    axi_scalars(h);
    const size_t fsz = (size_t)d.ld * (size_t)(nz + 1);
    cudaError_t e = cudaMalloc(&h->fields, sizeof(double) * fsz * GB_A_COUNT);
    if (e != cudaSuccess) { gb_set_error("gb_axi_create: %s", cudaGetErrorString(e)); delete h; return GB_ERR_ALLOC; }
    cudaMemset(h->fields, 0, sizeof(double) * fsz * GB_A_COUNT);
    for (int q = 0; q < GB_A_COUNT; ++q) d.f[q] = h->fields + (size_t)q * fsz;
    // pool: rval and its reciprocals, rc, rc32, rval32, then per level v, f, fac_r, fac_z and their FP32 forms
    size_t need = 3 * (size_t)(nr + 2) + fsz + fsz / 2 + (size_t)(nr + 2) / 2 + 8;
    for (int l = 1; l <= nlev; ++l) {
        const size_t n1 = (size_t)nr * 2 / ((size_t)1 << l), n2 = (size_t)nz * 2 / ((size_t)1 << l);
        need += 2 * (n1 + 1) * (n2 + 1) + 4 * n1 + n1 * 4 * (n2 + 1);
        need += ((n1 + 1) * (n2 + 1) * 2 + tdma32_len((int)n1) + n1 * tdma32_len((int)n2)) / 2 + 8;
    }
    const size_t work = 3 * (size_t)((nr > nz ? nr : nz) + 2) * (size_t)nlev;   // r-line coefficients, per level
    e = cudaMalloc(&h->pool, sizeof(double) * (need + work));
    if (e != cudaSuccess) { gb_axi_destroy(h); gb_set_error("gb_axi_create: multigrid pool"); return GB_ERR_ALLOC; }
    cudaMemset(h->pool, 0, sizeof(double) * (need + work));
    double *b = h->pool;
    d.rval = b; b += nr + 2;
    d.irv = b; b += nr + 2;
    d.irq = b; b += nr + 2;
    d.rc = b; b += fsz;
    {
        float *fb = (float *)b;
        d.rc32 = fb; fb += fsz;
        d.rval32 = fb; fb += nr + 2;
        b = (double *)(((uintptr_t)fb + 15) & ~(uintptr_t)15);
    }
    for (int l = 1; l <= nlev; ++l) {
        AxiLevel &L = d.lev[l];
        L.n1 = nr * 2 / (1 << l);
        L.n2 = nz * 2 / (1 << l);
        L.lf = (1 << l) / 2;
        L.hr = d.dr * (double)(1 << l) / 2.0;
        L.hz = d.dz * (double)(1 << l) / 2.0;
        L.hhr = L.hr * L.hr;
        L.hhz = L.hz * L.hz;
        L.ihr = 1.0 / L.hr;
        L.ihhr = 1.0 / L.hhr;
        L.ihhz = 1.0 / L.hhz;
        const size_t sz = (size_t)(L.n1 + 1) * (L.n2 + 1);
        L.v = b; b += sz;
        L.f = b; b += sz;
        L.fac_r = b; b += 4 * (size_t)L.n1;                          // tdma_fac_len(n1 - 1) and more
        L.fac_z = b; b += (size_t)L.n1 * 4 * (size_t)(L.n2 + 1);
        float *fb = (float *)b;
        L.v32 = fb; fb += sz;
        L.f32 = fb; fb += sz;
        fb = (float *)(((uintptr_t)fb + 15) & ~(uintptr_t)15);   // the tables are copied 16 bytes at a time
        L.fac_r32 = fb; fb += tdma32_len(std::max(L.n1 - 1, 1));
        L.fac_z32 = fb; fb += (size_t)(L.n1 - 1) * tdma32_len(std::max(L.n2 - 1, 1));
        b = (double *)(((uintptr_t)fb + 15) & ~(uintptr_t)15);
    }
    if ((size_t)(b - h->pool) > need) {
        gb_axi_destroy(h);
        gb_set_error("gb_axi_create: multigrid pool layout overflow");
        return GB_ERR_CUDA;
    }
    double *wk = h->pool + need;
    e = cudaMalloc(&h->small, 4096);
    if (e != cudaSuccess) { gb_axi_destroy(h); gb_set_error("gb_axi_create: state"); return GB_ERR_ALLOC; }
    cudaMemset(h->small, 0, 4096);
    char *sm = (char *)h->small;
    d.heat = (double *)(sm + 0);
    d.errmax = (unsigned long long *)(sm + 64);
    d.abort = (int *)(sm + 128);
    d.status = (int *)(sm + 192);
    d.step_index = (int *)(sm + 256);
    k_axi_rval<<<1, 256>>>(d);
    k_axi_factors<<<d.nlev, 128>>>(d, wk);
    k_axi_factors32<<<d.nlev, 128>>>(d);
    e = cl_prepare(k_axi_mg_solve, AXI_SMEM_BYTES);
    if (e == cudaSuccess) e = cl_prepare(k_axi_mg_solve_mixed, AXI_SMEM_BYTES);
    if (e == cudaSuccess) {
        h->ctas = cl_fit(k_axi_mg_solve, CL_MAX_CTAS, AXI_THREADS, AXI_SMEM_BYTES);
        if (p->precision == GB_PRB_MIXED) e = axi_mer_create(h);
    }
    if (e != cudaSuccess) { gb_axi_destroy(h); gb_set_error("gb_axi_create: %s", cudaGetErrorString(e)); return GB_ERR_CUDA; }
    e = cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking);
    if (e != cudaSuccess) { gb_axi_destroy(h); gb_set_error("gb_axi_create: stream"); return GB_ERR_CUDA; }
    e = cudaStreamSynchronize(0);   // the creation's kernels and copies, not other instances' streams
    if (e != cudaSuccess) { gb_set_error("gb_axi_create: %s", cudaGetErrorString(e)); gb_axi_destroy(h); return GB_ERR_CUDA; }
    *out = h;
    return GB_OK;
}

// The annulus on a stretched grid: the state, its transport tables and the
// stretched multigrid; no uniform multigrid.
extern "C" int gb_axi_create_stretched(const gb_axi_params *p, const gb_axi_grid *g, gb_axi **out, int *nlev_out)
{
    if (!p || !g || !out || !g->levels || !g->z || !g->cz || !g->hw) {
        gb_set_error("gb_axi_create_stretched: null argument");
        return GB_ERR_INVALID;
    }
    *out = nullptr;
    const int nr = p->nr, nz = p->nz;
    const gb_str_level &L1 = g->levels[0];
    if (g->nlev < 1 || L1.n1 != nr || L1.n2 != nz || nr < 4 || nz < 4 || !L1.r || !L1.cr || !L1.crr || !L1.czz ||
        !(p->zmax > 0.0) || p->nrel < 1 || p->maxsweeps < 1 || p->Re == 0.0 ||
        (p->precision != GB_PRB_FP64 && p->precision != GB_PRB_MIXED)) {
        gb_set_error("gb_axi_create_stretched: level 1 must be %d x %d with all tables (nr, nz >= 4, zmax > 0, "
                     "Re != 0, FP64 or mixed)", nr, nz);
        return GB_ERR_INVALID;
    }
    gb_axi *h = new gb_axi();
    h->p = *p;
    AxiDev &d = h->dev;
    memset(&d, 0, sizeof(d));
    d.nr = nr;
    d.nz = nz;
    d.ld = nr + 1;
    d.nlev = g->nlev;
    d.stretched = 1;
    axi_scalars(h);
    int st = gb_str_create(g->nlev, g->levels, p->tolcon, p->maxsweeps, p->nrel, p->smoother, &h->str);
    if (st != GB_OK) { delete h; return st; }
    const size_t fsz = (size_t)d.ld * (size_t)(nz + 1);
    cudaError_t e = cudaMalloc(&h->fields, sizeof(double) * fsz * GB_A_COUNT);
    if (e != cudaSuccess) { gb_axi_destroy(h); gb_set_error("gb_axi_create_stretched: %s", cudaGetErrorString(e)); return GB_ERR_ALLOC; }
    cudaMemset(h->fields, 0, sizeof(double) * fsz * GB_A_COUNT);
    for (int q = 0; q < GB_A_COUNT; ++q) d.f[q] = h->fields + (size_t)q * fsz;
    const size_t ntab = (size_t)(nr + 1) + (nz + 1) + 3 * (size_t)(nr - 1) + 4 * (size_t)(nr - 1) + 3 * (size_t)(nz - 1) +
                        4 * (size_t)(nz - 1);
    e = cudaMalloc(&h->stab, sizeof(double) * ntab);
    if (e != cudaSuccess) { gb_axi_destroy(h); gb_set_error("gb_axi_create_stretched: tables"); return GB_ERR_ALLOC; }
    double *b = h->stab;
    auto put = [&](const double *src, size_t n) {
        double *dst = b;
        cudaMemcpy(dst, src, sizeof(double) * n, cudaMemcpyHostToDevice);
        b += n;
        return (const double *)dst;
    };
    d.st.r = put(L1.r, (size_t)nr + 1);
    d.st.z = put(g->z, (size_t)nz + 1);
    d.st.cr = put(L1.cr, 3 * (size_t)(nr - 1));
    d.st.crr = put(L1.crr, 4 * (size_t)(nr - 1));
    d.st.cz = put(g->cz, 3 * (size_t)(nz - 1));
    d.st.czz = put(L1.czz, 4 * (size_t)(nz - 1));
    for (int q = 0; q < 5; ++q) d.st.hw[q] = g->hw[q];
    e = cudaMalloc(&h->small, 4096);
    if (e != cudaSuccess) { gb_axi_destroy(h); gb_set_error("gb_axi_create_stretched: state"); return GB_ERR_ALLOC; }
    cudaMemset(h->small, 0, 4096);
    char *sm = (char *)h->small;
    d.heat = (double *)(sm + 0);
    d.errmax = (unsigned long long *)(sm + 64);
    d.abort = (int *)(sm + 128);
    d.status = (int *)(sm + 192);
    d.step_index = (int *)(sm + 256);
    e = cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaStreamSynchronize(0);
    if (e != cudaSuccess) { gb_axi_destroy(h); gb_set_error("gb_axi_create_stretched: %s", cudaGetErrorString(e)); return GB_ERR_CUDA; }
    if (nlev_out) *nlev_out = g->nlev;
    *out = h;
    return GB_OK;
}

extern "C" int gb_axi_set_field(gb_axi *h, int field, const double *host, int ld)
{
    if (!h || !host || field < 0 || field >= GB_A_COUNT || ld < h->dev.nr + 1) {
        gb_set_error("gb_axi_set_field: invalid argument");
        return GB_ERR_INVALID;
    }
    GB_CUDA_TRY(cudaMemcpy2DAsync(h->dev.f[field], sizeof(double) * h->dev.ld, host, sizeof(double) * (size_t)ld,
                                  sizeof(double) * (h->dev.nr + 1), h->dev.nz + 1, cudaMemcpyHostToDevice, h->stream));
    GB_CUDA_TRY(cudaStreamSynchronize(h->stream));
    return GB_OK;
}

extern "C" int gb_axi_get_field(gb_axi *h, int field, double *host, int ld)
{
    if (!h || !host || field < 0 || field >= GB_A_COUNT || ld < h->dev.nr + 1) {
        gb_set_error("gb_axi_get_field: invalid argument");
        return GB_ERR_INVALID;
    }
    GB_CUDA_TRY(cudaMemcpy2DAsync(host, sizeof(double) * (size_t)ld, h->dev.f[field], sizeof(double) * h->dev.ld,
                                  sizeof(double) * (h->dev.nr + 1), h->dev.nz + 1, cudaMemcpyDeviceToHost, h->stream));
    GB_CUDA_TRY(cudaStreamSynchronize(h->stream));
    return GB_OK;
}

extern "C" void *gb_axi_stream(gb_axi *h) { return h ? (void *)h->stream : nullptr; }

static const int AXI_TPB = 256;

static void axi_launch_vort_vel(gb_axi *h, int what, cudaStream_t s)
{
    const int n = (h->dev.nr - 1) * (h->dev.nz - 1);
    if (h->dev.stretched) k_axi_vort_vel<true><<<gb_ceil_div(n, AXI_TPB), AXI_TPB, 0, s>>>(h->dev, what);
    else k_axi_vort_vel<false><<<gb_ceil_div(n, AXI_TPB), AXI_TPB, 0, s>>>(h->dev, what);
}

static void axi_launch_temperature(gb_axi *h, cudaStream_t s)
{
    const int n = (h->dev.nr - 1) * (h->dev.nz + 1);
    if (h->dev.stretched) k_axi_temperature<true><<<gb_ceil_div(n, AXI_TPB), AXI_TPB, 0, s>>>(h->dev);
    else k_axi_temperature<false><<<gb_ceil_div(n, AXI_TPB), AXI_TPB, 0, s>>>(h->dev);
}

static void axi_launch_update(gb_axi *h, cudaStream_t s)
{
    const int n = (h->dev.nr + 1) * (h->dev.nz + 1);
    if (h->dev.stretched) k_axi_update<true><<<gb_ceil_div(n, AXI_TPB), AXI_TPB, 0, s>>>(h->dev);
    else k_axi_update<false><<<gb_ceil_div(n, AXI_TPB), AXI_TPB, 0, s>>>(h->dev);
}

static void axi_launch_heat(gb_axi *h, cudaStream_t s)
{
    if (h->dev.stretched) k_axi_heat<true><<<1, 256, sizeof(double) * (h->dev.nz + 1), s>>>(h->dev);
    else k_axi_heat<false><<<1, 256, sizeof(double) * (h->dev.nz + 1), s>>>(h->dev);
}

// The resident solve with the parameters a caller may have changed.
static MerDev axi_mer(const gb_axi *h)
{
    MerDev m = h->mer;
    m.tolcon = h->dev.tolcon;
    m.maxcycles = h->dev.maxsweeps;
    m.nrel = h->dev.nrel;
    return m;
}

[[nodiscard]] static cudaError_t axi_launch_mg(gb_axi *h, cudaStream_t s)
{
    const AxiDev &d = h->dev;
    if (d.stretched)
        return gb_str_launch_device(h->str, d.f[GB_A_phi], d.f[GB_A_omegn], d.status, d.abort,
                                    h->p.precision == GB_PRB_MIXED, d.tolcon, d.maxsweeps, d.nrel, d.mode, s);
    // the reference's line order is one chain of lines: one CTA
    const int ctas = d.mode == GB_SMOOTHER_LEX ? 1 : h->ctas;
    if (h->p.precision != GB_PRB_MIXED) return cl_launch(k_axi_mg_solve, 1, ctas, AXI_THREADS, AXI_SMEM_BYTES, s, d);
    if (d.mode == GB_SMOOTHER_ZEBRA && h->mer_most) return mer_launch(axi_mer(h), h->mer_ctas, s);
    return cl_launch(k_axi_mg_solve_mixed, 1, ctas, AXI_THREADS, AXI_SMEM_BYTES, s, d);
}

static int axi_sync(gb_axi *h, const char *what)
{
    cudaError_t e = cudaStreamSynchronize(h->stream);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) { gb_set_error("%s: %s", what, cudaGetErrorString(e)); return GB_ERR_CUDA; }
    return GB_OK;
}

static void axi_begin(gb_axi *h)
{
    axi_scalars(h);
    cudaMemsetAsync(h->dev.abort, 0, sizeof(int), h->stream);
}

extern "C" int gb_axi_vorticity(gb_axi *h)
{
    if (!h) return GB_ERR_INVALID;
    axi_begin(h);
    axi_launch_vort_vel(h, 1, h->stream);
    return axi_sync(h, "gb_axi_vorticity");
}

extern "C" int gb_axi_velocity(gb_axi *h)
{
    if (!h) return GB_ERR_INVALID;
    axi_begin(h);
    axi_launch_vort_vel(h, 2, h->stream);
    return axi_sync(h, "gb_axi_velocity");
}

extern "C" int gb_axi_temperature(gb_axi *h)
{
    if (!h) return GB_ERR_INVALID;
    axi_begin(h);
    axi_launch_temperature(h, h->stream);
    return axi_sync(h, "gb_axi_temperature");
}

extern "C" int gb_axi_poisson(gb_axi *h, int *sweeps)
{
    if (!h) return GB_ERR_INVALID;
    axi_begin(h);
    GB_CUDA_TRY(axi_launch_mg(h, h->stream));
    int st[2] = {0, 0};
    GB_CUDA_TRY(cudaMemcpyAsync(st, h->dev.status, sizeof(st), cudaMemcpyDeviceToHost, h->stream));
    int r = axi_sync(h, "gb_axi_poisson");
    if (r != GB_OK) return r;
    if (sweeps) *sweeps = st[1];
    return st[0];
}

extern "C" int gb_axi_update(gb_axi *h)
{
    if (!h) return GB_ERR_INVALID;
    axi_begin(h);
    axi_launch_update(h, h->stream);
    GB_CUDA_TRY(cudaMemsetAsync(h->dev.errmax, 0, 3 * sizeof(unsigned long long), h->stream));
    return axi_sync(h, "gb_axi_update");
}

extern "C" int gb_axi_heat(gb_axi *h, double *trans)
{
    if (!h) return GB_ERR_INVALID;
    axi_begin(h);
    axi_launch_heat(h, h->stream);
    double t = 0.0;
    GB_CUDA_TRY(cudaMemcpyAsync(&t, h->dev.heat, sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    int r = axi_sync(h, "gb_axi_heat");
    if (trans) *trans = t;
    return r;
}

static int axi_build_graph(gb_axi *h)
{
    cudaGraph_t g;
    GB_CUDA_TRY(cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal));
    axi_launch_vort_vel(h, 3, h->stream);
    axi_launch_temperature(h, h->stream);
    const cudaError_t e = axi_launch_mg(h, h->stream);
    axi_launch_update(h, h->stream);
    axi_launch_heat(h, h->stream);
    k_axi_record<<<1, 32, 0, h->stream>>>(h->dev);
    const cudaError_t ended = cudaStreamEndCapture(h->stream, &g);   // also ends one that failed
    if (e != cudaSuccess && ended == cudaSuccess) cudaGraphDestroy(g);
    GB_CUDA_TRY(e);
    GB_CUDA_TRY(ended);
    GB_CUDA_TRY(cudaGraphInstantiate(&h->graph, g, 0));
    cudaGraphDestroy(g);
    return GB_OK;
}

// Asynchronous stepping (as for the 2D drivers).
extern "C" int gb_axi_run_begin(gb_axi *h, int nsteps_total)
{
    if (!h || nsteps_total < 0) { gb_set_error("gb_axi_run_begin: invalid argument"); return GB_ERR_INVALID; }
    AxiDev &d = h->dev;
    const int cap = nsteps_total > 0 ? nsteps_total : 1;
    if (h->hist_cap < cap) {
        cudaFree(h->hist);
        h->hist = nullptr;
        GB_CUDA_TRY(cudaMalloc(&h->hist, (sizeof(double) + sizeof(int)) * (size_t)cap));
        h->hist_cap = cap;
        if (h->graph) { cudaGraphExecDestroy(h->graph); h->graph = nullptr; }
    }
    d.nu_hist = (double *)h->hist;
    d.sweep_hist = (int *)((double *)h->hist + h->hist_cap);
    d.hist_cap = h->hist_cap;
    if (memcmp(&h->graph_params, &h->p, sizeof(gb_axi_params)) != 0) {
        if (h->graph) { cudaGraphExecDestroy(h->graph); h->graph = nullptr; }
        h->graph_params = h->p;
        axi_scalars(h);
    }
    GB_CUDA_TRY(cudaMemsetAsync(d.abort, 0, sizeof(int), h->stream));
    GB_CUDA_TRY(cudaMemsetAsync(d.step_index, 0, sizeof(int), h->stream));
    GB_CUDA_TRY(cudaMemsetAsync(d.errmax, 0, 3 * sizeof(unsigned long long), h->stream));
    return GB_OK;
}

extern "C" int gb_axi_run_enqueue(gb_axi *h, int nsteps)
{
    if (!h || nsteps < 0) { gb_set_error("gb_axi_run_enqueue: invalid argument"); return GB_ERR_INVALID; }
    int st;
    if (!h->graph && (st = axi_build_graph(h)) != GB_OK) return st;
    for (int s = 0; s < nsteps; ++s) GB_CUDA_TRY(cudaGraphLaunch(h->graph, h->stream));
    return GB_OK;
}

extern "C" int gb_axi_run_query(gb_axi *h)
{
    if (!h) return -GB_ERR_INVALID;
    const cudaError_t e = cudaStreamQuery(h->stream);
    if (e == cudaSuccess) return 1;
    if (e == cudaErrorNotReady) { cudaGetLastError(); return 0; }
    gb_set_error("gb_axi_run_query: %s", cudaGetErrorString(e));
    return -GB_ERR_CUDA;
}

extern "C" int gb_axi_run_end(gb_axi *h, int nsteps, double *nu, int *sweeps, int *steps_done)
{
    if (!h || nsteps < 0 || nsteps > h->hist_cap) { gb_set_error("gb_axi_run_end: invalid argument"); return GB_ERR_INVALID; }
    AxiDev &d = h->dev;
    int info[2] = {0, 0}, stat[2] = {0, 0};
    GB_CUDA_TRY(cudaMemcpyAsync(&info[0], d.step_index, sizeof(int), cudaMemcpyDeviceToHost, h->stream));
    GB_CUDA_TRY(cudaMemcpyAsync(&info[1], d.abort, sizeof(int), cudaMemcpyDeviceToHost, h->stream));
    GB_CUDA_TRY(cudaMemcpyAsync(stat, d.status, sizeof(stat), cudaMemcpyDeviceToHost, h->stream));
    std::vector<double> nuh((size_t)nsteps + 1);
    std::vector<int> swh((size_t)nsteps + 1);
    if (nsteps > 0) {
        GB_CUDA_TRY(cudaMemcpyAsync(nuh.data(), d.nu_hist, sizeof(double) * nsteps, cudaMemcpyDeviceToHost, h->stream));
        GB_CUDA_TRY(cudaMemcpyAsync(swh.data(), d.sweep_hist, sizeof(int) * nsteps, cudaMemcpyDeviceToHost, h->stream));
    }
    int st = axi_sync(h, "gb_axi_run_end");
    if (st != GB_OK) return st;
    if (nu) memcpy(nu, nuh.data(), sizeof(double) * nsteps);
    if (sweeps) memcpy(sweeps, swh.data(), sizeof(int) * nsteps);
    if (steps_done) *steps_done = info[0];
    if (info[1] == 1) {
        gb_set_error("gb_axi_step: multigrid failed at step %d (status %d)", info[0] + 1, stat[0]);
        return stat[0];
    }
    return GB_OK;
}

extern "C" int gb_axi_step(gb_axi *h, int nsteps, double *nu, int *sweeps, int *steps_done)
{
    if (!h || nsteps < 0) { gb_set_error("gb_axi_step: invalid argument"); return GB_ERR_INVALID; }
    if (steps_done) *steps_done = 0;
    if (nsteps == 0) return GB_OK;
    int st = gb_axi_run_begin(h, nsteps);
    if (st == GB_OK) st = gb_axi_run_enqueue(h, nsteps);
    if (st != GB_OK) return st;
    return gb_axi_run_end(h, nsteps, nu, sweeps, steps_done);
}

// ---------------------------------------------------------------------------
// Gangs of annulus instances of different grid sizes stepped together (as
// the PRB gangs in prb.cu): each phase of a step is one launch over all
// members' blocks, the streamfunction solves up to three (gb_axi_gang), a
// cluster per member; every member runs its own kernel bodies, so its results are
// bit-identical to stepping it alone.  A member whose step index reaches
// its step count sets its abort flag to GB_RUN_DONE.
// ---------------------------------------------------------------------------
enum AxiGangPhase { AG_VV, AG_T, AG_UPD, AG_HEAT, AG_REC, AG_COUNT };

struct AxiGangTab {
    const AxiDev *dev;    // [n]
    const int *off;       // [AG_COUNT][n + 1]
    const int *limit;     // [n]
    int n;
};

__device__ __forceinline__ int axi_gang_member(const int *off, int n, int b)
{
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (off[mid] <= b) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

template <int PH>
__global__ void k_axi_gang(AxiGangTab g)
{
    const int *off = g.off + (size_t)PH * (g.n + 1);
    const int m = axi_gang_member(off, g.n, blockIdx.x);
    const AxiDev &d = g.dev[m];
    const int b = blockIdx.x - off[m];
    switch (PH) {
    case AG_VV: k_axi_vort_vel_body<false>(d, 3, b); break;
    case AG_T: k_axi_temperature_body<false>(d, b); break;
    case AG_UPD: k_axi_update_body<false>(d, b); break;
    case AG_HEAT: k_axi_heat_body<false>(d, b); break;
    case AG_REC:
        k_axi_record_body(d, b);
        if (threadIdx.x == 0 && b == 0 && *d.abort == 0 && *d.step_index >= g.limit[m]) *d.abort = GB_RUN_DONE;
        break;
    default: break;
    }
}

// The solves of the members listed in `who`, a cluster each; registers as the
// single instance's kernels, free of spills.
template <bool MIXED>
__global__ void __maxnreg__(255) k_axi_gang_mg(AxiGangTab g, const int *who)
{
    const AxiDev &d = g.dev[who[blockIdx.x / cooperative_groups::this_cluster().num_blocks()]];
    if (MIXED) k_axi_mg_solve_mixed_body(d);
    else k_axi_mg_solve_body(d);
}

// The streamfunction solves of a gang step: every member's as one cluster,
// the resident ones of a mixed gang in one launch, the others in another per
// line order (the reference's order takes one CTA).  A cluster holds as many
// CTAs as leave every member its own SMs, at least what the largest resident
// member's arrays need; the results do not depend on it.
struct gb_axi_gang {
    int n = 0, mixed = 0;
    AxiDev *d_dev = nullptr;
    int *d_off = nullptr, *d_limit = nullptr, *d_who = nullptr;
    MerDev *d_mer = nullptr;
    int nmer = 0, mer_ctas = 0;
    size_t mer_smem = 0;
    int nz = 0, nlex = 0, z_ctas = 1;   // members on global memory: zebra, reference order (d_who in this order)
    int blocks[AG_COUNT], threads[AG_COUNT];
    size_t heat_smem = 0;
    cudaStream_t stream = nullptr;
    cudaGraphExec_t graph = nullptr;
};

extern "C" int gb_axi_gang_destroy(gb_axi_gang *g)
{
    if (!g) return GB_OK;
    if (g->graph) cudaGraphExecDestroy(g->graph);
    cudaFree(g->d_dev);
    cudaFree(g->d_off);
    cudaFree(g->d_limit);
    cudaFree(g->d_who);
    cudaFree(g->d_mer);
    if (g->stream) cudaStreamDestroy(g->stream);
    delete g;
    return GB_OK;
}

extern "C" int gb_axi_gang_create(gb_axi *const *members, const int *nsteps_total, int n, gb_axi_gang **out)
{
    if (!members || !nsteps_total || n < 1 || !out) {
        gb_set_error("gb_axi_gang_create: invalid argument");
        return GB_ERR_INVALID;
    }
    *out = nullptr;
    const int mixed = members[0]->p.precision == GB_PRB_MIXED;
    for (int q = 0; q < n; ++q) {
        const gb_axi *h = members[q];
        if (!h || h->dev.stretched || (h->p.precision == GB_PRB_MIXED) != (mixed != 0) || nsteps_total[q] < 0 ||
            nsteps_total[q] > h->hist_cap) {
            gb_set_error("gb_axi_gang_create: member %d must be a uniform-grid instance of the gang's precision, after "
                         "gb_axi_run_begin with at least its step count", q);
            return GB_ERR_INVALID;
        }
    }
    gb_axi_gang *g = new gb_axi_gang();
    g->n = n;
    g->mixed = mixed;
    const int tpb[AG_COUNT] = {AXI_TPB, AXI_TPB, AXI_TPB, 256, 32};
    std::vector<int> off((size_t)AG_COUNT * (n + 1));
    std::vector<AxiDev> devs(n);
    for (int ph = 0; ph < AG_COUNT; ++ph) {
        g->threads[ph] = tpb[ph];
        g->blocks[ph] = 0;
    }
    for (int q = 0; q < n; ++q) {
        gb_axi *h = members[q];
        axi_scalars(h);
        devs[q] = h->dev;
        const size_t nr = h->dev.nr, nz = h->dev.nz;
        const int nb[AG_COUNT] = {(int)gb_ceil_div((nr - 1) * (nz - 1), AXI_TPB), (int)gb_ceil_div((nr - 1) * (nz + 1), AXI_TPB),
                                  (int)gb_ceil_div((nr + 1) * (nz + 1), AXI_TPB), 1, 1};
        for (int ph = 0; ph < AG_COUNT; ++ph) {
            off[(size_t)ph * (n + 1) + q] = g->blocks[ph];
            g->blocks[ph] += nb[ph];
        }
        g->heat_smem = std::max(g->heat_smem, sizeof(double) * (nz + 1));
    }
    for (int ph = 0; ph < AG_COUNT; ++ph) off[(size_t)ph * (n + 1) + n] = g->blocks[ph];
    std::vector<MerDev> mers;
    std::vector<int> who, lex, res;
    int most = CL_MAX_CTAS;
    const int sms = gb_sm_count();
    for (int q = 0; q < n; ++q) {
        if (mixed && members[q]->p.smoother == GB_SMOOTHER_ZEBRA && members[q]->mer_most) {
            res.push_back(q);
            mers.push_back(axi_mer(members[q]));
            most = std::min(most, members[q]->mer_most);
        } else if (members[q]->p.smoother == GB_SMOOTHER_LEX) {
            lex.push_back(q);
        } else {
            who.push_back(q);
        }
    }
    auto per_member = [&](int members_) {
        int c = CL_MAX_CTAS;
        while (c > 1 && c * members_ > sms) c >>= 1;
        return c;
    };
    if (!mers.empty()) {
        std::vector<char> fits(mers.size());
        g->mer_ctas = mer_plan_many(mers.data(), (int)mers.size(), std::min(most, per_member((int)mers.size())), most, &g->mer_smem, fits.data());
        for (size_t q = 0; q < mers.size(); ++q) {
            if (fits[q]) mers[g->nmer++] = mers[q];
            else who.push_back(res[q]);
        }
        mers.resize(g->nmer);
    }
    g->nz = (int)who.size();
    g->nlex = (int)lex.size();
    who.insert(who.end(), lex.begin(), lex.end());
    if (g->nz) g->z_ctas = std::min(members[who[0]]->ctas, per_member(g->nz));
#define GTRY(x)                                                                   \
    do {                                                                          \
        cudaError_t _e = (x);                                                     \
        if (_e != cudaSuccess) {                                                  \
            gb_set_error("gb_axi_gang_create: %s: %s", #x, cudaGetErrorString(_e)); \
            gb_axi_gang_destroy(g);                                               \
            return GB_ERR_CUDA;                                                   \
        }                                                                         \
    } while (0)
    GTRY(cudaMalloc(&g->d_dev, sizeof(AxiDev) * n));
    GTRY(cudaMalloc(&g->d_off, sizeof(int) * off.size()));
    GTRY(cudaMalloc(&g->d_limit, sizeof(int) * n));
    GTRY(cudaMemcpy(g->d_dev, devs.data(), sizeof(AxiDev) * n, cudaMemcpyHostToDevice));
    GTRY(cudaMemcpy(g->d_off, off.data(), sizeof(int) * off.size(), cudaMemcpyHostToDevice));
    GTRY(cudaMemcpy(g->d_limit, nsteps_total, sizeof(int) * n, cudaMemcpyHostToDevice));
    if (!who.empty()) {
        GTRY(cudaMalloc(&g->d_who, sizeof(int) * who.size()));
        GTRY(cudaMemcpy(g->d_who, who.data(), sizeof(int) * who.size(), cudaMemcpyHostToDevice));
        GTRY(mixed ? cl_prepare(k_axi_gang_mg<true>, AXI_SMEM_BYTES) : cl_prepare(k_axi_gang_mg<false>, AXI_SMEM_BYTES));
    }
    if (g->nmer) {
        GTRY(cudaMalloc(&g->d_mer, sizeof(MerDev) * mers.size()));
        GTRY(cudaMemcpy(g->d_mer, mers.data(), sizeof(MerDev) * mers.size(), cudaMemcpyHostToDevice));
    }
    for (int q = 0; q < n; ++q) GTRY(cudaStreamSynchronize(members[q]->stream));
    GTRY(cudaStreamCreateWithFlags(&g->stream, cudaStreamNonBlocking));
    if (g->heat_smem > 48 * 1024)
        GTRY(cudaFuncSetAttribute(k_axi_gang<AG_HEAT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)g->heat_smem));
#undef GTRY
    *out = g;
    return GB_OK;
}

// Queues nsteps steps of every member (one CUDA graph launch per step) on
// `stream` (NULL: the gang's own).
extern "C" int gb_axi_gang_enqueue(gb_axi_gang *g, int nsteps, void *stream)
{
    if (!g || nsteps < 0) { gb_set_error("gb_axi_gang_enqueue: invalid argument"); return GB_ERR_INVALID; }
    cudaStream_t s = stream ? (cudaStream_t)stream : g->stream;
    if (!g->graph) {
        AxiGangTab t{g->d_dev, g->d_off, g->d_limit, g->n};
        cudaGraph_t gr;
        cudaStream_t cs = g->stream;
        GB_CUDA_TRY(cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal));
        k_axi_gang<AG_VV><<<g->blocks[AG_VV], g->threads[AG_VV], 0, cs>>>(t);
        k_axi_gang<AG_T><<<g->blocks[AG_T], g->threads[AG_T], 0, cs>>>(t);
        cudaError_t e = cudaSuccess;
        if (g->nmer) e = mer_launch_many(g->d_mer, g->nmer, 0, g->mer_ctas, g->mer_smem, cs);
        auto solves = [&](int count, int ctas, const int *who) {
            if (!count || e != cudaSuccess) return;
            e = g->mixed ? cl_launch(k_axi_gang_mg<true>, count, ctas, AXI_THREADS, AXI_SMEM_BYTES, cs, t, who)
                         : cl_launch(k_axi_gang_mg<false>, count, ctas, AXI_THREADS, AXI_SMEM_BYTES, cs, t, who);
        };
        solves(g->nz, g->z_ctas, g->d_who);
        solves(g->nlex, 1, g->d_who + g->nz);
        k_axi_gang<AG_UPD><<<g->blocks[AG_UPD], g->threads[AG_UPD], 0, cs>>>(t);
        k_axi_gang<AG_HEAT><<<g->blocks[AG_HEAT], g->threads[AG_HEAT], g->heat_smem, cs>>>(t);
        k_axi_gang<AG_REC><<<g->blocks[AG_REC], g->threads[AG_REC], 0, cs>>>(t);
        const cudaError_t ended = cudaStreamEndCapture(cs, &gr);
        if (e != cudaSuccess && ended == cudaSuccess) cudaGraphDestroy(gr);
        GB_CUDA_TRY(e);
        GB_CUDA_TRY(ended);
        GB_CUDA_TRY(cudaGraphInstantiate(&g->graph, gr, 0));
        cudaGraphDestroy(gr);
    }
    for (int k = 0; k < nsteps; ++k) GB_CUDA_TRY(cudaGraphLaunch(g->graph, s));
    return GB_OK;
}

extern "C" void *gb_axi_gang_stream(gb_axi_gang *g) { return g ? (void *)g->stream : nullptr; }

extern "C" int gb_axi_gang_query(gb_axi_gang *g)
{
    if (!g) return -GB_ERR_INVALID;
    const cudaError_t e = cudaStreamQuery(g->stream);
    if (e == cudaSuccess) return 1;
    if (e == cudaErrorNotReady) { cudaGetLastError(); return 0; }
    gb_set_error("gb_axi_gang_query: %s", cudaGetErrorString(e));
    return -GB_ERR_CUDA;
}
