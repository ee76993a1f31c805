// Velocity multigrid (prb_mg.cu's solves, the same bits) with every level in
// the shared memory of one thread-block cluster.
//
// A sweep of the 129 x 65 layer is about 64 short passes over four levels; on
// global memory each paid L2 round trips (5 k cycles a pass, whatever its
// size), as much as the FP64 eliminations themselves and ten times the FP32
// ones.  Here the lines k of every level are spread over the CTAs in
// contiguous blocks, so that a coarse line lives where its fine lines do; a
// line's right-hand side needs only the lines next to it, which are the
// CTA's own but at its block's two edges (distributed shared memory).  Factors
// and radii are loaded once per solve.
//
// FP64 (T = double): a line is eliminated in place by one thread, in the
// reference's order.  FP32 (the mixed solve's correction cycles): by up to 32
// lanes (warpline.cuh); the FP64 iterate stays in global memory.
//
// Measured on the 129 x 65 layer (GB300, three steps at tolerance 2e-6): FP64 25.6
// ms on one CTA (from global memory), 14.9 on a cluster of 16, most of it
// eliminations; mixed 8.7 and 5.9.
#include <string.h>

#include <algorithm>

#include "banded.cuh"
#include "cluster.cuh"
#include "gbcommon.cuh"
#include "mg_op.cuh"
#include "prb_internal.cuh"
#include "warpline.cuh"

#define PL_THREADS 256
#define PL_SMEM_MAX (220 * 1024)

// Column i of a line: plain in FP64 (one thread per line, odd pitch), a
// lane's rows padded to an odd stride in FP32.
template <class T> __host__ __device__ __forceinline__ int pl_col(int lg, int i)
{
    return sizeof(T) == 8 ? i : i < 1 ? i : i + ((i - 1) >> lg);
}

__device__ __forceinline__ float pl_load(unsigned addr, float)
{
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ double pl_load(unsigned addr, double)
{
    double v;
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ void pl_store(unsigned addr, float v) { asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory"); }
__device__ __forceinline__ void pl_store(unsigned addr, double v) { asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory"); }

// One level as a CTA sees it.
template <class T> struct PlView {
    int which, polar, xwall, n1, n3, rp, pitch, lg;
    int k0, k1;                 // own lines k0 .. k1 - 1, at local index k - k0 + 1 (line 0: local 0 of CTA 0)
    int klast;                  // last line that is solved
    T hhri, hhpi, hri;
    T *v, *f;                   // this CTA's
    const T *fac, *rvi, *rvq;
    const unsigned *rows;       // addresses of the lines of v, k = 0 .. n3
    __device__ __forceinline__ PlView(const MgEq &E, int l, const Cluster &cl)
    {
        extern __shared__ __align__(16) unsigned char s_pl[];
        const MgLevel &L = E.lev[l];
        which = E.which;
        polar = E.polar;
        xwall = E.xwall;
        n1 = L.n1;
        n3 = L.n3;
        rp = L.rp;
        pitch = L.pitch;
        lg = wl_log2m(which == 2 ? n1 : n1 - 1);
        k0 = cl.rank * rp + 1;
        k1 = min(k0 + rp, n3 + 1);
        klast = xwall && which == 2 ? n3 - 1 : n3;   // velvor2dhorconvtank.f:1170, :1216
        hhri = (T)L.hhri;
        hhpi = (T)L.hhpi;
        hri = (T)L.hri;
        v = (T *)(s_pl + L.o_v);
        f = (T *)(s_pl + L.o_f);
        fac = (const T *)(s_pl + L.o_fac);
        rvi = (const T *)(s_pl + L.o_rv);
        rvq = rvi + n1 + 2;
        rows = (const unsigned *)(s_pl + L.o_rows);
    }
    __device__ __forceinline__ int after(int k) const { return k == n3 ? (xwall ? 0 : 1) : k + 1; }
    __device__ __forceinline__ T *own(T *a, int k) const { return a + (k - k0 + 1) * pitch; }
    __device__ __forceinline__ int col(int i) const { return pl_col<T>(lg, i); }
    // row i of line k of v, wherever it lives
    __device__ __forceinline__ T at(int k, int i) const { return pl_load(rows[k] + (unsigned)sizeof(T) * col(i), T(0)); }
};

// One colour (lines first, first + 2, ...) of a sweep on level l in FP64.
__device__ __noinline__ void pl_colour64(const MgEq &E, int l, int first)
{
    const Cluster cl = Cluster::self();
    const PlView<double> L(E, l, cl);
    const int n = L.which == 2 ? L.n1 : L.n1 - 1;
    const int kb = L.k0 + ((first - L.k0) & 1), ke = min(L.k1, L.klast + 1);   // own lines kb, kb + 2, ... < ke
    const int nl = kb < ke ? (ke - 1 - kb) / 2 + 1 : 0;
    // right-hand sides in place (nothing reads this colour's lines now)
    const RowSplit split(n);
    for (int idx = threadIdx.x; idx < nl * n; idx += PL_THREADS) {
        int t, q;
        split(idx, t, q);
        const int k = kb + 2 * t, i = q + 1;
        double r = -(L.at(L.after(k), i) + L.at(k - 1, i)) * L.hhpi;
        if (L.polar) r = r * L.rvq[i];
        L.own(L.v, k)[i] = r + L.own(L.f, k)[i];
    }
    __syncthreads();
    for (int t = threadIdx.x; t < nl; t += PL_THREADS) {
        double *x = L.own(L.v, kb + 2 * t) + 1;
        if (L.which == 2) pdma_staged<2>(L.fac, n, x, 1);
        else tdma_staged<2>(L.fac, n, x, 1);
    }
    if (ke - 1 == L.n3 && nl > 0 && ((L.n3 - kb) & 1) == 0) {   // line n3 was solved: k = 0 repeats it
        __syncthreads();
        for (int i = 1 + threadIdx.x; i <= n; i += PL_THREADS) pl_store(L.rows[0] + 8u * L.col(i), L.xwall ? 0.0 : L.own(L.v, L.n3)[i]);
    }
    cl.sync();
}

// The relaxations' sweeps on level l, colour by colour (lines 1, 3, ... and 2,
// 4, ...).  One table serves all lines of a level: in FP32 the lanes load their
// rows of it once for all the sweeps of a visit (layer 129 x 65 mixed, four
// steps: 13.5 -> 12.4 ms); the FP64 chains gain nothing from it.
__device__ __noinline__ void pl_sweeps32(const MgEq &E, int l)
{
    using T = float;
    const Cluster cl = Cluster::self();
    const PlView<T> L(E, l, cl);
    const int n = L.which == 2 ? L.n1 : L.n1 - 1, phases = 2 * E.nrelax;
    const int ke = min(L.k1, L.klast + 1);
    auto seam = [&](int i, T x) { pl_store(L.rows[0] + (unsigned)sizeof(T) * L.col(i), L.xwall ? T(0) : x); };
    // own lines of phase ph: kb, kb + 2, ... < ke, nl of them
    auto begin = [&](int ph) { return L.k0 + ((1 + ph - L.k0) & 1); };
    auto count = [&](int kb) { return kb < ke ? (ke - 1 - kb) / 2 + 1 : 0; };
    auto lines = [&](auto m, auto penta) {
        constexpr int M = decltype(m)::value;
        constexpr bool PENTA = decltype(penta)::value;
        const int lw = wl_log2w(n), per = 32 >> lw;
        const int sub = (threadIdx.x & 31) >> lw, lane = threadIdx.x & ((1 << lw) - 1);
        const int slot = (threadIdx.x >> 5) * per + sub, nslots = (PL_THREADS / 32) * per;
        WlTab<M, PENTA> tab;
        tab.load((const float *)L.fac, lw);
#pragma unroll 1
        for (int ph = 0; ph < phases; ++ph) {
            const int kb = begin(ph), nl = count(kb);
            for (int tb = 0; tb < nl; tb += nslots) {
                if (tb + slot - sub >= nl) continue;   // no line for this warp
                const bool live = tb + slot < nl;
                const int k = kb + 2 * (live ? tb + slot : tb + slot - sub);   // idle groups repeat a line and store nothing
                const int c0 = 1 + lane * (M + 1);
                const unsigned ra = L.rows[L.after(k)] + 4 * c0, rm = L.rows[k - 1] + 4 * c0;
                const T *fr = L.own(L.f, k) + c0;
                T t[M], a[M], b[M];
#pragma unroll
                for (int u = 0; u < M; ++u) {
                    a[u] = pl_load(ra + 4 * u, T(0));
                    b[u] = pl_load(rm + 4 * u, T(0));
                }
#pragma unroll
                for (int u = 0; u < M; ++u) {
                    T r = -(a[u] + b[u]) * L.hhpi;
                    if (L.polar) r = r * L.rvq[min(lane * M + u + 1, L.n1 + 1)];
                    t[u] = lane * M + u < n ? r + fr[u] : T(0);
                }
                tab.solve(n, t);
                if (live) {
                    T *vr = L.own(L.v, k) + c0;
#pragma unroll
                    for (int u = 0; u < M; ++u)
                        if (lane * M + u < n) {
                            vr[u] = t[u];
                            if (k == L.n3) seam(lane * M + u + 1, t[u]);
                        }
                }
            }
            cl.sync();
        }
    };
    if (L.lg == 3) {
        if (L.which == 2) lines(std::integral_constant<int, 8>(), std::true_type());
        else lines(std::integral_constant<int, 8>(), std::false_type());
    } else {
        if (L.which == 2) lines(std::integral_constant<int, 16>(), std::true_type());
        else lines(std::integral_constant<int, 16>(), std::false_type());
    }
}
template <class T> __device__ __forceinline__ void pl_sweeps(const MgEq &E, int l)
{
    if constexpr (sizeof(T) == 4) {
        pl_sweeps32(E, l);
    } else {
        for (int irel = 0; irel < E.nrelax; ++irel)
            for (int c = 1; c <= 2; ++c) pl_colour64(E, l, c);
    }
}

// The residual of level l into rc (own lines; not followed by a barrier): its
// largest magnitude over the calling thread's points and whether one is a NaN.
template <class T> __device__ __noinline__ T pl_residual(const MgEq &E, int l, int *nan_out)
{
    extern __shared__ __align__(16) unsigned char s_pl[];
    const Cluster cl = Cluster::self();
    const PlView<T> L(E, l, cl);
    T *rc = (T *)(s_pl + E.o_rc);
    const int n = L.which == 2 ? L.n1 : L.n1 - 1;
    const int nl = min(L.k1, L.klast + 1) - L.k0;
    const RowSplit split(n);
    T m = T(0);
    int nan = 0;
    for (int idx = threadIdx.x; idx < nl * n; idx += PL_THREADS) {
        int t, i;
        split(idx, t, i);
        ++i;
        const int k = L.k0 + t;
        const T *row = L.own(L.v, k);
        T r = mg_apply_op<T>([&](int q) { return row[L.col(q)]; }, L.at(L.after(k), i), L.at(k - 1, i), i, L.which, L.polar, L.n1,
                             L.hhri, L.hhpi, L.hri, L.rvi, L.rvq);
        r = L.own(L.f, k)[L.col(i)] - r;
        L.own(rc, k)[L.col(i)] = r;
        r = fabs(r);
        if (r != r) nan = 1;
        if (r > m) m = r;
    }
    *nan_out = nan;
    return m;
}

// corser (PRB:2603-2718); the annulus keeps the residual stored at the seam
// line n3c of the coarse level.  The coarse solution is cleared.
template <class T> __device__ __noinline__ void pl_corser(const MgEq &E, int l)
{
    const Cluster cl = Cluster::self();
    const PlView<T> F(E, l, cl), L(E, l + 1, cl);
    const int to_rc = E.o_rc - E.lev[l].o_v;   // rc's lines lie as v's do
    const int nl = L.k1 - L.k0;
    const RowSplit split(L.n1);
    for (int idx = threadIdx.x; idx < nl * L.n1; idx += PL_THREADS) {
        int t, i;
        split(idx, t, i);
        ++i;
        const int k = L.k0 + t;
        T r = T(0);
        auto rc = [&](int kk, int ii) { return pl_load(F.rows[kk] + to_rc + (unsigned)sizeof(T) * F.col(ii), T(0)); };
        if (i <= L.n1 - 1 && k <= L.n3 - 1) {
            const int ii = 2 * i, kk = 2 * k;
            r = mg_full_weight(rc(kk, ii), rc(kk, ii + 1), rc(kk, ii - 1), rc(kk + 1, ii), rc(kk - 1, ii), rc(kk + 1, ii + 1),
                               rc(kk - 1, ii + 1), rc(kk + 1, ii - 1), rc(kk - 1, ii - 1));
        } else if (E.seam_keep && i <= L.n1 - 1) {
            r = rc(k, i);
        }
        L.own(L.f, k)[L.col(i)] = r;
        L.own(L.v, k)[L.col(i)] = T(0);
    }
    if (cl.rank == 0)
        for (int i = threadIdx.x; i <= L.n1; i += PL_THREADS) L.v[L.col(i)] = T(0);
    cl.sync();
}

// finer (PRB:2721-2803): bilinear prolongation added, line 0 with the first CTA.
template <class T> __device__ __noinline__ void pl_finer(const MgEq &E, int l)
{
    const Cluster cl = Cluster::self();
    const PlView<T> C(E, l, cl), L(E, l - 1, cl);
    const int kb = cl.rank == 0 ? 0 : L.k0, nl = L.k1 - kb;
    const RowSplit split(L.n1);
    for (int idx = threadIdx.x; idx < nl * L.n1; idx += PL_THREADS) {
        int t, i;
        split(idx, t, i);
        ++i;
        const int k = kb + t;
        const bool io = i & 1, ko = k & 1;
        const int i1 = i >> 1, k1 = k >> 1;
        const T p = mg_prolong(io, ko, C.at(k1, i1), io ? C.at(k1, i1 + 1) : T(0), ko ? C.at(k1 + 1, i1) : T(0),
                               io && ko ? C.at(k1 + 1, i1 + 1) : T(0));
        T *v = L.own(L.v, k) + L.col(i);
        *v = p + *v;
    }
    cl.sync();
}

// mg_legs of prb_mg.cu
template <class T, class Relax> __device__ __forceinline__ void pl_legs(const MgEq &E, Relax relax)
{
    const int nlev = E.nlev;
    if (nlev < 2) return;
    for (int leg = 0; leg < nlev; ++leg) {
        // up to level nlev - leg (not before the first), down to the coarsest
        const int top = leg == 0 ? 1 : nlev - leg;
        if (leg > 0)
            for (int l = nlev; l > top; --l) {
                pl_finer<T>(E, l);
                relax(l - 1, l - 1 == top);
            }
        for (int l = top; l <= nlev - 1; ++l) {
            pl_corser<T>(E, l);
            relax(l + 1, l + 1 < nlev);
        }
    }
    for (int l = nlev; l >= 2; --l) {
        pl_finer<T>(E, l);
        relax(l - 1, false);
    }
}

// Shared memory of the solve: zeroed, then the descriptor, factors, radii and
// line addresses.
template <class T> __device__ __forceinline__ void pl_setup(MgEq &E, const MgEq &src, const Cluster &cl)
{
    extern __shared__ __align__(16) unsigned char s_pl[];
    for (int q = threadIdx.x; q < (int)(sizeof(MgEq) / 4); q += PL_THREADS) ((unsigned *)&E)[q] = ((const unsigned *)&src)[q];
    __syncthreads();
    for (int q = threadIdx.x; q < E.smem / 4; q += PL_THREADS) ((unsigned *)s_pl)[q] = 0u;
    __syncthreads();
    for (int l = 1; l <= E.nlev; ++l) {
        const MgLevel &L = E.lev[l];
        const int n = E.which == 2 ? L.n1 : L.n1 - 1;
        T *fac = (T *)(s_pl + L.o_fac), *rv = (T *)(s_pl + L.o_rv), *v = (T *)(s_pl + L.o_v);
        unsigned *rows = (unsigned *)(s_pl + L.o_rows);
        if constexpr (sizeof(T) == 8) {
            const int len = (int)(E.which == 2 ? pdma_fac_len(n) : tdma_fac_len(n));
            for (int q = threadIdx.x; q < len; q += PL_THREADS) fac[q] = L.fac[q];
            for (int q = threadIdx.x; q <= L.n1 + 1; q += PL_THREADS) {
                rv[q] = L.rvi[q];
                rv[L.n1 + 2 + q] = L.rvq[q];
            }
        } else {
            const int len = (int)(E.which == 2 ? pdma32_len(n) : tdma32_len(n));
            for (int q = threadIdx.x; q < len; q += PL_THREADS) fac[q] = L.fac32[q];
            for (int q = threadIdx.x; q <= L.n1 + 1; q += PL_THREADS) {
                rv[q] = L.rvi32[q];
                rv[L.n1 + 2 + q] = L.rvq32[q];
            }
        }
        for (int k = threadIdx.x; k <= L.n3; k += PL_THREADS) {
            const int o = min((max(k, 1) - 1) / L.rp, cl.size - 1);
            const unsigned a = (unsigned)__cvta_generic_to_shared(v + (k - o * L.rp) * L.pitch);
            unsigned p = a;
            if (o != cl.rank) asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(p) : "r"(a), "r"(o));
            rows[k] = p;
        }
    }
    __syncthreads();
}

// poisson2 / poisson3 (PRB:1796-1927 / PRB:1930-2059): k_mg_solve.
__global__ void __maxnreg__(255) k_pl_solve(const MgEq *eqs, int first_eq)
{
    extern __shared__ __align__(16) unsigned char s_pl[];
    __shared__ ClMaxState s_max;
    __shared__ MgEq E;
    const Cluster cl = Cluster::self();
    const MgEq &src = eqs[first_eq + blockIdx.x / cl.size];
    if (*src.abort == GB_RUN_DONE) return;   // a gang member past its last step (the same for every CTA)
    pl_setup<double>(E, src, cl);
    int turn = 0;
    const int ld = E.ld, np = E.np, nlev = E.nlev;
    const int imax = (E.which == 2) ? E.nr + 1 : E.nr;
    const PlView<double> L(E, 1, cl);
    double *psip_s = (double *)(s_pl + E.o_psip);   // the previous iterate, laid out as v
    double *psi = E.psi, *psip = E.psip;
    // own lines with every row i = 0 .. imax; line 0 with the first CTA
    const int kb = cl.rank == 0 ? 0 : L.k0, own = (L.k1 - kb) * (imax + 1);
    const RowSplit split(imax + 1);
    auto each = [&](auto fn) {
        for (int idx = threadIdx.x; idx < own; idx += PL_THREADS) {
            int t, i;
            split(idx, t, i);
            const int k = kb + t;
            fn(i, k, (k - L.k0 + 1) * L.pitch + i, i + ld * k);
        }
    };
    each([&](int i, int, int s, int c) {
        L.v[s] = 2.0 * psi[c] - psip[c];
        psip_s[s] = psip[c];
        if (i <= L.n1) L.f[s] = E.rhs[c];
    });
    cl.sync();
    int status = GB_MAXSWEEPS, sweeps = 0, nan1 = 0;
    double res1 = 0.0;
    auto relax = [&](int l, bool restricted) {
        pl_sweeps<double>(E, l);
        if (l != 1 && !restricted) return;
        int nan;
        const double m = pl_residual<double>(E, l, &nan);
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
            each([&](int, int, int s, int) {
                const double pf = psip_s[s] + E.sor * (L.v[s] - psip_s[s]);
                L.v[s] = pf;
                psip_s[s] = pf;
            });
            cl.sync();
        }
        if (sweep == 1 || nlev == 1) {
            relax(1, true);
            each([&](int, int, int s, int) { psip_s[s] = L.v[s]; });
        }
        pl_legs<double>(E, relax);
        // The last relax of a sweep is on level 1; its NaN flag decides.
        if (nan1) {
            status = GB_NAN;
            break;
        }
        if (res1 < E.tolcon) {
            status = GB_OK;
            break;
        }
    }
    if (status == GB_OK) {
        // the tank: v on k = 1..np-1, u on k = 1..np, zero side walls
        // (velvor2dhorconvtank.f:1032-1043, :1129-1140)
        const int kend = (E.which == 2) ? np - 1 : np;
        each([&](int i, int k, int s, int c) {
            psip[c] = psi[c];
            psi[c] = i == 0 || i == imax || (E.xwall && (k == 0 || k > kend)) ? 0.0 : L.v[s];
        });
        if (E.xwall && E.which == 3)
            for (int i = cl.tid(); i <= imax; i += cl.nthr()) psi[GIX(i, np + 1, ld)] = 0.0;
    } else {
        each([&](int, int, int s, int c) { psip[c] = psip_s[s]; });
    }
    if (cl.tid() == 0) {
        E.status[0] = status;
        E.status[1] = sweeps;
        *E.resmax = res1;
        if (status == GB_NAN || (status == GB_MAXSWEEPS && E.stop_on_max)) *E.abort = 1;
    }
    cl.sync();   // no CTA leaves while another may still read its shared memory
}

// The mixed solve: k_mg_solve_mixed.
__global__ void __maxnreg__(255) k_pl_solve_mixed(const MgEq *eqs, int first_eq)
{
    __shared__ ClMaxState s_max;
    __shared__ MgEq E;
    const Cluster cl = Cluster::self();
    const MgEq &src = eqs[first_eq + blockIdx.x / cl.size];
    if (*src.abort == GB_RUN_DONE) return;   // a gang member past its last step (the same for every CTA)
    pl_setup<float>(E, src, cl);
    int turn = 0;
    const int ld = E.ld, np = E.np;
    const int imax = (E.which == 2) ? E.nr + 1 : E.nr;
    const PlView<float> L(E, 1, cl);
    const MgLevel &L1 = E.lev[1];
    const int n1 = L.n1, n3 = L.n3, rows = imax + 1, tot = rows * (np + 1);
    const int nrow = (E.which == 2) ? n1 : n1 - 1;
    const double hhri = L1.hhri, hhpi = L1.hhpi, hri = L1.hri;
    double *psif = E.psif, *psi = E.psi, *psip = E.psip;
    const double *rhs = E.rhs, *rvi = L1.rvi, *rvq = L1.rvq;
    const int which = E.which, polar = E.polar;
    const RowSplit split(rows), inner(nrow);
    for (int idx = cl.tid(); idx < tot; idx += cl.nthr()) {
        int k, i;
        split(idx, k, i);
        const int c = i + ld * k;
        psif[c] = 2.0 * psi[c] - psip[c];
    }
    cl.sync();
    auto relax = [&](int l, bool restricted) {
        pl_sweeps<float>(E, l);
        if (!restricted) return;
        int nan;
        pl_residual<float>(E, l, &nan);
        cl.sync();
    };
    int status = GB_MAXSWEEPS, cycles = 0;
    double res = 0.0;
    for (int it = 0;; ++it) {
        // FP64 residual of the iterate on the CTA's own lines; its FP32 copy is the cycle's right-hand side
        double m = 0.0;
        int nan = 0;
        for (int idx = threadIdx.x; idx < (L.k1 - L.k0) * nrow; idx += PL_THREADS) {
            int t, i;
            inner(idx, t, i);
            ++i;
            const int k = L.k0 + t;
            const double *row = psif + (size_t)ld * k;
            const double a = mg_apply_op<double>([&](int q) { return row[q]; }, psif[i + (size_t)ld * (k == n3 ? 1 : k + 1)],
                                                 psif[i + (size_t)ld * (k - 1)], i, which, polar, n1, hhri, hhpi, hri, rvi, rvq);
            const double r = rhs[i + (size_t)ld * k] - a;
            L.own(L.f, k)[L.col(i)] = (float)r;
            const double ar = fabs(r);
            if (ar != ar) nan = 1;
            if (ar > m) m = ar;
        }
        res = cl_max(cl, s_max, turn, m, nan);
        if (nan) { status = GB_NAN; break; }
        if (res < E.tolcon) { status = GB_OK; break; }
        if (it == E.maxsweeps) break;
        relax(1, E.nlev > 1);
        pl_legs<float>(E, relax);
        // psi += w e, and e = 0 for the next cycle
        const double w = (it == 0) ? 1.0 : E.sor;
        const int kb = cl.rank == 0 ? 0 : L.k0;
        for (int idx = threadIdx.x; idx < (L.k1 - kb) * nrow; idx += PL_THREADS) {
            int t, i;
            inner(idx, t, i);
            ++i;
            const int k = kb + t;
            float *e = L.own(L.v, k) + L.col(i);
            psif[i + (size_t)ld * k] += w * (double)*e;
            *e = 0.f;
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

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
void prb_resident_plan(MgEq &E, int mixed, int ctas)
{
    const size_t word = mixed ? 4 : 8;
    size_t at = 0;
    auto take = [&](size_t bytes) {
        const size_t o = at;
        at += (bytes + 15) & ~(size_t)15;
        return (int)o;
    };
    E.smem = 0;
    for (int l = 1; l <= E.nlev; ++l) {
        MgLevel &L = E.lev[l];
        const int n = E.which == 2 ? L.n1 : L.n1 - 1;
        // one segment of a warp in FP32; FP64 lines only have to fit
        if (n < 1 || (mixed && n > 32 * WL_MAXM) || n > 2048) return;
        L.rp = (L.n3 + ctas - 1) / ctas;
        L.pitch = mixed ? std::max(1 + wl_pitch(n), pl_col<float>(wl_log2m(n), L.n1 + 1) + 1) : (L.n1 + 2) | 1;
        const size_t lines = word * (size_t)(L.rp + 1) * L.pitch;
        if (lines > PL_SMEM_MAX) return;
        L.o_v = take(lines);
        L.o_f = take(lines);
        L.o_fac = take(word * (mixed ? (E.which == 2 ? pdma32_len(n) : tdma32_len(n)) : (E.which == 2 ? pdma_fac_len(n) : tdma_fac_len(n))));
        L.o_rv = take(word * 2 * (size_t)(L.n1 + 2));
        L.o_rows = take(4 * (size_t)(L.n3 + 1));
    }
    const size_t lines1 = word * (size_t)(E.lev[1].rp + 1) * E.lev[1].pitch;
    E.o_rc = take(lines1);
    E.o_psip = mixed ? 0 : take(lines1);
    if (at <= PL_SMEM_MAX) E.smem = (int)at;
}

cudaError_t prb_resident_prepare()
{
    cudaError_t e = cl_prepare(k_pl_solve, PL_SMEM_MAX);
    return e == cudaSuccess ? cl_prepare(k_pl_solve_mixed, PL_SMEM_MAX) : e;
}

int prb_resident_fit(int mixed, int ctas, int smem)
{
    return cl_fit(mixed ? k_pl_solve_mixed : k_pl_solve, ctas, PL_THREADS, smem);
}

cudaError_t prb_resident_launch(const MgEq *d_eqs, int first, int neq, int mixed, int ctas, int smem, cudaStream_t s)
{
    return cl_launch(mixed ? k_pl_solve_mixed : k_pl_solve, neq, ctas, PL_THREADS, (size_t)smem, s, d_eqs, first);
}
