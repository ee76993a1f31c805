// Mixed-precision streamfunction solve of the axisymmetric annulus on its
// uniform and its stretched grid: FP64 defect correction around FP32 V-cycles
// of line relaxation (the schedule of rotann2.f:598-666 and rcsc.f:1118-1195)
// that never leave the shared memory of one thread-block cluster.
//
// A cycle is about 90 relaxation half-sweeps of a few hundred lines each, and
// every one of them must finish before the next begins, so its cost is
// latency: with the levels in HBM/L2 a half-sweep paid two or three dependent
// L2 round trips, the eliminations' serial chains and a release of its global
// stores, 8.6 k cycles on average at 257 x 257 whatever the level.  Here
// every level's correction and right-hand side is spread over the cluster's
// CTAs by rows j (contiguous blocks, so that a coarse row lives where its
// fine rows do), a line is the registers of up to 32 lanes (warpline.cuh), and CTAs meet
// at the hardware cluster barrier with distributed shared memory between
// them.  r-lines are local to a CTA except for the rows at its block's edges;
// a z-line crosses all CTAs, so each CTA forms its rows' right-hand sides and
// stores them into the line's owner, which eliminates and stores the solution
// back: one value per unknown each way.
//
// The FP64 residual is the one part bound by arithmetic (the FP64 pipe issues
// two lanes a cycle and SM): its divisions are products with stored reciprocals
// and a correction, the conversions and the norm go to the integer pipe.
//
// Measured (GB300, mixed solve, a step's whole time): 257 x 257 stretched, five
// cycles, 22.3 ms on one SM and global memory, 2.6 ms resident on a cluster of 16.
#include "meridian.cuh"

#include <algorithm>

#include "cluster.cuh"
#include "convert.cuh"
#include "warpline.cuh"

#define MER_THREADS 256
#define MER_SMEM_MAX (220 * 1024)
// Floats of a warp's staging buffer for one neighbour row of each of its lines.
#define MER_STAGE(n) ((32 >> wl_log2w(n)) * (wl_pitch(n) + 2))
// The thread that starts the table copies: the last warp has lines only when
// every other has.
#define MER_FETCHER (MER_THREADS - 32)
// Polls of a table copy's barrier before a solve gives up (about a second), and
// before it ends without a copy that is still on its way.
#ifndef MER_POLLS
#define MER_POLLS (1 << 22)
#endif
#define MER_DRAIN_POLLS (1 << 22)

// Column i of a row: two leading pads (the far point of i = 1 is never read
// with a nonzero weight, but is read), then a lane's rows padded to an odd
// stride as the line eliminations want them.
__host__ __device__ __forceinline__ int mer_col(int lg, int i) { return i < 1 ? i + 1 : 1 + i + ((i - 1) >> lg); }

// Shared-memory addresses that may be another CTA's (the row and line address
// tables hold these, resolved once per solve: an owner's index is an integer
// division and its window a mapa, 300 cycles a row when formed on the way).
__device__ __forceinline__ float cld(unsigned addr)
{
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ void cst(unsigned addr, float v) { asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory"); }
__device__ __forceinline__ unsigned cta_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned peer_addr(const void *p, int rank)
{
    unsigned a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(cta_addr(p)), "r"(rank));
    return a;
}

// x / h for h > 0 from ih, the rounded 1 / h: a product and two corrections.  The
// first leaves a faithful quotient, the second the correctly rounded one (the
// remainder is exact then; Markstein, IBM J. Res. Dev. 34(1), 1990).  Divided by
// itself, a lane's rows go one after the other through the division's branch, 290
// cycles each (16 x 16, an r half-sweep: 4.0 k cycles, 2.1 k this way).  Both corrections
// need x away from the ends of the exponent's range, MerLevel::quick the same of
// the divisors; else `bad` is set and the caller divides.
__device__ __forceinline__ float mer_quot(float x, float h, float ih, bool &bad)
{
    const unsigned e = (__float_as_uint(x) >> 23) & 0xffu;
    if (e - (127u - 95u) > 2u * 95u && x != 0.f) bad = true;
    float q = x * ih;
    q = __fmaf_rn(__fmaf_rn(-h, q, x), ih, q);
    q = __fmaf_rn(__fmaf_rn(-h, q, x), ih, q);
    return x == 0.f ? x : q;
}

// Own rows of a level: j0 .. j1 - 1 at local indices 1, 2, ...
struct MerOwn {
    int j0, j1;
    int lo, hi;   // the rows this CTA holds, a boundary row included
    __device__ __forceinline__ MerOwn(const MerLevel &L, const Cluster &cl)
    {
        j0 = cl.rank * L.rp + 1;
        j1 = min(j0 + L.rp, L.n2);
        lo = cl.rank == 0 ? 0 : j0;
        hi = cl.rank == cl.size - 1 ? L.n2 : min(j0 + L.rp - 1, L.n2);
    }
    // the first line of colour c
    template <int NC> __device__ __forceinline__ int first(int c) const { return j0 + ((c - j0) % NC + NC) % NC; }
};

// z-lines of a colour per CTA, from the largest colour's: the l-th line of
// every colour then has the same owner and place.
template <int NC> __device__ __forceinline__ int mer_share(int ni, int ctas) { return ((ni - 1) / NC + ctas) / ctas; }

// The line tables of the next half-sweep are copied into shared memory by
// bulk copies while this one runs (a fetch into registers between the halves
// of a barrier made the barrier wait for L2, 1.4 k cycles).  `k` counts
// half-sweeps: stage k & 1 holds the tables of half-sweep k.
struct MerPipe {
    unsigned long long bar[2];
    int timeout;   // 0, or 1 + the half-sweep whose wait gave up: no copy is started any more
};

// One thread of the CTA: starts the copy of the CTA's tables of colour c of
// direction dir into stage k & 1 (consumed last in half-sweep k - 2, which a
// cluster barrier has ended).
template <bool PENTA> __device__ __forceinline__ void mer_fetch(const MerLevel &L, MerPipe &pipe, int tab, int tab_floats, int dir, int c, int k)
{
    extern __shared__ __align__(16) float s_mer[];
    const int timeout = *(volatile int *)&pipe.timeout;   // on its way while the rest is formed
    const Cluster cl = Cluster::self();
    constexpr int NC = PENTA ? 4 : 2;
    const int n = dir == 0 ? L.n1 - 1 : L.n2 - 1;
    const int len = (int)(PENTA ? pdma32_len(n) : tdma32_len(n));
    int line, count, step;
    const float *src;
    if (dir == 0) {
        const MerOwn own(L, cl);
        line = own.template first<NC>(c);
        count = line < own.j1 ? (own.j1 - 1 - line) / NC + 1 : 0;
        step = L.fac_r_step;
        src = L.fac_r;
        if (step == 0) count = min(count, 1);   // one table for all lines
    } else {
        const int ni = L.n1 - 1, nl = c <= ni ? (ni - c) / NC + 1 : 0;
        const int share = mer_share<NC>(ni, cl.size), l0 = cl.rank * share;
        count = max(0, min(nl - l0, share));
        line = c + NC * l0;
        step = L.fac_z_step;
        src = L.fac_z;
    }
    if (timeout) return;   // the stage may still be waiting for the copy before
    const unsigned bar = cta_addr(&pipe.bar[k & 1]);
    const unsigned dst = cta_addr(s_mer + tab + (k & 1) * tab_floats);
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(count * len * 4) : "memory");
    for (int t = 0; t < count; ++t)
        asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst + 4u * t * len),
                     "l"(src + (size_t)(line - 1 + NC * t) * step), "r"(len * 4), "r"(bar)
                     : "memory");
}
// Whether half-sweep k's tables have landed.
__device__ __forceinline__ bool mer_landed(MerPipe &pipe, int k)
{
    unsigned ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok)
                 : "r"(cta_addr(&pipe.bar[k & 1])), "r"((k >> 1) & 1)
                 : "memory");
    return ok;
}
// Waits for them; gives up after MER_POLLS polls, once.
__device__ __forceinline__ void mer_tables(MerPipe &pipe, int k)
{
    bool ok = false;
    for (int q = 0; !ok && q < MER_POLLS; ++q) {
        if ((q & 1023) == 1023 && *(volatile int *)&pipe.timeout) return;
        ok = mer_landed(pipe, k);
    }
    if (!ok && !*(volatile int *)&pipe.timeout) pipe.timeout = k + 1;
}
// The end of a solve: the copies still on their way (the one prepared for a cycle
// that is not run, k's, or the one that a wait gave up on and the one after it)
// land before the block leaves.
__device__ __forceinline__ void mer_drain(MerPipe &pipe, int k)
{
    const int timeout = *(volatile int *)&pipe.timeout;
    for (int c = timeout ? timeout - 1 : k; c <= (timeout ? timeout : k); ++c)
        for (int q = 0; !mer_landed(pipe, c) && q < MER_DRAIN_POLLS; ++q) {
        }
}

// The r-lines of one sweep, colour by colour: the CTA's lines of the colour go
// round its warps, 32 / W at a time.  Returns the next half-sweep's number.
//
// A lane's rows lie M + 1 words from the next lane's, so a neighbour row read
// that way from another CTA would cost eight requests to each 128 bytes of it;
// such a row is first copied, contiguously, into the line's staging buffer.
template <int M, bool PENTA> __device__ __noinline__ int mer_r_sweep(const MerLevel &lev, MerPipe &pipe, int stage, int tab, int tab_floats, int k)
{
    extern __shared__ __align__(16) float s_mer[];
    const MerLevel L = lev;
    const Cluster cl = Cluster::self();
    constexpr int NC = PENTA ? 4 : 2;
    const int n = L.n1 - 1, lw = wl_log2w(n), per = 32 >> lw;
    const int len = L.fac_r_step ? (int)(PENTA ? pdma32_len(n) : tdma32_len(n)) : 0;
    const int sub = (threadIdx.x & 31) >> lw, lane = threadIdx.x & ((1 << lw) - 1);
    const int slot = (threadIdx.x >> 5) * per + sub, nslots = (MER_THREADS / 32) * per;
    const MerOwn own(L, cl);
    const float4 *cj = (const float4 *)(s_mer + L.ocj);
    const unsigned *rows = (const unsigned *)(s_mer + L.rows);
    const int col = 2 + lane * (M + 1);
    for (int c = 1; c <= NC; ++c, ++k) {
        if (threadIdx.x == MER_FETCHER) mer_fetch<PENTA>(L, pipe, tab, tab_floats, c < NC ? 0 : 1, c < NC ? c + 1 : 1, k + 1);
        const int jc = own.template first<NC>(c);
        bool ready = false;
        for (int tb = 0; jc + NC * tb < own.j1; tb += nslots) {
            if (jc + NC * (tb + slot - sub) >= own.j1) continue;   // no line for this warp
            const bool live = jc + NC * (tb + slot) < own.j1;
            const int t0 = live ? tb + slot : tb + slot - sub, j = jc + NC * t0;   // idle groups repeat a line and store nothing
            const int row = (j - own.j0 + 1) * L.pitch + col;
            // the neighbours in the order their terms are added
            constexpr int NN = PENTA ? 3 : 2;
            int near[NN];
            float weight[NN];
            if constexpr (PENTA) {
                const float4 w = cj[j];
                const bool low = j <= L.n2 / 2;
                near[0] = low ? j - 1 : j - 2;
                near[1] = low ? j + 1 : j - 1;
                near[2] = low ? j + 2 : j + 1;
                weight[0] = w.x;
                weight[1] = low ? w.z : w.y;
                weight[2] = w.w;
            } else {
                near[0] = j + 1;
                near[1] = j - 1;
            }
            float t[M];
#pragma unroll
            for (int u = 0; u < M; ++u) t[u] = s_mer[L.f + row + u];
            const float *src[NN];
#pragma unroll
            for (int q = 0; q < NN; ++q) {
                if (near[q] >= own.lo && near[q] <= own.hi) {
                    src[q] = s_mer + L.v + (near[q] - own.j0 + 1) * L.pitch + col;
                } else {
                    float *buf = s_mer + stage + ((threadIdx.x >> 5) * NN + q) * MER_STAGE(n) + sub * (wl_pitch(n) + 2);
                    const unsigned r = rows[near[q]] + 8;
                    float v[M + 1];   // W lanes' rows and their padding: M + 1 words a lane
#pragma unroll
                    for (int e = 0; e <= M; ++e) v[e] = cld(r + 4 * (lane + (e << lw)));
#pragma unroll
                    for (int e = 0; e <= M; ++e) buf[lane + (e << lw)] = v[e];
                    src[q] = buf + col - 2;
                }
            }
            __syncwarp();
            if constexpr (PENTA) {
#pragma unroll
                for (int u = 0; u < M; ++u) t[u] = -(weight[0] * src[0][u] + weight[1] * src[1][u] + weight[2] * src[2][u]) + t[u];
            } else {
                float s[M], q[M];
                bool bad = !L.quick;
#pragma unroll
                for (int u = 0; u < M; ++u) s[u] = -(src[0][u] + src[1][u]);
#pragma unroll
                for (int u = 0; u < M; ++u) q[u] = mer_quot(s[u], L.hhz, L.ihhz, bad);
                if (bad) {
#pragma unroll
                    for (int u = 0; u < M; ++u) q[u] = s[u] / L.hhz;
                }
#pragma unroll
                for (int u = 0; u < M; ++u) t[u] = q[u] + t[u];
            }
            if (!ready) {
                mer_tables(pipe, k);
                ready = true;
            }
            WlTab<M, PENTA> T;
            T.load(s_mer + tab + (k & 1) * tab_floats + (size_t)t0 * len, lw);
            T.solve(n, t);
            if (live) {
#pragma unroll
                for (int u = 0; u < M; ++u)
                    if (lane * M + u < n) s_mer[L.v + row + u] = t[u];
            }
        }
        cl.sync();
    }
    return k;
}

// The z-lines of one sweep: each warp forms its rows' right-hand sides of the
// colour and stores them into the lines' owners (a row's neighbours in r are
// its own, so this needs no other CTA), a barrier, the owners eliminate and
// store the solutions into the rows' owners, a barrier.  Stores, because a
// load from another CTA costs its requester nine cycles a request (a colour's
// solutions fetched by the rows' owners: 2.4 k cycles, stored by the lines':
// 0.8 k); the line buffer holds [row][line], so that a row's values for one
// owner are contiguous.  `last`: the relaxation's last sweep, whose
// successor's tables the caller fetches.
template <int M, bool PENTA>
__device__ __noinline__ int mer_z_sweep(const MerLevel &lev, MerPipe &pipe, int xoff, int tab, int tab_floats, int lg, bool last, int k)
{
    extern __shared__ __align__(16) float s_mer[];
    const MerLevel L = lev;
    const Cluster cl = Cluster::self();
    constexpr int NC = PENTA ? 4 : 2;
    constexpr int LGM = M == 8 ? 3 : 4;
    const int n = L.n2 - 1, lw = wl_log2w(n), per = 32 >> lw;
    const int len = (int)(PENTA ? pdma32_len(n) : tdma32_len(n));
    const int sub = (threadIdx.x & 31) >> lw, zl = threadIdx.x & ((1 << lw) - 1);
    const int slot = (threadIdx.x >> 5) * per + sub, nslots = (MER_THREADS / 32) * per;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = MER_THREADS / 32;
    const MerOwn own(L, cl);
    const int ni = L.n1 - 1;
    const float4 *ci = (const float4 *)(s_mer + L.oci);
    const unsigned *rows = (const unsigned *)(s_mer + L.rows), *xline = (const unsigned *)(s_mer + L.xline);
    const float *x = s_mer + xoff;
    const int share = mer_share<NC>(ni, cl.size), l0 = cl.rank * share;
    for (int c = 1; c <= NC; ++c, ++k) {
        if (threadIdx.x == MER_FETCHER && (c < NC || !last))
            mer_fetch<PENTA>(L, pipe, tab, tab_floats, c < NC ? 1 : 0, c < NC ? c + 1 : 1, k + 1);
        const int nl = c <= ni ? (ni - c) / NC + 1 : 0;
        for (int j = own.j0 + warp; j < own.j1; j += nw) {
            const float *vr = s_mer + L.v + (j - own.j0 + 1) * L.pitch;
            const float *fr = s_mer + L.f + (j - own.j0 + 1) * L.pitch;
            const int xj = 4 * ((j - 1) * share + ((j - 1) >> LGM));
            for (int l = lane; l < nl; l += 32) {
                const int i = c + NC * l;
                const float f = fr[mer_col(lg, i)];
                float r;
                if constexpr (PENTA) {
                    const float4 a = ci[2 * i], b = ci[2 * i + 1];
                    const bool low = i <= L.n1 / 2;
                    const float p0 = vr[mer_col(lg, low ? i - 1 : i - 2)], p1 = vr[mer_col(lg, low ? i + 1 : i - 1)];
                    const float p2 = vr[mer_col(lg, low ? i + 2 : i + 1)];
                    const float over = (b.x * (low ? p0 : p1) + b.z * (low ? p1 : p2)) * b.w;
                    r = -(a.x * p0 + (low ? a.z : a.y) * p1 + a.w * p2 + over) + f;
                } else {
                    const float vp = vr[mer_col(lg, i + 1)], vm = vr[mer_col(lg, i - 1)];
                    const float4 a = ci[i];
                    const float s = -(vp + vm), e = (vp - vm) * 0.5f;
                    bool bad = !L.quick;
                    r = mer_quot(s, L.hhr, L.ihhr, bad) + f - mer_quot(mer_quot(e, a.x, a.z, bad), L.hr, L.ihr, bad);
                    if (bad) r = s / L.hhr + f - e / a.x / L.hr;
                }
                cst(xline[l] + xj, r);
            }
        }
        cl.sync();
        const int mine = min(nl - l0, share);   // lines l0 .. l0 + mine - 1 of the colour
        bool ready = false;
        for (int tb = 0; tb < mine; tb += nslots) {
            if (tb + slot - sub >= mine) continue;
            const bool live = tb + slot < mine;
            const int t = live ? tb + slot : tb + slot - sub;
            const float *xs = x + zl * (M * share + 1) + t;
            float r[M];
#pragma unroll
            for (int u = 0; u < M; ++u) r[u] = xs[u * share];
            if (!ready) {
                mer_tables(pipe, k);
                ready = true;
            }
            WlTab<M, PENTA> T;
            T.load(s_mer + tab + (k & 1) * tab_floats + (size_t)t * len, lw);
            T.solve(n, r);
            if (live) {
                const unsigned col = 4 * mer_col(lg, c + NC * (l0 + t));
                const int j = zl * M + 1;
#pragma unroll
                for (int u = 0; u < M; ++u)
                    if (j + u < L.n2) cst(rows[j + u] + col, r[u]);
            }
        }
        cl.sync();
    }
    return k;
}

// The correction's residual on a level into rc (own rows).
template <bool PENTA> __device__ __noinline__ void mer_residual(const MerLevel &lev, int rc, int lg)
{
    extern __shared__ __align__(16) float s_mer[];
    const MerLevel L = lev;
    const Cluster cl = Cluster::self();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = MER_THREADS / 32;
    const MerOwn own(L, cl);
    const float4 *ci = (const float4 *)(s_mer + L.oci), *cj = (const float4 *)(s_mer + L.ocj);
    const unsigned *rows = (const unsigned *)(s_mer + L.rows);
    for (int j = own.j0 + warp; j < own.j1; j += nw) {
        const bool lowj = j <= L.n2 / 2;
        const unsigned vm = rows[j - 1], vp = rows[j + 1], vf = PENTA ? rows[lowj ? j + 2 : j - 2] : vm;
        const int row = (j - own.j0 + 1) * L.pitch;
        const float *v = s_mer + L.v + row, *f = s_mer + L.f + row;
        float *out = s_mer + rc + row;
#pragma unroll 2
        for (int i = 1 + lane; i < L.n1; i += 32) {
            const int c = mer_col(lg, i);
            const float d = cld(vm + 4 * c), u = cld(vp + 4 * c), e = PENTA ? cld(vf + 4 * c) : 0.f;
            const float p = v[c], pm = v[mer_col(lg, i - 1)], pp = v[mer_col(lg, i + 1)];
            float t;
            if constexpr (PENTA) {
                const float4 a = ci[2 * i], b = ci[2 * i + 1], w = cj[j];
                const bool low = i <= L.n1 / 2;
                const float far = v[mer_col(lg, low ? i + 2 : i - 2)];
                const float over = (b.x * pm + b.y * p + b.z * pp) * b.w, overq = p * (b.w * b.w);
                t = a.x * (low ? pm : far) + a.y * (low ? p : pm) + a.z * (low ? pp : p) + a.w * (low ? far : pp) + over - overq;
                t = t + w.x * (lowj ? d : e) + w.y * (lowj ? p : d) + w.z * (lowj ? u : p) + w.w * (lowj ? e : u);
            } else {
                const float4 a = ci[i];
                const float s = pp + pm, g = (pp - pm) * 0.5f, y = u + d;
                bool bad = !L.quick;
                t = mer_quot(s, L.hhr, L.ihhr, bad) + mer_quot(mer_quot(g, L.hr, L.ihr, bad), a.x, a.z, bad) - mer_quot(p, a.y, a.w, bad) +
                    mer_quot(y, L.hhz, L.ihhz, bad) - p * L.drdz;
                if (bad) t = s / L.hhr + g / L.hr / a.x - p / a.y + y / L.hhz - p * L.drdz;
            }
            out[c] = f[c] - t;
        }
    }
    cl.sync();
}

// corser (rotann2.f:755-801, rcsc.f:1343-1390): nine-point restriction; the
// row j = n1c that both clear (n1 of the coarse level in both directions) is
// zero, and the coarse correction is cleared.
template <bool PENTA> __device__ __noinline__ void mer_corser(const MerLevel &fine, const MerLevel &coarse, int rc)
{
    extern __shared__ __align__(16) float s_mer[];
    const MerLevel F = fine, L = coarse;
    const Cluster cl = Cluster::self();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = MER_THREADS / 32;
    const MerOwn own(L, cl);
    const int lgf = wl_log2m(F.n1 - 1), lg = wl_log2m(L.n1 - 1);
    const unsigned *rows = (const unsigned *)(s_mer + F.rows);
    const int to_rc = 4 * (rc - F.v);   // rc's rows lie as v's do
    for (int j = own.j0 + warp; j < own.j1; j += nw) {
        const unsigned q0 = rows[2 * j] + to_rc, qm = rows[2 * j - 1] + to_rc, qp = rows[2 * j + 1] + to_rc;
        const int row = (j - own.j0 + 1) * L.pitch;
        for (int i = 1 + lane; i < L.n1; i += 32) {
            const int a = 4 * mer_col(lgf, 2 * i - 1), b = 4 * mer_col(lgf, 2 * i), c = 4 * mer_col(lgf, 2 * i + 1);
            const float o0 = cld(q0 + b), e = cld(q0 + c), w = cld(q0 + a), n = cld(qp + b), s = cld(qm + b);
            const float ne = cld(qp + c), sw = cld(qm + a), se = cld(qm + c), nw_ = cld(qp + a);
            float t;
            if (PENTA) {   // the sums as each of the two references orders them
                t = o0 * 2.f + e + w;
                t = t + n + s;
                t = t * 2.f + ne + sw;
                t = (t + se + nw_) * 0.0625f;
            } else {
                t = 0.25f * o0 + 0.125f * (e + w + n + s) + 0.0625f * (ne + sw + se + nw_);
            }
            const int o = row + mer_col(lg, i);
            s_mer[L.f + o] = j == L.n1 ? 0.f : t;
            s_mer[L.v + o] = 0.f;
        }
    }
    cl.sync();
}

// finer (rotann2.f:803-854, rcsc.f:1392-1444): bilinear prolongation added.
__device__ __noinline__ void mer_finer(const MerLevel &coarse, const MerLevel &fine)
{
    extern __shared__ __align__(16) float s_mer[];
    const MerLevel C = coarse, L = fine;
    const Cluster cl = Cluster::self();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = MER_THREADS / 32;
    const MerOwn own(L, cl);
    const int lgc = wl_log2m(C.n1 - 1), lg = wl_log2m(L.n1 - 1);
    const unsigned *rows = (const unsigned *)(s_mer + C.rows);
    for (int j = own.j0 + warp; j < own.j1; j += nw) {
        const unsigned q0 = rows[j >> 1], q1 = rows[(j + 1) >> 1];
        float *v = s_mer + L.v + (j - own.j0 + 1) * L.pitch;
#pragma unroll 2
        for (int i = 1 + lane; i < L.n1; i += 32) {
            const int a = 4 * mer_col(lgc, i >> 1), b = 4 * mer_col(lgc, (i + 1) >> 1);
            const float u = cld(q0 + a) + cld(q1 + b);   // one point twice, two, or two of four
            v[mer_col(lg, i)] += i & j & 1 ? (u + cld(q1 + a) + cld(q0 + b)) * 0.25f : u * 0.5f;
        }
    }
    cl.sync();
}

// relax on level l; half-sweep k's tables are on their way.
template <bool PENTA> __device__ __forceinline__ int mer_relax(const MerDev &d, MerPipe &pipe, int l, bool restricted, int k)
{
    const MerLevel &L = d.lev[l];
    const int lgr = wl_log2m(L.n1 - 1), lgz = wl_log2m(L.n2 - 1);
    for (int irel = 0; irel < d.nrel; ++irel) {
        const bool last = irel == d.nrel - 1;
        if (lgr == 3) k = mer_r_sweep<8, PENTA>(L, pipe, d.stage, d.tab, d.tab_floats, k);
        else k = mer_r_sweep<16, PENTA>(L, pipe, d.stage, d.tab, d.tab_floats, k);
        if (lgz == 3) k = mer_z_sweep<8, PENTA>(L, pipe, d.x, d.tab, d.tab_floats, lgr, last, k);
        else k = mer_z_sweep<16, PENTA>(L, pipe, d.x, d.tab, d.tab_floats, lgr, last, k);
    }
    if (restricted) mer_residual<PENTA>(L, d.rc, lgr);
    return k;
}

// x / h: the IEEE quotient up to the sign of a zero (divrn.cuh).
__device__ __forceinline__ double mer_over(double x, double h, double ih)
{
    const double q = __dmul_rn(x, ih);
    return __fma_rn(__fma_rn(-h, q, x), ih, q);
}

// FP64 residual of the iterate over this CTA's rows: its FP32 rounding is the
// cycle's right-hand side.  Returns the largest magnitude's bit pattern (NaNs
// excluded; the order of non-negative doubles is the order of their bits).
// The terms stand in the reference's order: with the weights of a row combined
// (9 operations instead of 32) the last bits of a small residual, and with them
// the whole correction, round differently: 3e-9 of the streamfunction.
template <bool PENTA> __device__ __noinline__ double mer_residual64(const MerDev &d, int *nan_out)
{
    extern __shared__ __align__(16) float s_mer[];
    const Cluster cl = Cluster::self();
    const MerLevel L = d.lev[1];
    const double *dv = d.v, *drhs = d.rhs;
    const MerRow *di = d.d_i;
    const MerCol *dj = d.d_j;
    const MerOver hr = d.hr, hhr = d.hhr, hhz = d.hhz;
    const double drdz = d.drdz;
    const int ld = L.n1 + 1, ni = L.n1 - 1, lg = wl_log2m(ni);
    const MerOwn own(L, cl);
    const int j0 = own.j0, j1 = own.j1;
    const RowSplit split(ni);
    unsigned long long m = 0;
    int nan = 0;
    for (int idx = threadIdx.x; idx < (j1 - j0) * ni; idx += MER_THREADS) {
        int jj, i;
        split(idx, jj, i);
        ++i;
        const int j = j0 + jj;
        const double *v = dv + (size_t)j * ld + i;
        const MerRow &a = di[i];
        const double p = v[0], pm = v[-1], pp = v[1], pd = v[-ld], pu = v[ld];
        double t;
        if constexpr (PENTA) {
            const MerCol &w = dj[j];
            const bool low = i <= L.n1 / 2, lowj = j <= L.n2 / 2;
            const double far = v[low ? 2 : -2], farj = v[lowj ? 2 * ld : -2 * ld];
            t = a.crr[0] * (low ? pm : far) + a.crr[1] * (low ? p : pm) + a.crr[2] * (low ? pp : p) + a.crr[3] * (low ? far : pp) +
                mer_over(a.cr[0] * pm + a.cr[1] * p + a.cr[2] * pp, a.r, a.ir) - mer_over(p, a.rr, a.irr);
            t = t + w.czz[0] * (lowj ? pd : farj) + w.czz[1] * (lowj ? p : pd) + w.czz[2] * (lowj ? pu : p) + w.czz[3] * (lowj ? farj : pu);
        } else {
            t = mer_over(pp + pm, hhr.h, hhr.ih) + mer_over(mer_over((pp - pm) * 0.5, hr.h, hr.ih), a.r, a.ir) - mer_over(p, a.rr, a.irr) +
                mer_over(pu + pd, hhz.h, hhz.ih) - p * drdz;
        }
        const double r = drhs[(size_t)j * ld + i] - t;
        const unsigned long long bits = (unsigned long long)__double_as_longlong(r) & 0x7fffffffffffffffull;
        if (bits > 0x7ff0000000000000ull) nan = 1;
        else if (bits > m) m = bits;
        s_mer[L.f + (1 + jj) * L.pitch + mer_col(lg, i)] = d2f_rn(r);
    }
    *nan_out = nan;
    return __longlong_as_double((long long)m);
}

// The functions above take copies of the level descriptors they use: behind a
// reference, every field would be fetched again after each barrier (which
// invalidates L1), 600 cycles from L2.  The descriptor itself is kept in
// shared memory for the same reason.
template <bool PENTA> __device__ __forceinline__ void mer_solve_body(const MerDev &desc)
{
    extern __shared__ __align__(16) float s_mer[];
    __shared__ ClMaxState s_max;
    __shared__ MerDev d;
    __shared__ __align__(8) MerPipe pipe;
    constexpr int NC = PENTA ? 4 : 2;
    const Cluster cl = Cluster::self();
    if (desc.abort && *desc.abort) return;   // the same for every CTA: nothing sets it while the solve runs
    for (int q = threadIdx.x; q < (int)(sizeof(MerDev) / 4); q += MER_THREADS) ((unsigned *)&d)[q] = ((const unsigned *)&desc)[q];
    __syncthreads();
    int turn = 0;
    const int nlev = d.nlev;
    const MerLevel L = d.lev[1];
    const int ld = L.n1 + 1, tp = ld * (L.n2 + 1), lg = wl_log2m(L.n1 - 1);
    for (int q = threadIdx.x; q < d.smem_floats; q += MER_THREADS) s_mer[q] = 0.f;
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the zeros of the table stages, before the first copy
    __syncthreads();
    if (threadIdx.x == 0) {
        pipe.timeout = 0;
        for (int q = 0; q < 2; ++q)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(cta_addr(&pipe.bar[q])) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int l = 1; l <= nlev; ++l) {
        const MerLevel &K = d.lev[l];
        for (int i = threadIdx.x; i < (PENTA ? 2 : 1) * (K.n1 + 1); i += MER_THREADS) ((float4 *)(s_mer + K.oci))[i] = K.ci[i];
        for (int j = threadIdx.x; j <= K.n2; j += MER_THREADS) {
            if (PENTA) ((float4 *)(s_mer + K.ocj))[j] = K.cj[j];
            const int o = min((max(j, 1) - 1) / K.rp, cl.size - 1);
            const float *p = s_mer + K.v + (j - o * K.rp) * K.pitch;
            ((unsigned *)(s_mer + K.rows))[j] = o == cl.rank ? cta_addr(p) : peer_addr(p, o);
        }
        const int nl = (K.n1 - 2) / NC + 1, share = mer_share<NC>(K.n1 - 1, cl.size);
        for (int q = threadIdx.x; q < nl; q += MER_THREADS) {
            const int o = q / share;
            const float *p = s_mer + d.x + (q - o * share);
            ((unsigned *)(s_mer + K.xline))[q] = o == cl.rank ? cta_addr(p) : peer_addr(p, o);
        }
    }
    for (int idx = cl.tid(); idx < tp; idx += cl.nthr()) d.v[idx] = d.psi[idx];
    cl.sync();
    const MerOwn own(L, cl);
    const int j0 = own.j0, j1 = own.j1;
    const RowSplit split(L.n1 - 1);
    int status = GB_MAXSWEEPS, cycles = 0, k = 0;
    // starts the copy of the tables that half-sweep k needs
    auto fetch = [&](int l) {
        if (threadIdx.x == MER_FETCHER) mer_fetch<PENTA>(d.lev[l], pipe, d.tab, d.tab_floats, 0, 1, k);
    };
    for (int it = 0;; ++it) {
        fetch(1);
        int flags;
        const double m = mer_residual64<PENTA>(d, &flags);
        if (*(volatile int *)&pipe.timeout) flags |= 2;
        const double res = cl_max(cl, s_max, turn, m, flags);
        if (flags & 2) { status = GB_TIMEOUT; break; }
        if (flags) { status = GB_NAN; break; }
        if (res < d.tolcon) { status = GB_OK; break; }
        if (it == d.maxcycles) break;
        k = mer_relax<PENTA>(d, pipe, 1, nlev > 1, k);
        for (int l = 1; l < nlev; ++l) {
            fetch(l + 1);
            mer_corser<PENTA>(d.lev[l], d.lev[l + 1], d.rc);
            k = mer_relax<PENTA>(d, pipe, l + 1, l + 1 < nlev, k);
        }
        for (int l = nlev; l >= 2; --l) {
            fetch(l - 1);
            mer_finer(d.lev[l], d.lev[l - 1]);
            k = mer_relax<PENTA>(d, pipe, l - 1, false, k);
        }
        // psi += e, and e = 0 for the next cycle
        for (int idx = threadIdx.x; idx < (j1 - j0) * split.n; idx += MER_THREADS) {
            int jj, i;
            split(idx, jj, i);
            ++i;
            float *e = s_mer + L.v + (1 + jj) * L.pitch + mer_col(lg, i);
            d.v[(size_t)(j0 + jj) * ld + i] += f2d(*e);
            *e = 0.f;
        }
        cl.sync();
        cycles = it + 1;
    }
    if (status == GB_OK)
        for (int idx = cl.tid(); idx < tp; idx += cl.nthr()) d.psi[idx] = d.v[idx];
    if (cl.tid() == 0) {
        d.status[0] = status;
        d.status[1] = cycles;
        if ((status == GB_NAN || status == GB_TIMEOUT) && d.abort) *d.abort = 1;
    }
    mer_drain(pipe, k);
    cl.sync();   // no CTA leaves while another may still read its shared memory
}

template <bool PENTA> __global__ void __maxnreg__(255) k_mer_solve(const __grid_constant__ MerDev d) { mer_solve_body<PENTA>(d); }
template <bool PENTA> __global__ void __maxnreg__(255) k_mer_many(const MerDev *devs)
{
    const MerDev &d = devs[blockIdx.x / cooperative_groups::this_cluster().num_blocks()];
    mer_solve_body<PENTA>(d);
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
bool mer_plan(MerDev &d, int ctas)
{
    int at = 0;
    auto take = [&](int floats) {
        const int o = at;
        at += (floats + 3) & ~3;
        return o;
    };
    int xneed = 0, tneed = 0, sneed = 0;
    const int nc = d.penta ? 4 : 2;
    for (int l = 1; l <= d.nlev; ++l) {
        MerLevel &L = d.lev[l];
        if (L.n1 - 1 > 32 * WL_MAXM || L.n2 - 1 > 32 * WL_MAXM || L.n1 < 2 || L.n2 < 2) return false;
        const int lg = wl_log2m(L.n1 - 1);
        L.rp = (L.n2 - 1 + ctas - 1) / ctas;
        // all rows of all W lanes are read: a row of the array holds them, two pads before and one after
        L.pitch = std::max(2 + wl_pitch(L.n1 - 1), mer_col(lg, L.n1 + 1) + 1);
        L.v = take((L.rp + 2) * L.pitch);
        L.f = take((L.rp + 2) * L.pitch);
        L.oci = take((d.penta ? 8 : 4) * (L.n1 + 1));
        L.ocj = take(d.penta ? 4 * (L.n2 + 1) : 0);
        const int lines = (L.n1 - 2) / nc + 1, share = (lines + ctas - 1) / ctas;
        L.rows = take(L.n2 + 1);
        L.xline = take(lines);
        xneed = std::max(xneed, share * wl_rows(L.n2 - 1) + (wl_rows(L.n2 - 1) >> wl_log2m(L.n2 - 1)));
        sneed = std::max(sneed, (MER_THREADS / 32) * (d.penta ? 3 : 2) * MER_STAGE(L.n1 - 1));
        auto len = [&](int n) { return (int)(d.penta ? pdma32_len(n) : tdma32_len(n)); };
        const int rl = L.fac_r_step ? std::min((L.rp - 1) / nc + 1, L.rp) : 1;
        tneed = std::max(tneed, std::max(rl * len(L.n1 - 1), share * len(L.n2 - 1)));
    }
    d.rc = take((d.lev[1].rp + 2) * d.lev[1].pitch);
    d.x = take(xneed);
    d.stage = take(sneed);
    d.tab_floats = (tneed + 3) & ~3;
    d.tab = take(2 * d.tab_floats);
    d.smem_floats = at;
    return (size_t)at * sizeof(float) <= MER_SMEM_MAX;
}

size_t mer_weight_bytes(const MerDev &d)
{
    size_t b = sizeof(MerRow) * (size_t)(d.lev[1].n1 + 1) + sizeof(MerCol) * (size_t)(d.lev[1].n2 + 1);
    for (int l = 1; l <= d.nlev; ++l) b += sizeof(float4) * (size_t)(2 * (d.lev[l].n1 + 1) + d.lev[l].n2 + 1);
    return b;
}

void mer_weight_layout(MerDev &d, void *mem)
{
    MerRow *r = (MerRow *)mem;
    d.d_i = r; r += d.lev[1].n1 + 1;
    MerCol *c = (MerCol *)r;
    d.d_j = c; c += d.lev[1].n2 + 1;
    float4 *q = (float4 *)c;
    for (int l = 1; l <= d.nlev; ++l) {
        d.lev[l].ci = q; q += 2 * (d.lev[l].n1 + 1);
        d.lev[l].cj = q; q += d.lev[l].n2 + 1;
    }
}

int mer_fit(MerDev &d, int want)
{
    cudaError_t e = d.penta ? cl_prepare(k_mer_solve<true>, MER_SMEM_MAX) : cl_prepare(k_mer_solve<false>, MER_SMEM_MAX);
    if (e == cudaSuccess) e = d.penta ? cl_prepare(k_mer_many<true>, MER_SMEM_MAX) : cl_prepare(k_mer_many<false>, MER_SMEM_MAX);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    for (int c = want; c >= 1; c >>= 1) {
        if (!mer_plan(d, c)) return 0;   // fewer CTAs need more memory each
        const size_t smem = sizeof(float) * (size_t)d.smem_floats;
        const int got = d.penta ? cl_fit(k_mer_solve<true>, c, MER_THREADS, smem) : cl_fit(k_mer_solve<false>, c, MER_THREADS, smem);
        if (got == c) return c;
    }
    return 0;
}

int mer_alone(MerDev &d, int most)
{
    if (cl_small_grid(d.lev[1].n1, d.lev[1].n2) && mer_plan(d, 1)) return 1;
    mer_plan(d, most);
    return most;
}

int mer_plan_many(MerDev *d, int n, int want, int most, size_t *smem, char *fits)
{
    for (int c = want;; c <<= 1) {
        bool all = true;
        *smem = 0;
        for (int q = 0; q < n; ++q) {
            fits[q] = mer_plan(d[q], c);
            all = all && fits[q];
            if (fits[q]) *smem = std::max(*smem, sizeof(float) * (size_t)d[q].smem_floats);
        }
        if (all || 2 * c > most) return c;
    }
}

cudaError_t mer_launch(const MerDev &d, int ctas, cudaStream_t s)
{
    const size_t smem = sizeof(float) * (size_t)d.smem_floats;
    if (d.penta) return cl_launch(k_mer_solve<true>, 1, ctas, MER_THREADS, smem, s, d);
    return cl_launch(k_mer_solve<false>, 1, ctas, MER_THREADS, smem, s, d);
}

cudaError_t mer_launch_many(const MerDev *d_devs, int n, int penta, int ctas, size_t smem, cudaStream_t s)
{
    if (penta) return cl_launch(k_mer_many<true>, n, ctas, MER_THREADS, smem, s, d_devs);
    return cl_launch(k_mer_many<false>, n, ctas, MER_THREADS, smem, s, d_devs);
}
