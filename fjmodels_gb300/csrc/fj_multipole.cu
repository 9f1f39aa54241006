// fj_multipole.cu -- the multipole side of one iteration: Legendre
// projection of the moment grids, the radial Poisson integrals, the sum of
// component potentials and the tensor-virial sums.  All FP64; each is small
// next to the phase-space kernel.
#include <cooperative_groups.h>

#include "fj_group_qags.cuh"
#include "fj_internal.h"

namespace cg = cooperative_groups;

namespace fj {

// get_Ylm, 6 fields (include/UtilsLeg.h:200-253), with computeRhl's rho[0][0]
// extrapolation (pot/potLeg.cpp:68).  One thread per output coefficient.
__global__ void k_project(int nr, int ngauss, int npoly, const double *ar, const double *poly,
                          const double *grids6, double *coef6)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int ncoef = nr * npoly, npts = nr * ngauss;
    if (t >= 6 * ncoef) return;
    const int q = t / ncoef, n = (t % ncoef) / npoly, l = t % npoly;
    const double *Q = grids6 + (size_t)q * npts;
    double v;
    if (n == 0) {
        if (l != 0) v = 0;
        else if (q == 0)
            v = 2 * ((Q[2 * ngauss] - Q[ngauss]) / (ar[2] - ar[1]) * (ar[0] - ar[1]) + Q[ngauss]);
        else v = 2 * Q[0];
    } else {
        double s = 0;
        for (int g = 0; g < ngauss; g++) s += poly[l * ngauss + g] * Q[n * ngauss + g];
        v = s;
    }
    coef6[t] = v;
}

cudaError_t launch_project(int nr, int ngauss, int npoly, const double *ar, const double *poly,
                           const double *grids6, double *coef6, cudaStream_t s)
{
    const int n = 6 * nr * npoly;
    k_project<<<(n + 127) / 128, 128, 0, s>>>(nr, ngauss, npoly, ar, poly, grids6, coef6);
    return cudaGetLastError();
}

// ------------------------------------------------------------------ Poisson
// linear interpolation of one multipole column (include/Utils.h:122-128): rec[n] =
// 1 / (ar[n+1] - ar[n]), or null to divide; the bracket by the radii's logarithms
// (lg: log2 of the first and the intervals per unit) and a search from there
// (bracket_near), the interval that topbottom's bisection finds (the upper one on a
// node).  A linear grid of 600 radii, l <= 6:
// 1.65 ms, 3.0 with neighbour tests one by one, 2.5 by bisection with a warp per pair.
struct RadialTab {
    const double *ar, *rhl, *rec;
    int npoly, col, nr;
    float2 lg;
    __device__ __forceinline__ double linterp(double x) const
    {
        if (x <= ar[0]) return rhl[col];
        if (x >= ar[nr - 1]) return rhl[(nr - 1) * npoly + col];
        const long long xb = __double_as_longlong(x);
        const int hi = (int)(xb >> 32);
        const float m = __int_as_float(0x3f800000 | ((hi & 0xfffff) << 3) | (int)(((unsigned)xb) >> 29));
        int b = (int)(((float)((hi >> 20) - 1023) + __log2f(m) - lg.x) * lg.y);
        b = b < 0 ? 0 : (b > nr - 2 ? nr - 2 : b);
        b = bracket_near([this](int i) { return ar[i]; }, nr, x, b);
        const double ab = ar[b], yb = rhl[b * npoly + col], yt = rhl[(b + 1) * npoly + col];
        const double f = rec ? div_by(x - ab, ar[b + 1] - ab, rec[b]) : (x - ab) / (ar[b + 1] - ab);
        return yb + f * (yt - yb);
    }
};

struct IInternal {  // I_internal (pot/Potential.cpp:83-89); multipole column col, degree l = 2*col
    RadialTab T; int l;
    __device__ double operator()(double x) const { return pow(x, l + 2) * T.linterp(x); }
};
struct IExternalT {  // I_external (pot/Potential.cpp:90-101) on x = a + (1-t)/t, divided by t^2
    RadialTab T; int l; double a;
    __device__ double operator()(double t) const
    {
        const double x = a + (1 - t) / t;
        double rhol;
        if (x > T.ar[T.nr - 1]) rhol = dmax(0., T.rhl[(T.nr - 1) * T.npoly + T.col] * pow(T.ar[T.nr - 1] / x, 4));
        else rhol = T.linterp(x);
        const double y = rhol / pow(x, l - 1);
        return (y / t) / t;
    }
};

// A warp per integral (2 nr npoly of them: internal, then external).  The function
// values of each Gauss-Kronrod panel (21 or 15, 42 or 30 per bisection) are spread
// over the lanes and summed in the order of one thread running the same QAGS: the
// same function values enter the same sums.  The bookkeeping (fj_group_qags.cuh) is
// over an interval list in shared memory: no device workspace.
// The solve lasts as long as its longest integrals, which are FP64 latency: up to
// 213 bisections on 80 x 7, an external integral tried again with doubled
// tolerances up to four times.  A new try bisects the same intervals until its
// tolerance tells, so the panels of the last try's bisections are kept (kPoissonLog
// of them) and only new intervals are evaluated.  80 x 7: 2.7-2.9 ms; 3.6 ms without
// that, half a warp per integral and bracket searches by bisection; 3.9-4.4 ms with a
// warp per (n, l) pair taking its two integrals one after the other and the panel
// sums on every lane; 33 ms with one thread per pair.
constexpr int kPoissonLanes = 32;
constexpr int kPoissonBlock = 64;
constexpr int kPoissonGroups = kPoissonBlock / kPoissonLanes;
constexpr int kPoissonLog = 64;
constexpr int kPoissonTabled = 2048;  // radii whose reciprocals fit shared memory beside the lists
using PoissonQags = GroupQags<double, kPoissonCap, false, true>;
struct PoissonPanels { double a, b, res, err, rc, res2, err2, rc2; };  // one bisection's two panels

// QAGS of f on [a, b] by the group's lanes (every lane of the warp calls it; `on`
// per group); retry: with doubled tolerances until it succeeds (computeInts,
// pot/Potential.cpp:146-150).  The result is valid on the group's first lane.
template <int RULE, class F>
__device__ double poisson_integral(const F &f, bool on, double a, double b, bool retry, PoissonQags::List &L,
                                   PoissonPanels *log, double *vals, bool &full)
{
    constexpr int N = GKRule<RULE>::npts, G = kPoissonLanes;
    const int lane = threadIdx.x & 31, gi = lane % G, lead = lane - gi;
    double epsabs = 1e-4, epsrel = 1e-3, result = 0, res0 = 0, err0 = 0, ra0 = 0, rc0 = 0, a1 = 0, b2 = 0;
    int tries = 0, step = 0, logged = 0;  // the bisection of this try; bisections logged
    bool run = false;
    PoissonQags st;
    if (on) {
        for (int e = gi; e < N; e += G) vals[e] = f(gk_abscissa<RULE>(a, b, e));
    }
    __syncwarp();
    // the next call: finished by its first panel, or the bisections begin
    auto start = [&]() {
        for (;;) {
            double r, ae;
            const int h = qags_head(res0, err0, ra0, rc0, epsabs, epsrel, 1000, r, ae);
            if (h < 0) {
                st.begin(L, a, b, res0, err0, ra0);
                a1 = a; b2 = b;
                step = 0;
                run = true;
                return;
            }
            result = r;
            run = false;
            if (!retry || h == 0 || ++tries >= 60) return;
            epsabs *= 2; epsrel *= 2;
        }
    };
    if (on && gi == 0) {
        gk_sum<RULE>(a, b, vals, res0, err0, ra0, rc0);
        start();
    }
    for (;;) {
        // 0: finished, 1: evaluate, 2: logged
        const bool known = gi == 0 && run && step < logged && log[step].a == a1 && log[step].b == b2;
        const int go = __shfl_sync(0xffffffffu, run ? (known ? 2 : 1) : 0, lead);
        if (!__any_sync(0xffffffffu, go)) return result;
        a1 = __shfl_sync(0xffffffffu, a1, lead);
        b2 = __shfl_sync(0xffffffffu, b2, lead);
        const double b1 = 0.5 * (a1 + b2);
        double res = 0, err = 0, ra, rc = 0;
        if (go == 1) {
            for (int e = gi; e < 2 * N; e += G) {
                const bool second = e >= N;
                vals[e] = f(gk_abscissa<RULE>(second ? b1 : a1, second ? b2 : b1, second ? e - N : e));
            }
        }
        __syncwarp();
        if (go == 1 && gi % (G / 2) == 0)
            gk_sum<RULE>(gi ? b1 : a1, gi ? b2 : b1, vals + (gi ? N : 0), res, err, ra, rc);
        double res2 = __shfl_sync(0xffffffffu, res, lead + G / 2), err2 = __shfl_sync(0xffffffffu, err, lead + G / 2),
               rc2 = __shfl_sync(0xffffffffu, rc, lead + G / 2);
        if (go && gi == 0) {
            if (go == 2) {
                const PoissonPanels &p = log[step];
                res = p.res; err = p.err; rc = p.rc; res2 = p.res2; err2 = p.err2; rc2 = p.rc2;
            } else if (retry && step < kPoissonLog) {
                log[step] = PoissonPanels{a1, b2, res, err, rc, res2, err2, rc2};
                if (logged == step) logged = step + 1;
            }
            step++;
        }
        if (go && gi == 0) {
            double r = 0;
            if (st.update(L, res, err, rc, res2, err2, rc2, epsabs, epsrel, r, full)) {
                result = r;
                run = false;
                if (retry && st.ier_class != 0 && ++tries < 60) {
                    epsabs *= 2; epsrel *= 2;
                    start();
                }
            } else {
                a1 = L.iv[st.maxerr].a;
                b2 = L.iv[st.maxerr].b;
            }
        }
        __syncwarp();
    }
}

// computeInts (pot/Potential.cpp:110-155): the internal integrals into phil, the
// external ones into Pr, for k_poisson_tables
__global__ void __launch_bounds__(kPoissonBlock) k_poisson(int nr, int npoly, const double *ar, const double *rhl,
                                                           double *phil, double *Pr, unsigned long long *counters)
{
    __shared__ PoissonQags::List s_list[kPoissonGroups];
    __shared__ PoissonPanels s_log[kPoissonGroups][kPoissonLog];
    __shared__ double s_vals[kPoissonGroups][43];
    extern __shared__ double s_rec[];  // of grids that fit: 1 / (ar[n+1] - ar[n])
    const bool tabled = nr <= kPoissonTabled;
    for (int i = threadIdx.x; tabled && i < nr - 1; i += kPoissonBlock) s_rec[i] = recip(ar[i + 1] - ar[i]);
    __syncthreads();
    const int g = threadIdx.x / kPoissonLanes, nt = nr * npoly;
    const int i = blockIdx.x * kPoissonGroups + g;  // [0, nt): external (the longer ones), then internal
    const bool ext = i < nt;
    const int t = ext ? i : i - nt;
    const bool on = t < nt;
    const int n = on ? t / npoly : 0, np = on ? t % npoly : 0, l = 2 * np;
    bool full = false;
    double v;
    const float l0 = log2f((float)ar[0]);
    const RadialTab T{ar, rhl, tabled ? s_rec : nullptr, npoly, np, nr, make_float2(l0, (nr - 1) / (log2f((float)ar[nr - 1]) - l0))};
    if (!ext) v = poisson_integral<21>(IInternal{T, l}, on, 0., ar[n], false, s_list[g], s_log[g], s_vals[g], full);
    else v = poisson_integral<15>(IExternalT{T, l, ar[n]}, on, 0., 1., true, s_list[g], s_log[g], s_vals[g], full);
    if (!on || threadIdx.x % kPoissonLanes) return;
    if (full && counters) atomicAdd(&counters[kCntPoisson], 1ull);
    (ext ? Pr : phil)[t] = v;
}

// computePhil (pot/Potential.cpp:157-200) from the integrals, in place
__global__ void k_poisson_tables(int nr, int npoly, const double *ar, const double *rhl, double *phil, double *Pr,
                                 double *Pr2)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nr * npoly) return;
    const int n = t / npoly, l = 2 * (t % npoly);
    const double r = ar[n], Iint = phil[t], Iext = Pr[t];
    const double G = 1;
    phil[t] = -kTPI * G * (Iint / pow(r, l + 1) + Iext * pow(r, l));
    Pr[t] = -kTPI * G * (-(l + 1) * Iint / pow(r, l + 2) + l * Iext * pow(r, l - 1));
    Pr2[t] = -kTPI * G * ((l + 2) * (l + 1) * Iint / pow(r, l + 3) + (l - 1) * l * Iext * pow(r, l - 2) -
                          (2 * l + 1) * rhl[t]);
}

cudaError_t launch_poisson(int nr, int npoly, const double *ar, const double *rhl, double *phil,
                           double *Pr, double *Pr2, unsigned long long *counters, cudaStream_t s)
{
    const int nt = nr * npoly;
    const size_t smem = nr <= kPoissonTabled ? (nr - 1) * sizeof(double) : 0;
    k_poisson<<<(2 * nt + kPoissonGroups - 1) / kPoissonGroups, kPoissonBlock, smem, s>>>(nr, npoly, ar, rhl, phil, Pr,
                                                                                         counters);
    k_poisson_tables<<<(nt + 63) / 64, 64, 0, s>>>(nr, npoly, ar, rhl, phil, Pr, Pr2);
    return cudaGetLastError();
}

// ------------------------------------------- exact cumulative Poisson solve
// The integrals of computeInts (pot/Potential.cpp:82-155) taken exactly: the
// integrands are x^(l+2) rho_l(x) and rho_l(x) x^(1-l) with rho_l the linear
// interpolation of the density multipoles (linterp, include/Utils.h:122-128:
// constant below ar[0]) and rho_l(x) = max(0, rho_l[nr-1] (ar[nr-1]/x)^4)
// beyond the grid (Potential.cpp:90-99), so each grid interval contributes a
// closed form and the integrals are prefix sums over the intervals, added in
// a fixed order.  No adaptive decisions: the potential is a smooth function of
// the density, where the reference's QAGS (epsabs 1e-4, epsrel 1e-3) moves it
// by up to ~1e-3 when a small change of the density flips a subdivision.
// One cluster of kCumCluster blocks per multipole l.  The powers of the radii are
// most of the work (nine per radius, ~190 FP64 instructions each): the cluster's
// blocks, on SMs of their own, share them, a thread per power, into the first
// block's shared memory; that block goes on with a thread per interval, the two
// prefix sums on a thread each, and a thread per radius.  40 radii, l <= 8: 16.9 us;
// 22.4 us with one block taking all powers, ~58 us with a thread per interval taking
// its own eight and a thread per radius seven.

// int_a^b x^m (c0 + c1 x) dx from a^(m+1), b^(m+1) (p0) and a^(m+2), b^(m+2) (p1)
__device__ __forceinline__ double seg_power_integral(double a, double b, int m, double c0, double c1, double p0a,
                                                     double p0b, double p1a, double p1b)
{
    const double t0 = m == -1 ? log(b / a) : (p0b - p0a) / (m + 1);
    const double t1 = m == -2 ? log(b / a) : (p1b - p1a) / (m + 2);
    return c0 * t0 + c1 * t1;
}

constexpr int kCumPowers = 9, kCumBlock = 128, kCumCluster = 8;

__global__ void __launch_bounds__(kCumBlock) __cluster_dims__(kCumCluster, 1, 1)
    k_poisson_cumulative(int nr, int npoly, const double *ar,
                                                                  const double *rhl, double *phil, double *Pr,
                                                                  double *Pr2, bool tabled)
{
    extern __shared__ double sh[];
    double *s_in = sh, *s_ex = sh + nr;  // interval i = [ar[i], ar[i+1]] (s_in[nr-1]: [0, ar[0]]; s_ex[nr-1]: tail)
    const int np = blockIdx.x / kCumCluster, l = 2 * np;
    cg::cluster_group cluster = cg::this_cluster();
    // pw[j][n] = ar[n]^(l - 2 + j), j < 7; pw[7][n] = ar[n]^(2 - l), pw[8][n] = ar[n]^(3 - l); of grids too large
    // for shared memory where they are used
    double *pw = sh + 2 * nr;
    auto power = [&](int j, int n) { return pow(ar[n], j < 7 ? l - 2 + j : j == 7 ? 2 - l : 3 - l); };
    const int rank = (int)cluster.block_rank();
    if (tabled) {
        // The first block's shared memory may be written only once that block runs: every block
        // arrives at the cluster's barrier as it starts and waits there with its first power at hand.
        cluster.barrier_arrive();
        double *first = cluster.map_shared_rank(pw, 0);
        int i = rank * kCumBlock + threadIdx.x;
        const double p0 = i < kCumPowers * nr ? power(i / nr, i % nr) : 0.;
        cluster.barrier_wait();
        if (i < kCumPowers * nr) first[i] = p0;
        for (i += kCumCluster * kCumBlock; i < kCumPowers * nr; i += kCumCluster * kCumBlock)
            first[i] = power(i / nr, i % nr);
        cluster.sync();  // the powers are in the first block's shared memory
    }
    if (rank != 0) return;
    auto q = [&](int j, int n) { return tabled ? pw[j * nr + n] : power(j, n); };
    for (int t = threadIdx.x; t < 2 * nr; t += blockDim.x) {
        const int i = t % nr;
        const bool ex = t >= nr;
        if (i < nr - 1) {
            const double a = ar[i], b = ar[i + 1], ya = rhl[i * npoly + np], yb = rhl[(i + 1) * npoly + np];
            const double s = (yb - ya) / (b - a), c0 = ya - s * a;
            if (!ex) s_in[i] = seg_power_integral(a, b, l + 2, c0, s, q(5, i), q(5, i + 1), q(6, i), q(6, i + 1));
            else s_ex[i] = seg_power_integral(a, b, 1 - l, c0, s, q(7, i), q(7, i + 1), q(8, i), q(8, i + 1));
        } else if (!ex) {
            s_in[i] = rhl[np] * q(5, 0) / (l + 3);
        } else {
            const double yN = rhl[(nr - 1) * npoly + np];
            s_ex[i] = (yN > 0 ? yN : 0.) * q(7, nr - 1) / (l + 2);
        }
    }
    __syncthreads();
    // prefix sums in place: s_in[n] = I_int(ar[n]), s_ex[n] = I_ext(ar[n])
    if (threadIdx.x == 0) {
        double acc = s_in[nr - 1], seg = s_in[0];
        s_in[0] = acc;
        for (int n = 1; n < nr; n++) {
            acc += seg;
            seg = s_in[n];
            s_in[n] = acc;
        }
    } else if (threadIdx.x == 32) {
        double acc = s_ex[nr - 1];
        for (int n = nr - 1; n >= 0; n--) {
            const double cur = n < nr - 1 ? s_ex[n] : 0.;
            if (n < nr - 1) acc += cur;
            s_ex[n] = acc;
        }
    }
    __syncthreads();
    for (int n = threadIdx.x; n < nr; n += blockDim.x) {  // computePhil (Potential.cpp:163-200)
        const double Ii = s_in[n], Ie = s_ex[n], G = 1;
        const int t = n * npoly + np;
        phil[t] = -kTPI * G * (Ii / q(3, n) + Ie * q(2, n));
        Pr[t] = -kTPI * G * (-(l + 1) * Ii / q(4, n) + l * Ie * q(1, n));
        Pr2[t] = -kTPI * G * ((l + 2) * (l + 1) * Ii / q(5, n) + (l - 1) * l * Ie * q(0, n) - (2 * l + 1) * rhl[t]);
    }
}

cudaError_t launch_poisson_cumulative(int nr, int npoly, const double *ar, const double *rhl, double *phil,
                                      double *Pr, double *Pr2, cudaStream_t s)
{
    if (nr < 2 || nr > kPoissonCumulativeMaxNr) return cudaErrorInvalidValue;
    const bool tabled = (2 + kCumPowers) * nr * sizeof(double) <= 48 * 1024;
    k_poisson_cumulative<<<npoly * kCumCluster, kCumBlock, (tabled ? 2 + kCumPowers : 2) * nr * sizeof(double), s>>>(
        nr, npoly, ar, rhl, phil, Pr, Pr2, tabled);
    return cudaGetLastError();
}

// ------------------------------------------------------------ updatePhil
__global__ void k_sum3(int n, const double *a0, const double *a1, const double *a2, const double *b0,
                       const double *b1, const double *b2, double *o0, double *o1, double *o2)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    o0[t] = a0[t] + b0[t];
    o1[t] = a1[t] + b1[t];
    o2[t] = a2[t] + b2[t];
}

cudaError_t launch_sum3(int n, const double *a0, const double *a1, const double *a2, const double *b0,
                        const double *b1, const double *b2, double *o0, double *o1, double *o2, cudaStream_t s)
{
    k_sum3<<<(n + 255) / 256, 256, 0, s>>>(n, a0, a1, a2, b0, b1, b2, o0, o1, o2);
    return cudaGetLastError();
}

__global__ void k_add(int n, const double *a, const double *b, double *o)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) o[i] = a[i] + b[i];
}

cudaError_t launch_add(int n, const double *a, const double *b, double *o, cudaStream_t s)
{
    k_add<<<(n + 255) / 256, 256, 0, s>>>(n, a, b, o);
    return cudaGetLastError();
}

// ------------------------------------------------------------------ vir2
constexpr int kVirBlock = 256;

// vir2 (libs/Stats.cpp:12-41) with the 5-field ev_dens / int_dens of
// include/UtilsLeg.h:300-354, whose interpolation weight is a float (:312).
__global__ void __launch_bounds__(kVirBlock) k_vir2(PotView P, int ngauss, const double *ci, const double *wi,
                                                   const double *coef6, double *out7)
{
    const int nr = P.nr, npoly = P.npoly, nc = nr * npoly;
    const double *ar = P.ar, *rhl = coef6, *sigRl = coef6 + 2 * nc, *sigpl = coef6 + 3 * nc, *sigzl = coef6 + 4 * nc;
    double acc[5] = {0, 0, 0, 0, 0};  // pot, KRR, Kzz, WRR, Wzz
    const int ncell = (nr - 1) * ngauss;
    for (int cell = threadIdx.x; cell < ncell; cell += kVirBlock) {
        const int i = 1 + cell / ngauss, j = cell % ngauss;
        const double r = .5 * (ar[i - 1] + ar[i]), dr = ar[i] - ar[i - 1];
        const double sij = sqrt(1 - ci[j] * ci[j]);
        const double z = r * ci[j], R = r * sij;
        const double rr = sqrt(R * R + z * z), c = z / rr;
        double dens = 0, Su = 0, Sp = 0, Sv = 0;
        if (!(rr > ar[nr - 1])) {
            int top = 0, bot = 0;
            topbottom(ar, nr, rr, bot, top);
            const float f = (float)((rr - ar[bot]) / (ar[top] - ar[bot]));
            const float omf = 1 - f;
            const double c2 = c * c;
            double pm2 = 1, pm1 = 0;
            for (int np = 0; np < npoly; np++) {
                const double dp = f * rhl[top * npoly + np] + omf * rhl[bot * npoly + np];
                const double up = f * sigRl[top * npoly + np] + omf * sigRl[bot * npoly + np];
                const double pp = f * sigpl[top * npoly + np] + omf * sigpl[bot * npoly + np];
                const double vp = f * sigzl[top * npoly + np] + omf * sigzl[bot * npoly + np];
                if (np == 0) { dens = .5 * dp; Su = .5 * up; Sp = .5 * pp; Sv = .5 * vp; continue; }
                double pol;
                if (np == 1) { pol = 1.5 * c2 - .5; pm1 = pol; }
                else { pol = evenleg_next(np, c2, pm2, pm1); pm2 = pm1; pm1 = pol; }
                const double fac = .5 * (4 * np + 1);
                dens += fac * dp * pol;
                Su += fac * up * pol;
                Sp += fac * pp * pol;
                Sv += fac * vp * pol;
            }
        }
        double phi, dR, dz;
        pot_grad(P, R, z, phi, dR, dz);
        acc[0] += .5 * wi[j] * dens * phi * r * r * dr;
        acc[1] += .5 * wi[j] * dens * ((r * Su) * (r * Su) + (r * Sp) * (r * Sp)) * dr;
        acc[2] += .5 * wi[j] * dens * ((r * Sv) * (r * Sv)) * dr;
        acc[3] -= wi[j] * dens * R * dR * r * r * dr;
        acc[4] -= wi[j] * dens * z * dz * r * r * dr;
    }
    __shared__ double red[kVirBlock / 32][5];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < 5; q++) {
        double v = acc[q];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) red[warp][q] = v;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double s[5] = {0, 0, 0, 0, 0};
        for (int w = 0; w < kVirBlock / 32; w++)
            for (int q = 0; q < 5; q++) s[q] += red[w][q];
        const double fpi = 4 * kPI;
        out7[0] = s[1] * fpi;  // KRR
        out7[1] = s[2] * fpi;  // Kzz
        out7[2] = s[3] * fpi;  // WRR
        out7[3] = s[4] * fpi;  // Wzz
        out7[4] = s[0] * fpi;  // PE
        out7[5] = ar[nr - 1] * ar[nr - 1] * P.Pr[(nr - 1) * npoly];
        // mass check (Stats.cpp:35-37)
        double sum = 0.;
        for (int i = 0; i < nr; i++) {
            int top = 0, bot = 0;
            topbottom(ar, nr, ar[i], bot, top);
            const double f = (ar[i] - ar[bot]) / (ar[top] - ar[bot]);
            double dens = .5 * (f * rhl[top * npoly] + (1 - f) * rhl[bot * npoly]);
            double pm2 = 1, pm1 = 0;
            for (int np = 1; np < npoly; np++) {
                double pol;
                if (np == 1) { pol = -.5; pm1 = pol; }
                else { pol = evenleg_next(np, 0.0, pm2, pm1); pm2 = pm1; pm1 = pol; }
                dens += .5 * (4 * np + 1) * (f * rhl[top * npoly + np] + (1 - f) * rhl[bot * npoly + np]) * pol;
            }
            sum += 2 * kTPI * ar[i] * ar[i] * dens;
        }
        out7[6] = sum;
    }
}

cudaError_t launch_vir2(PotView P, int ngauss, const double *ci, const double *wi, const double *coef6,
                        double *out7, cudaStream_t s)
{
    k_vir2<<<1, kVirBlock, 0, s>>>(P, ngauss, ci, wi, coef6, out7);
    return cudaGetLastError();
}

size_t poisson_local_bytes()
{
    cudaFuncAttributes at;
    return cudaFuncGetAttributes(&at, k_poisson) == cudaSuccess ? at.localSizeBytes : 0;
}

size_t multipole_local_bytes()
{
    size_t m = 0;
    cudaFuncAttributes at;
    if (cudaFuncGetAttributes(&at, k_poisson) == cudaSuccess && at.localSizeBytes > m) m = at.localSizeBytes;
    if (cudaFuncGetAttributes(&at, k_vir2) == cudaSuccess && at.localSizeBytes > m) m = at.localSizeBytes;
    return m;
}

}  // namespace fj
