// fj_solve64.cuh -- the plain FP64 action solves of a list of phase points by
// one block: the steps of the turning points phase by phase, a point per lane,
// the momentum integrals by groups of lanes (fj_group_qags.cuh).
//
// The GB300's FP64 pipe takes a warp instruction every ~18 cycles per SM
// whether one lane is active or 32 (measured: 103 per SM and microsecond with 1
// to 32 active lanes, and already with one block of 4 warps), so the time of
// these solves is the number of FP64 warp instructions.  Hence
//  - all 32 lanes evaluate an integrand at every step of the quadrature: first
//    every integral's first panel, then the bisections of those that go on, each
//    group of kSolveLanes lanes on its own integral;
//  - the sines and cosines of the quadrature angles come from a table over the
//    bisection tree (its panels are the same for every orbit), the divisions of
//    the potential by grid constants from reciprocals (PotView::itab), and what
//    an orbit's equations repeat is computed once (Fudge::prepare).
// The turning points are those of a point on one thread bit for bit (up to div_by's
// rounding), the integrals to rounding (PotFast).
// Measured (GB300), one thread per orbit with in-place divisions before, this
// after: one iteration of a 16x6 model with 22^3 nodes 556 -> 160 ms, moments at
// 6 points 95-111 -> 12.2 ms, 40 line-profile values 171 -> 39.8 ms, 20 001 actions
// 33.4 -> 6.0 ms (10.2 before its items were cut to whole rounds).  Of these steps, the integrals by groups, the table and the
// reciprocals gave 581 -> 230 ms on the first, the turning points phase by phase
// 230 -> 216 ms, the integrands' own potential and exponential 216 -> 160 ms.
#pragma once

#include "fj_group_qags.cuh"

namespace fj {

constexpr int kSolveBlock = 128;                        // threads of a solving block
constexpr int kSolveLanes = 4;                          // lanes per momentum integral (2: large launches 3-9 % faster, 6 points 20 % slower)
constexpr int kSolveGroups = kSolveBlock / kSolveLanes;  // integrals in flight
constexpr int kTrigPanels = 1024;                       // bisection tree down to 1/512 of the range

// One point's solve: its constants, the brackets of its roots (u0; inner and
// outer u; v), its actions
struct OrbitRec {
    Fudge o;
    double pu2, pv2, w;       // squared momenta; pi/2 - vturn
    double lo[4], hi[4];
    double fju, fjv, Jr, Jz;  // factors of the integrals; results
    unsigned todo;            // kOrbit*
    unsigned rootfail[3];     // the roots of inner u, outer u, v
    int more[2], full[2];     // Ju, Jv: goes on after its first panel; its list was full
    __device__ unsigned status() const { return o.fail | rootfail[0] | rootfail[1] | rootfail[2] | (full[0] | full[1] ? kFailQuad : 0u); }
};
// steps left: bound at all; roots of u (Ju to integrate later) and v to refine
enum : unsigned { kOrbitJu = 1u, kOrbitJv = 2u, kOrbitBound = 4u, kOrbitRootU = 8u, kOrbitRootV = 16u };

using OrbitQags = GroupQags<double, kQagsCap, true>;

// A block's scratch in device memory
struct SolveScratch {
    OrbitRec *rec;                          // [chunk]
    double2 *head;                          // [2 chunk]: first panels of the integrals that go on (result, error)
    OrbitQags::List *lists;      // [kSolveGroups]
};
FJ_HD size_t solve_scratch_bytes(int chunk)
{
    return chunk * (sizeof(OrbitRec) + 2 * sizeof(double2)) + kSolveGroups * sizeof(OrbitQags::List);
}
FJ_HD SolveScratch solve_scratch(char *base, int chunk)
{
    SolveScratch s;
    s.lists = (OrbitQags::List *)base;
    s.head = (double2 *)(s.lists + kSolveGroups);
    s.rec = (OrbitRec *)(s.head + 2 * chunk);
    return s;
}

// A block's shared memory of the solver
struct SolveShared {
    double vals[kSolveGroups][43];  // panel values (43: the groups' columns start in different banks)
    int next[7], nmore;             // list positions of the phases; whether any integral goes on
};

// The potential as the integrands evaluate it: besides PotView's tables the
// differences d[n][k] = phil[n+1][k] - phil[n][k], and the quadratic correction's
// e = phil[thr][k] - phil[n][k] - f3 d per interval and side (below, above).  The
// roots need the reference's operations one by one (a sign test or the |f| < 5e-4
// shortcut decides with the last bit); an integrand only enters sums, so here the
// same interpolation and recurrences are written with FMAs and folded constants: 5
// FP64 instructions per multipole instead of 14, and sinh and cosh from one
// exponential.  Measured against 113-bit values (4000 orbits of an 80-radius, l <=
// 12 potential, focal distances 1e-3 to 1, errors relative to the orbit's
// integrand): Ju median 1.2e-15, rms 3.6e-14 (the plain form 1.35e-15, 4.1e-14), Jv
// 8.4e-16, 4.7e-13 (9.6e-16, 4.6e-13: the one figure of the four that is not smaller,
// by 2 %, one orbit's cancellation).  One iteration of the 16x6 model 216 -> 160
// ms, 40 line-profile values 65 -> 39.8 ms.
struct PotFast {
    int nr, npoly;
    const double *ar, *phil, *d, *e, *itab;  // d null: no such tables, evaluate with PotView
};
FJ_HD int fast_table_size(int nr, int npoly) { return nr * npoly + 2 * kQuadTab * npoly; }
__device__ __forceinline__ PotFast fast_tables(const PotView &P, double *tab)  // threads of a block; P's tables complete
{
    const int nr = P.nr, np_ = P.npoly, nt = nr * np_;
    double *d = tab, *e = tab + nt;
    for (int i = threadIdx.x; i < nt; i += blockDim.x) d[i] = i < nt - np_ ? P.phil[i + np_] - P.phil[i] : 0.;
    for (int i = threadIdx.x; i < 2 * kQuadTab * np_; i += blockDim.x) {
        const int n = i / (2 * np_), up = (i / np_) & 1, k = i % np_, thr = up ? n + 2 : n - 1;
        double v = 0;
        if (thr >= 0 && thr < nr && n + 1 < nr) {
            const double f3 = P.itab[1 + nr + 3 * (2 * n + up) + 2], vb = P.phil[n * np_ + k];
            v = P.phil[thr * np_ + k] - vb - f3 * (P.phil[(n + 1) * np_ + k] - vb);
        }
        e[i] = v;
    }
    return PotFast{nr, np_, P.ar, P.phil, d, e, P.itab};
}

// P_2k = pm1 (C c2 - CB) - CA pm2 (evenleg_next with its constants multiplied out)
struct LegFold { double C, CB, CA; };
struct LegFoldTable { LegFold c[kMaxPoly]; };
constexpr LegFoldTable make_leg_fold()
{
    LegFoldTable t{};
    for (int np = 2; np < kMaxPoly; np++) {
        const int l = 2 * (np - 1), l2 = 2 * l;
        const double C = (l2 + 1) * (l2 + 3) / (double)((l + 1) * (l + 2));
        t.c[np].C = C;
        t.c[np].CB = C * ((l2 * l + l2 - 1) / (double)((l2 - 1) * (l2 + 3)));
        t.c[np].CA = C * (l * (l - 1) / (double)((l2 + 1) * (l2 - 1)));
    }
    return t;
}
static __constant__ LegFoldTable kLegFold_d = make_leg_fold();

__device__ __forceinline__ double pot_fast(const PotFast &F, double R, double z)
{
    const double *ar = F.ar;
    const int nr = F.nr, np_ = F.npoly;
    const double r2 = fma(R, R, z * z), y = rsqrt(r2), r0 = r2 * y, r = fma(0.5 * y, fma(-r0, r0, r2), r0);
    const double c = z * y, c2 = c * c;
    double pm2 = 1.0, pm1 = fma(1.5, c2, -.5);
    const long long rb = __double_as_longlong(r);
    if (rb >= __double_as_longlong(ar[nr - 1])) {  // beyond the grid (or not a number)
        const double x = ar[nr - 1] * y, x2 = x * x;
        const double *T = F.phil + (nr - 1) * np_;
        double xp = x, phi = T[0] * x;
        for (int k = 1; k < np_; k++) {
            xp *= x2;
            double p = pm1;
            if (k > 1) {
                const LegFold &L = kLegFold_d.c[k];
                p = fma(-L.CA, pm2, pm1 * fma(L.C, c2, -L.CB));
                pm2 = pm1; pm1 = p;
            }
            phi = fma(T[k] * xp, p, phi);
        }
        return phi;
    }
    const double *tab = F.itab;
    const float2 g = *(const float2 *)tab;
    const bool inside = rb < __double_as_longlong(ar[0]);
    const double re = inside ? ar[0] : r;
    const long long reb = inside ? __double_as_longlong(ar[0]) : rb;
    const int hi = (int)(reb >> 32);  // interval guess and neighbour tests as interp_setup
    const float m = __int_as_float(0x3f800000 | ((hi & 0xfffff) << 3) | (int)(((unsigned)reb) >> 29));
    int b = (int)(((float)((hi >> 20) - 1023) + __log2f(m) - g.x) * g.y);
    b = b < 0 ? 0 : (b > nr - 2 ? nr - 2 : b);
    while (b > 0 && reb < __double_as_longlong(ar[b])) --b;
    while (b < nr - 2 && reb > __double_as_longlong(ar[b + 1])) ++b;
    const double db = re - ar[b], f1 = db * tab[1 + b];
    const double *T = F.phil + b * np_, *D = F.d + b * np_;
    if (b < kQuadTab) {
        const bool up = !(f1 < 0.5 && b > 0);
        const int side = 2 * b + (up ? 1 : 0);
        const double f2 = (re - ar[b + 1]) * db * tab[1 + nr + 3 * side + 1];
        const double *e = F.e + side * np_;
        double phi = fma(f2, e[0], fma(f1, D[0], T[0]));
        for (int k = 1; k < np_; k++) {
            double p = pm1;
            if (k > 1) {
                const LegFold &L = kLegFold_d.c[k];
                p = fma(-L.CA, pm2, pm1 * fma(L.C, c2, -L.CB));
                pm2 = pm1; pm1 = p;
            }
            phi = fma(fma(f2, e[k], fma(f1, D[k], T[k])), p, phi);
        }
        return phi;
    }
    double phi = fma(f1, D[0], T[0]);
    if (np_ > 1) phi = fma(fma(f1, D[1], T[1]), pm1, phi);
    for (int k = 2; k < np_; k++) {
        const LegFold &L = kLegFold_d.c[k];
        const double p = fma(-L.CA, pm2, pm1 * fma(L.C, c2, -L.CB));
        phi = fma(fma(f1, D[k], T[k]), p, phi);
        pm2 = pm1; pm1 = p;
    }
    return phi;
}

// sinh and cosh of u: from one exponential where they do not cancel, else their
// power series (|u| <= 3/4: the next terms are below 1e-18 of the sums)
__device__ __forceinline__ void sinh_cosh(double u, double &s, double &c)
{
    const double au = fabs(u);
    if (au > 0.75 && au < 700.) {
        const double e = exp(au), g = 0.5 * recip(e);
        s = copysign(fma(0.5, e, -g), u);
        c = fma(0.5, e, g);
    } else if (au <= 0.75) {
        const double w = u * u;
        double a = 1. / 355687428096000., b = 1. / 20922789888000.;  // 17!, 16!
        a = fma(a, w, 1. / 1307674368000.); b = fma(b, w, 1. / 87178291200.);
        a = fma(a, w, 1. / 6227020800.);    b = fma(b, w, 1. / 479001600.);
        a = fma(a, w, 1. / 39916800.);      b = fma(b, w, 1. / 3628800.);
        a = fma(a, w, 1. / 362880.);        b = fma(b, w, 1. / 40320.);
        a = fma(a, w, 1. / 5040.);          b = fma(b, w, 1. / 720.);
        a = fma(a, w, 1. / 120.);           b = fma(b, w, 1. / 24.);
        a = fma(a, w, 1. / 6.);             b = fma(b, w, .5);
        s = fma(a * w, u, u);
        c = fma(b, w, 1.);
    } else {
        s = sinh(u);
        c = cosh(u);
    }
}

__device__ __forceinline__ double orbit_integrand(const PotView &P, const PotFast &F, const OrbitRec &r, bool kv,
                                                  double sn, double cs)
{
    const Fudge &c = r.o;
    double R, z, s2;
    if (!kv) {  // uvOrb.cpp:226-239
        double shu, chu;
        sinh_cosh(fma(-c.Deltau, cs, c.ubar), shu, chu);
        s2 = shu * shu;
        R = c.Delta * shu * c.sinv;
        z = c.Delta * chu * c.cosv;
    } else {  // uvOrb.cpp:247-257
        double s, k;
        sincos(fma(-r.w, cs, kPIH), &s, &k);
        s2 = s * s;
        R = c.Dshu * s;
        z = c.Dchu * k;
    }
    const double phi = F.d ? pot_fast(F, R, z) : pot_phi(P, R, z);
    double f;
    if (!kv) {
        const double dUv = fma(s2 + c.sv2, phi, -c.B0);
        f = fma(-c.LzD2, recip(s2) - c.ish1, fma(c.E, s2 - c.sh1sq, c.Erch) - dUv);
    } else {
        const double dV = fma(-(c.shu2 + s2), phi, c.C0);
        f = fma(c.E, s2, c.Iv) + dV - c.hL / (c.DD * s2);
    }
    return sqrt(dmax(0., f)) * sn;
}

// sine and cosine of abscissa e of panel `heap` ([a, b]) of the Ju or Jv tree
__device__ __forceinline__ void panel_sincos(const double2 *trig, bool kv, unsigned heap, double a, double b, int e,
                                             double &sn, double &cs)
{
    if (heap - 1u < (unsigned)(kTrigPanels - 1)) {
        const double2 t = trig[((kv ? kTrigPanels : 0) + heap) * 21 + e];
        sn = t.x; cs = t.y;
    } else {
        sincos(gk_abscissa<21>(a, b, e), &sn, &cs);
    }
}

// A phase of the turning-point solves: every lane works on an item of its own and
// takes the next one when it finishes, and all lanes of a warp come together at
// each step's function value.  (A thread that ran its point through all phases by
// itself met the other lanes in other phases and at other steps: 44 % of the lanes
// active in a quarter of the solver's time.)
// begin(item) returns false where there is nothing to do; step() evaluates and
// advances the current item, returning true when it is finished.
template <class Begin, class Step>
__device__ __forceinline__ void lane_phase(int items, int *next, Begin begin, Step step)
{
    int item = -1;
    for (;;) {
        if (item < 0) {
            do item = atomicAdd(next, 1);
            while (item < items && !begin(item));
        }
        if (!__any_sync(0xffffffffu, item < items)) break;
        if (item < items && step(item)) item = -1;
    }
}

// the walk of getu0 (uvOrb.cpp:109-129)
struct U0Walk {
    double utry, ui, uo;
    int mode, it;
    __device__ void begin() { utry = kUmidStart; mode = 0; it = 0; }
    __device__ bool step(Fudge &o)
    {
        const double dut = o.duturnfn(utry);
        bool done = false;
        if (mode == 0) { ui = uo = utry; mode = dut > 0 ? 1 : 2; }
        else if (++it > kLoopCap) { o.fail |= kFailBracket; done = true; }
        if (!done) {
            if (mode == 1) {
                if (dut > 0) { ui = utry; utry *= 1.2; } else done = true;
            } else {
                if (dut < 0) { uo = utry; utry *= .8; } else done = true;
            }
        }
        if (done) { if (mode == 1) uo = utry; else ui = utry; }
        return done;
    }
};

// the bracket walks of get_turn_u (uvOrb.cpp:131-201): [uin, u1] and [u2, uout],
// or degenerate (uin = uout)
struct UWalk {
    enum : int { kStart, kClimb, kFall, kOutIn, kOut, kIn };
    double utry, eps, u1, u2, uin, uout, fu1;
    int mode, it;
    bool degenerate;
    __device__ void begin() { utry = u1 = u2 = uin = uout = 1; eps = .1; mode = kStart; it = 0; degenerate = false; }
    __device__ bool step(Fudge &o)
    {
        double ut = o.uturnfn(utry), dut = 0;
        if (mode == kStart) {
            fu1 = ut;
            if (ut < 0) {
                dut = o.duturnfn(utry);
                if (dut > 0) { uin = utry; mode = kClimb; } else mode = kFall;
            } else mode = kOutIn;
        } else {
            if ((mode == kClimb || mode == kFall) && ut < 0) dut = o.duturnfn(utry);
            if (++it > kLoopCap) {
                o.fail |= kFailBracket;
                uin = uout = utry;
                return degenerate = true;
            }
        }
        if (mode == kClimb) {
            if (ut < 0 && dut > 0) { uin = utry; utry *= (1 + eps); return false; }
            if (!(ut >= 0)) {
                utry /= (1 + eps); eps *= .2;
                if (eps < kTINY) { uin = uout = utry; return degenerate = true; }
                utry *= (1 + eps);
                return false;
            }
            u1 = utry; mode = kOut;
        } else if (mode == kFall) {
            if (ut < 0 && dut < 0) { uout = utry; utry /= (1 + eps); return false; }
            if (!(ut >= 0)) {
                utry *= (1 + eps); eps *= .2;
                if (eps < kTINY) { uin = uout = utry; return degenerate = true; }
                utry /= (1 + eps);
                return false;
            }
            u2 = utry; mode = kIn;
        }
        if (mode == kOut || mode == kOutIn) {
            if (ut > 0) { u2 = utry; utry *= 1.1; return false; }
            uout = utry;
            if (mode == kOut) return true;
            ut = fu1; mode = kIn;
        }
        if (ut > 0) { u1 = utry; utry *= .9; return false; }
        uin = utry;
        return true;
    }
};

// the walk of get_turn_v (uvOrb.cpp:203-224): [vlo, vhi], or a turning point at a limit
struct VWalk {
    double vtop, vbot, turn;
    int mode, it;
    bool limit;
    __device__ void begin() { vtop = vbot = .5 * kPIH; mode = 0; it = 0; limit = false; }
    __device__ bool step(Fudge &o)
    {
        const double f = o.vturnfn(mode == 2 ? vtop : vbot);
        if (mode == 0) mode = f < 0 ? 1 : 2;
        if (mode == 1) {
            if (!(f < 0)) return true;
            vbot = .5 * (kPIH + vbot);
            if (kPIH - vbot < kTINY) { turn = kPIH; return limit = true; }
            if (++it > kLoopCap) { o.fail |= kFailBracket; turn = kPIH; return limit = true; }
        } else {
            if (!(f > 0)) return true;
            vtop *= .5;
            if (vtop < kTINY) { turn = 0; return limit = true; }
            if (++it > kLoopCap) { o.fail |= kFailBracket; turn = 0; return limit = true; }
        }
        return false;
    }
};

// The actions of n phase points: load(q, Delta, R, z, Phi, vR, vphi, vz) gives
// point q (q < n <= chunk); results and status in S.rec[q].  All threads of a
// kSolveBlock-thread block call it; it ends with a __syncthreads().
template <class Load>
__device__ void solve_orbits64(const PotView &P, const PotFast &F, const GLRule &gl, const double2 *trig, int n, const SolveScratch &S,
                               SolveShared &sh, Load load)
{
    OrbitRec *rec = S.rec;
    if (threadIdx.x < 7) sh.next[threadIdx.x] = 0;
    if (threadIdx.x == 0) sh.nmore = 0;
    for (int q = threadIdx.x; q < n; q += kSolveBlock) {
        double Delta, R, z, Phi, vR, vp, vz;
        load(q, Delta, R, z, Phi, vR, vp, vz);
        OrbitRec &r = rec[q];
        Fudge o;
        const bool bound = fudge_point(P, Delta, R, z, Phi, vR, vp, vz, o, r.pu2, r.pv2);
        r.o = o;
        r.Jr = r.Jz = bound ? 0. : 1e31;
        r.todo = bound ? kOrbitBound : 0u;
        r.more[0] = r.more[1] = r.full[0] = r.full[1] = 0;
        r.rootfail[0] = r.rootfail[1] = r.rootfail[2] = 0;
    }
    __syncthreads();
    {   // u0: bracket, root, then the constants of the equations
        U0Walk w;
        lane_phase(n, &sh.next[0], [&](int q) { w.begin(); return (rec[q].todo & kOrbitBound) != 0; },
                   [&](int q) {
                       if (!w.step(rec[q].o)) return false;
                       rec[q].lo[0] = w.ui; rec[q].hi[0] = w.uo;
                       return true;
                   });
        __syncthreads();
        BrentState b;
        lane_phase(n, &sh.next[1],
                   [&](int q) {
                       if (!(rec[q].todo & kOrbitBound)) return false;
                       b.begin(rec[q].lo[0], rec[q].hi[0]);
                       return true;
                   },
                   [&](int q) {
                       if (!b.feed(rec[q].o.duturnfn(b.x))) return false;
                       rec[q].o.umid = b.root;
                       rec[q].o.fail |= b.fail;
                       return true;
                   });
    }
    __syncthreads();
    for (int q = threadIdx.x; q < n; q += kSolveBlock) {
        if (!(rec[q].todo & kOrbitBound)) continue;
        Fudge o = rec[q].o;
        fudge_constants(o, rec[q].pu2, rec[q].pv2);
        rec[q].o = o;
    }
    __syncthreads();
    {   // turning points: brackets of u and v, then the roots
        UWalk w;
        lane_phase(n, &sh.next[2], [&](int q) { w.begin(); return (rec[q].todo & kOrbitBound) != 0; },
                   [&](int q) {
                       OrbitRec &r = rec[q];
                       if (!w.step(r.o)) return false;
                       r.o.uinner = w.uin; r.o.uouter = w.uout;
                       r.lo[1] = w.uin; r.hi[1] = w.u1; r.lo[2] = w.u2; r.hi[2] = w.uout;
                       if (!w.degenerate) r.todo |= kOrbitRootU;
                       return true;
                   });
        __syncthreads();
        VWalk v;
        lane_phase(n, &sh.next[3], [&](int q) { v.begin(); return (rec[q].todo & kOrbitBound) != 0; },
                   [&](int q) {
                       OrbitRec &r = rec[q];
                       if (!v.step(r.o)) return false;
                       if (v.limit) r.o.vturn = v.turn;
                       else {
                           r.lo[3] = v.vbot < v.vtop ? v.vbot : v.vtop;
                           r.hi[3] = v.vbot < v.vtop ? v.vtop : v.vbot;
                           r.todo |= kOrbitRootV;
                       }
                       return true;
                   });
        __syncthreads();
        BrentState b;
        lane_phase(2 * n, &sh.next[4],
                   [&](int i) {
                       const int k = i < n ? 1 : 2;
                       const OrbitRec &r = rec[i < n ? i : i - n];
                       if (!(r.todo & kOrbitRootU)) return false;
                       b.begin(r.lo[k], r.hi[k]);
                       return true;
                   },
                   [&](int i) {
                       OrbitRec &r = rec[i < n ? i : i - n];
                       if (!b.feed(r.o.uturnfn(b.x))) return false;
                       if (i < n) r.o.uinner = b.root; else r.o.uouter = b.root;
                       r.rootfail[i < n ? 0 : 1] = b.fail;
                       return true;
                   });
        lane_phase(n, &sh.next[5],
                   [&](int q) {
                       if (!(rec[q].todo & kOrbitRootV)) return false;
                       b.begin(rec[q].lo[3], rec[q].hi[3]);
                       return true;
                   },
                   [&](int q) {
                       if (!b.feed(rec[q].o.vturnfn(b.x))) return false;
                       rec[q].o.vturn = b.root;
                       rec[q].rootfail[2] = b.fail;
                       return true;
                   });
    }
    __syncthreads();
    for (int q = threadIdx.x; q < n; q += kSolveBlock) {
        OrbitRec &r = rec[q];
        if (!(r.todo & kOrbitBound)) continue;
        Fudge &o = r.o;
        o.ubar = .5 * (o.uinner + o.uouter);
        o.Deltau = .5 * (o.uouter - o.uinner);
        r.w = kPIH - o.vturn;
        r.fju = fudge_ju_factor(o);
        r.fjv = fudge_jv_factor(o);
        const unsigned todo = (fudge_ju_zero(o) ? 0u : kOrbitJu) | (fudge_jv_zero(o) ? 0u : kOrbitJv);
        r.todo = todo;
        for (int kv = 0; kv < 2 && gl.n > 0; kv++) {  // fixed Gauss-Legendre integrals: on the spot
            if (!(todo & (kv ? kOrbitJv : kOrbitJu))) continue;
            const double b = kv ? kPIH : kPI;
            double s = 0;
            for (int i = 0; i < gl.n; i++) {
                double sn, cs;
                sincos(b * gl.x01[i], &sn, &cs);
                s += (b * gl.w01[i]) * orbit_integrand(P, F, r, kv, sn, cs);
            }
            if (kv) r.Jz = r.fjv * s / kPI; else r.Jr = r.fju * s / kPI;
        }
    }
    __syncthreads();
    if (gl.n > 0) return;
    const int lane = threadIdx.x & 31, g = threadIdx.x / kSolveLanes, gi = threadIdx.x % kSolveLanes;
    const int lead = lane & ~(kSolveLanes - 1);
    const double epsabs = 1e-5, epsrel = 1e-3;  // wrp_GSLinteg, include/Utils.h:173-185
    double *vals = sh.vals[g];
    // first panels of all integrals (item = point, Ju; then point, Jv); an
    // integral that goes on is listed in S.head under its item number
    for (int base = 0; base < 2 * n; base += kSolveGroups) {
        const int item = base + g;
        const bool kv = item >= n;
        const int q = kv ? item - n : item;
        const bool on = item < 2 * n && (rec[q].todo & (kv ? kOrbitJv : kOrbitJu));
        const double b = kv ? kPIH : kPI;
        if (on) {
            const OrbitRec &c = S.rec[q];
            for (int e = gi; e < 21; e += kSolveLanes) {
                double sn, cs;
                panel_sincos(trig, kv, 1u, 0., b, e, sn, cs);
                vals[e] = orbit_integrand(P, F, c, kv, sn, cs);
            }
        }
        __syncwarp();
        if (on && gi == 0) {
            double res, err, ra, rc, r, ae;
            gk_sum<21>(0., b, vals, res, err, ra, rc);
            OrbitRec &c = S.rec[q];
            if (qags_head(res, err, ra, rc, epsabs, epsrel, 1000, r, ae) >= 0) {
                if (kv) c.Jz = c.fjv * r / kPI; else c.Jr = c.fju * r / kPI;
            } else {
                S.head[item] = make_double2(res, err);
                c.more[kv ? 1 : 0] = 1;
                sh.nmore = 1;
            }
        }
        __syncwarp();
    }
    __syncthreads();
    // bisections: items that go on, taken in order as groups free up
    if (sh.nmore > 0) {
        OrbitQags::List &L = S.lists[g];
        OrbitQags st;
        int item = -1;
        double a1 = 0, b2 = 0;
        unsigned heap = 0;
        for (;;) {
            if (gi == 0 && item < 0) {
                for (;;) {
                    item = atomicAdd(&sh.next[6], 1);
                    if (item >= 2 * n) break;
                    const bool kv = item >= n;
                    if (S.rec[kv ? item - n : item].more[kv ? 1 : 0]) {
                        const double2 h = S.head[item];
                        a1 = 0.; b2 = kv ? kPIH : kPI; heap = 1;
                        st.begin(L, a1, b2, h.x, h.y);
                        break;
                    }
                }
            }
            item = __shfl_sync(0xffffffffu, item, lead);
            a1 = __shfl_sync(0xffffffffu, a1, lead);
            b2 = __shfl_sync(0xffffffffu, b2, lead);
            heap = __shfl_sync(0xffffffffu, heap, lead);
            const bool on = item < 2 * n, kv = item >= n;
            if (!__any_sync(0xffffffffu, on)) break;
            const double b1 = 0.5 * (a1 + b2);
            const unsigned h1 = heap < (1u << 30) ? 2 * heap : 0u, h2 = h1 ? h1 + 1u : 0u;
            if (on) {
                const OrbitRec &c = S.rec[kv ? item - n : item];
                for (int e = gi; e < 42; e += kSolveLanes) {
                    const bool second = e >= 21;
                    double sn, cs;
                    panel_sincos(trig, kv, second ? h2 : h1, second ? b1 : a1, second ? b2 : b1, second ? e - 21 : e,
                                 sn, cs);
                    vals[e] = orbit_integrand(P, F, c, kv, sn, cs);
                }
            }
            __syncwarp();
            // the panels' sums on two of the group's lanes
            double res = 0, err = 0, ra, rc = 0;
            if (on && gi % (kSolveLanes / 2) == 0)
                gk_sum<21>(gi ? b1 : a1, gi ? b2 : b1, vals + (gi ? 21 : 0), res, err, ra, rc);
            const double res2 = __shfl_sync(0xffffffffu, res, lead + kSolveLanes / 2), err2 = __shfl_sync(0xffffffffu, err, lead + kSolveLanes / 2),
                         rc2 = __shfl_sync(0xffffffffu, rc, lead + kSolveLanes / 2);
            if (on && gi == 0) {
                double r = 0;
                bool full = false;
                if (st.update(L, res, err, rc, res2, err2, rc2, epsabs, epsrel, r, full)) {
                    OrbitRec &c = S.rec[kv ? item - n : item];
                    if (kv) c.Jz = c.fjv * r / kPI; else c.Jr = c.fju * r / kPI;
                    if (full) c.full[kv ? 1 : 0] = 1;
                    item = -1;
                } else {
                    a1 = L.iv[st.maxerr].a;
                    b2 = L.iv[st.maxerr].b;
                    heap = L.heap[st.maxerr];
                }
            }
            __syncwarp();
        }
    }
    __syncthreads();
}

}  // namespace fj
