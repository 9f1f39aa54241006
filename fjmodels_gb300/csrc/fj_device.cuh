// fj_device.cuh -- device (and host) math of the fJmodels phase-space path:
// multipole potential and gradient, Brent roots, QUADPACK QAGS, the Staeckel
// fudge and the distribution function.
//
// The building blocks of the kernels: which threads work on an orbit, and where
// its interval lists live, is theirs (fj_solve64.cuh).
//
// Arithmetic follows the reference's expression order where that is free,
// so FP64 results agree with the reference to rounding level.  Deliberate
// differences (all rounding-level): Phi and its gradient at one point share
// one interpolation; cos(acos(c)) is replaced by c; pow(x, 2k+1) by repeated
// products; Phi(pi/2) of the v-equation is evaluated once per orbit.
#pragma once

#include <cfloat>
#include <cmath>

#include "fj_kronrod.h"

#if defined(__CUDACC__)
#define FJ_HD __host__ __device__ __forceinline__
#define FJ_HDNI static __host__ __device__ __noinline__
#define FJ_UNROLL _Pragma("unroll")
#define FJ_UNROLL1 _Pragma("unroll 1")
#else
#define FJ_HD inline
#define FJ_HDNI static inline
#define FJ_UNROLL
#define FJ_UNROLL1
#endif

namespace fj {

// literals of include/Utils.h:56-60
constexpr double kPI = 3.141592653589793;
constexpr double kPIH = 1.570796326794897;
constexpr double kTPI = 6.283185307179586;
constexpr double kFPI = 12.56637061435917;
constexpr double kTINY = 1e-12;

constexpr int kMaxPoly = 24;      // largest supported npoly (l_max = 46)
constexpr int kLoopCap = 4096;    // cap on every bracketing loop (unbounded in the reference)
constexpr int kRootMaxIt = 200;   // cap on Brent iterations
constexpr int kQagsCap = 128;     // interval capacity of a momentum integral's QAGS list

// status bits of one phase-space evaluation
constexpr unsigned kFailBracket = 1u;  // a bracketing loop hit kLoopCap
constexpr unsigned kFailRoot = 2u;     // Brent hit kRootMaxIt
constexpr unsigned kFailQuad = 4u;     // QAGS interval list full (estimate kept)

FJ_HD double dmax(double a, double b) { return a > b ? a : b; }  // MAX of include/Utils.h:47-48

// ----------------------------------------------------------------------------
// multipole potential: tables of include/Grid.h:19-22
// ----------------------------------------------------------------------------
struct PotView {
    int nr, npoly;
    const double *ar, *phil, *Pr, *Pr2;
    const double *itab;  // interpolation constants (interp_table), or null: divide in place
};

// a / b for a divisor whose correctly rounded reciprocal y is at hand: the
// quotient estimate corrected once by its exact remainder (Markstein, IBM J.
// Res. Dev. 34, 1990).  It is the correctly rounded quotient in all but ~2^-50
// of the cases (a tie of the corrected estimate with a rounding boundary), for
// three FP64 operations instead of a division's nine or more: on the GB300 an
// FP64 instruction occupies an SM's FP64 pipe for ~18 cycles whatever the
// number of active lanes, so the kernels that use it are bound by their count.
FJ_HD double div_by(double a, double b, double y)
{
#ifdef __CUDA_ARCH__
    const double q = __dmul_rn(a, y);
    return __fma_rn(__fma_rn(-q, b, a), y, q);
#else
    (void)y;
    return a / b;
#endif
}

// correctly rounded reciprocal of b (the y of div_by)
FJ_HD double recip(double b)
{
#ifdef __CUDA_ARCH__
    return __drcp_rn(b);
#else
    return 1.0 / b;
#endif
}

// Interpolation constants of a radial grid (PotView::itab): two floats for the
// interval guess, then {1 / (ar[n+1] - ar[n])} per interval, then for the
// intervals whose top node is below 10 and each third point (below, above)
// {den, 1/den, f3}, den = (ar[thr]-ar[top]) (ar[thr]-ar[bot]).
constexpr int kQuadTab = 9;
FJ_HD int interp_table_size(int nr) { return 1 + nr + 6 * kQuadTab; }

// entries i0, i0 + stride, .. (a block's threads share the work)
FJ_HD void interp_table(int nr, const double *ar, double *tab, int i0, int stride)
{
    if (i0 == 0) {
        float *g = (float *)tab;
        const float l0 = log2f((float)ar[0]);
        g[0] = l0;
        g[1] = (nr - 1) / (log2f((float)ar[nr - 1]) - l0);
    }
    for (int n = i0; n < nr - 1; n += stride) tab[1 + n] = recip(ar[n + 1] - ar[n]);
    for (int i = i0; i < 2 * kQuadTab; i += stride) {
        const int n = i >> 1, thr = (i & 1) ? n + 2 : n - 1;
        double *q = tab + 1 + nr + 3 * i;
        q[0] = q[1] = q[2] = 0.0;
        if (thr >= 0 && thr < nr && n + 1 < nr) {
            q[0] = (ar[thr] - ar[n + 1]) * (ar[thr] - ar[n]);
            q[1] = recip(q[0]);
            q[2] = (ar[thr] - ar[n]) / (ar[n + 1] - ar[n]);
        }
    }
}

// bracketing search with the semantics of topbottom (include/Utils.h:103-119)
FJ_HD int topbottom(const double *xm, int n, double x, int &bot, int &top)
{
    int t = n - 1, b = 0;
    if ((xm[t] - x) * (x - xm[b]) < 0.) {
        if (fabs(xm[t] - x) < 1e-5 * fabs(x - xm[b])) { top = t; bot = t - 1; return 1; }
        if (fabs(x - xm[b]) < 1e-5 * fabs(x - xm[t])) { top = b + 1; bot = b; return 1; }
        return 0;
    }
    while (t - b > 1) {
        int m = (t + b) / 2;
        if ((xm[t] - x) * (x - xm[m]) >= 0) b = m; else t = m;
    }
    top = t; bot = b;
    return 1;
}

// The interval b with ar[b] <= x < ar[b + 1] (b <= nr - 2) of an increasing grid of
// positive radii, ar[0] <= x <= ar[nr - 1], from a guess: doubling steps away from it until
// x is enclosed, then halving.  A guess that is right costs two reads of the grid
// (at(i)), one that is d intervals off 2 log2(d) + 4: on a grid that is not the guess's
// (which assumes a logarithmic one) never much more than a search without it.
template <class At>
FJ_HD int bracket_near(const At &at, int nr, double x, int guess)
{
#ifdef __CUDA_ARCH__
    // the bit patterns of positive values are ordered as they are, and leave the FP64 pipe alone
    const long long v = __double_as_longlong(x);
    auto below = [&](int i) { return v < __double_as_longlong(at(i)); };
#else
    auto below = [&](int i) { return x < at(i); };
#endif
    int lo = guess, hi = guess + 1;
    if (lo > 0 && below(lo)) {
        int step = 1;
        do {
            hi = lo;
            lo = lo - step > 0 ? lo - step : 0;
            step *= 2;
        } while (lo > 0 && below(lo));
    } else {
        int step = 1;
        while (hi < nr - 1 && !below(hi)) {
            lo = hi;
            hi = hi + step < nr - 1 ? hi + step : nr - 1;
            step *= 2;
        }
    }
    while (hi - lo > 1) {
        const int m = (lo + hi) >> 1;
        if (below(m)) hi = m; else lo = m;
    }
    return lo;
}

// interpolation weights of intpo2 (include/UtilsLeg.h:96-158) at one radius
struct Interp {
    int bot, top, thr;
    bool ext, quad;
    double f1, f2, f3, x;  // x = ar[nr-1]/r beyond the grid
};

FJ_HD void interp_setup(const PotView &P, double r, Interp &I)
{
    const double *ar = P.ar;
    const int nr = P.nr;
    // every field is set on both branches: the callers' ternaries read both
    I.bot = I.top = I.thr = 0;
    I.f1 = I.f2 = I.f3 = 0.0;
    I.x = 0.0;
    if (r >= ar[nr - 1]) { I.ext = true; I.quad = false; I.x = ar[nr - 1] / r; return; }
    I.ext = false;
#ifdef __CUDA_ARCH__
    if (P.itab && __double_as_longlong(r) >= __double_as_longlong(ar[0])) {
        const double *tab = P.itab;
        const float2 g = *(const float2 *)tab;
        // interval from the logarithmic spacing (log2 of the leading bits, no
        // FP64 operation), corrected by neighbour tests on the bit patterns
        // (ordered like the positive values): any increasing grid gives the
        // bracketing interval.  A radius on a grid node may take either
        // neighbour, which give the same value.
        const long long rb = __double_as_longlong(r);
        const int hi = (int)(rb >> 32);
        const float m = __int_as_float(0x3f800000 | ((hi & 0xfffff) << 3) | (int)(((unsigned)rb) >> 29));
        const float lr = (float)((hi >> 20) - 1023) + __log2f(m);
        int b = (int)((lr - g.x) * g.y);
        b = b < 0 ? 0 : (b > nr - 2 ? nr - 2 : b);
        while (b > 0 && rb < __double_as_longlong(ar[b])) --b;
        while (b < nr - 2 && rb > __double_as_longlong(ar[b + 1])) ++b;
        const double ab = ar[b], at = ar[b + 1], db = r - ab;
        I.f1 = div_by(db, at - ab, tab[1 + b]);
        I.bot = b; I.top = b + 1; I.thr = b + 1;
        I.quad = b < kQuadTab;
        if (I.quad) {
            const bool up = !(I.f1 < 0.5 && b > 0);
            I.thr = up ? b + 2 : b - 1;
            const double *q = tab + 1 + nr + 3 * (2 * b + (up ? 1 : 0));
            I.f2 = div_by((r - at) * db, q[0], q[1]);
            I.f3 = q[2];
        }
        return;
    }
#endif
    int top = 0, bot = 0;
    topbottom(ar, nr, r, bot, top);
    const double db = r - ar[bot];
    I.f1 = db / (ar[top] - ar[bot]);
    I.bot = bot; I.top = top;
    I.quad = top < 10;
    if (I.quad) {
        const int thr = (I.f1 < 0.5 && bot > 0) ? bot - 1 : top + 1;
        const double dt = r - ar[top];
        I.f2 = dt * db / ((ar[thr] - ar[top]) * (ar[thr] - ar[bot]));
        I.f3 = (ar[thr] - ar[bot]) / (ar[top] - ar[bot]);
        I.thr = thr;
    } else {
        I.thr = top; I.f2 = 0; I.f3 = 0;
    }
}

FJ_HD double interp_in(const Interp &I, const double *T, int npoly, int k)
{
    const double vt = T[I.top * npoly + k], vb = T[I.bot * npoly + k];
    double v = I.f1 * vt + (1 - I.f1) * vb;
    if (I.quad) {
        const double vh = T[I.thr * npoly + k];
        v += I.f2 * (vh - vb - I.f3 * (vt - vb));
    }
    return v;
}

// next even Legendre polynomial P_{2np} from P_{2np-4}, P_{2np-2} (UtilsLeg.h:68-79), np >= 2
// (on the device the divisions by functions of np come from a table: one
// corrected product and two products instead of three divisions)
struct LegCoef { double l, lm1, D, rD, B, C; };
struct LegTable { LegCoef c[kMaxPoly]; };
constexpr LegTable make_leg_table()
{
    LegTable t{};
    for (int np = 2; np < kMaxPoly; np++) {
        const int l = 2 * (np - 1), l2 = 2 * l;
        LegCoef &o = t.c[np];
        o.l = l; o.lm1 = l - 1;
        o.D = (double)((l2 + 1) * (l2 - 1));
        o.rD = 1.0 / o.D;
        o.B = (l2 * l + l2 - 1) / (double)((l2 - 1) * (l2 + 3));
        o.C = (l2 + 1) * (l2 + 3) / (double)((l + 1) * (l + 2));
    }
    return t;
}
// reciprocals of the small integers (the full recurrence divides by its degree)
struct IntRecip { double y[2 * kMaxPoly + 2]; };
constexpr IntRecip make_int_recip()
{
    IntRecip t{};
    for (int i = 1; i < 2 * kMaxPoly + 2; i++) t.y[i] = 1.0 / i;
    return t;
}
#if defined(__CUDACC__)
static __constant__ LegTable kLeg_d = make_leg_table();
static __constant__ IntRecip kIntRecip_d = make_int_recip();
#endif

FJ_HD double evenleg_next(int np, double c2, double pm2, double pm1)
{
#ifdef __CUDA_ARCH__
    const LegCoef &t = kLeg_d.c[np];
    return (div_by(-pm2 * t.l * t.lm1, t.D, t.rD) + pm1 * (c2 - t.B)) * t.C;
#endif
    const int l = 2 * (np - 1), l2 = 2 * l;
    double p = -pm2 * l * (l - 1) / (double)((l2 + 1) * (l2 - 1)) +
               pm1 * (c2 - (l2 * l + l2 - 1) / (double)((l2 - 1) * (l2 + 3)));
    p *= (l2 + 1) * (l2 + 3) / (double)((l + 1) * (l + 2));
    return p;
}

// P_i of the full Legendre recurrence from P_{i-1}, P_{i-2} (dlegend, UtilsLeg.h:43-57), i >= 2
FJ_HD double fullleg_next(int i, double c, double Pl, double Pl_m1)
{
    const double a = (2 * i - 1) * c * Pl - (i - 1) * Pl_m1;
#ifdef __CUDA_ARCH__
    return div_by(a, (double)i, kIntRecip_d.y[i]);
#else
    return a / (double)i;
#endif
}

// Phi(R,z): Potential::operator() (pot/Potential.cpp:206-219)
FJ_HDNI double pot_phi(const PotView &P, double R, double z)
{
    const double r = sqrt(R * R + z * z);
    const double c = z / r;
    Interp I;
    interp_setup(P, (r >= P.ar[P.nr - 1]) ? r : dmax(r, P.ar[0]), I);
    const int np_ = P.npoly;
    const double *T = P.phil;
    const double x2 = I.ext ? I.x * I.x : 0.0;
    double xp = I.x;
    double phi = I.ext ? T[(P.nr - 1) * np_] * xp : interp_in(I, T, np_, 0);
    if (np_ < 2) return phi;
    const double c2 = c * c;
    double pm2 = 1.0, pm1 = 1.5 * c2 - .5;
    xp *= x2;
    phi += (I.ext ? T[(P.nr - 1) * np_ + 1] * xp : interp_in(I, T, np_, 1)) * pm1;
    for (int k = 2; k < np_; k++) {
        const double pk = evenleg_next(k, c2, pm2, pm1);
        xp *= x2;
        phi += (I.ext ? T[(P.nr - 1) * np_ + k] * xp : interp_in(I, T, np_, k)) * pk;
        pm2 = pm1; pm1 = pk;
    }
    return phi;
}

// Phi, dPhi/dR, dPhi/dz at one point: operator(), dR, dz of pot/Potential.cpp:206-276
// sharing one bracket search.  dtheta uses the full Legendre recurrence
// (dlegend, UtilsLeg.h:43-57), dr the even one, as the reference does.
FJ_HDNI void pot_grad(const PotView &P, double R, double z, double &phi, double &dR, double &dz)
{
    const double *ar = P.ar;
    const int np_ = P.npoly, nr = P.nr;
    const double r0 = sqrt(R * R + z * z);
    double r = r0;
    if (r < ar[0]) r = ar[0];
    // the four quotients by r share its reciprocal while that is a normal number
    const bool near = r < 1e150;
    const double ir = near ? recip(r) : 1.0;
    auto over_r = [&](double a) { return near ? div_by(a, r, ir) : a / r; };
    const double s = over_r(R);
    double c = over_r(z);
    const double cphi = r == r0 ? c : z / r0;
    if (c == 1) c -= 1e-8;
    Interp I;
    interp_setup(P, r, I);
    const double x2 = I.ext ? I.x * I.x : 0.0;
    double xp = I.x;
    const double cp2 = cphi * cphi, cc2 = c * c, omc = 1 - c * c, iomc = recip(omc);
    const bool same = cp2 == cc2;  // inside the grid: one even recurrence serves both
    // even polys at cphi (potential) and at c (radial derivative)
    double ep2 = 1, ep1 = 0, ec2 = 1, ec1 = 0;
    // full recurrence at c: Pl_m1 = P_{n-1}, Pl = P_n
    double Pl_m1 = 0, Pl = 1;
    double gphi = 0, gdr = 0, gdth = 0;
    for (int k = 0; k < np_; k++) {
        double ph, dph;
        if (I.ext) {
            const double t = P.phil[(nr - 1) * np_ + k];
            ph = t * xp;
            dph = over_r(-(2 * k + 1) * t * xp);
            xp *= x2;
        } else {
            ph = interp_in(I, P.phil, np_, k);
            dph = interp_in(I, P.Pr, np_, k);
        }
        double pe_phi, pe_c;
        if (k == 0) { pe_phi = 1; pe_c = 1; }
        else if (k == 1) { pe_phi = 1.5 * cp2 - .5; pe_c = 1.5 * cc2 - .5; ep1 = pe_phi; ec1 = pe_c; }
        else {
            pe_phi = evenleg_next(k, cp2, ep2, ep1); ep2 = ep1; ep1 = pe_phi;
            if (same) pe_c = pe_phi;
            else pe_c = evenleg_next(k, cc2, ec2, ec1);
            ec2 = ec1; ec1 = pe_c;
        }
        // advance the full recurrence to n = 2k
        double dleg = 0;
        if (k > 0) {
            const int n = 2 * k;
            const double P1 = k == 1 ? c : fullleg_next(n - 1, c, Pl, Pl_m1);
            const double P2 = fullleg_next(n, c, P1, Pl);
            Pl_m1 = P1; Pl = P2;
            dleg = div_by(n * Pl_m1 - n * c * Pl, omc, iomc);
        }
        if (k == 0) gphi = ph; else gphi += ph * pe_phi;
        gdr += dph * pe_c;
        gdth += ph * dleg;
    }
    gdth *= -sqrt(omc);
    phi = gphi;
    dR = gdth * over_r(c) + gdr * s;
    dz = gdth * over_r(-s) + gdr * c;
}

// Potential::dr with its second derivative (pot/Potential.cpp:224-234); r not clamped
FJ_HD double pot_dr2(const PotView &P, double r, double c, double &d2)
{
    const int np_ = P.npoly, nr = P.nr;
    Interp I;
    interp_setup(P, r, I);
    const double x2 = I.ext ? I.x * I.x : 0.0, cc2 = c * c;
    double xp = I.x, ec2 = 1, ec1 = 0, g1 = 0, g2 = 0;
    for (int k = 0; k < np_; k++) {
        double dph, d2ph;
        if (I.ext) {
            const double t = P.phil[(nr - 1) * np_ + k];
            dph = -(2 * k + 1) * t * xp / r;
            d2ph = (2 * k + 2) * (2 * k + 1) * t * xp / r / r;
            xp *= x2;
        } else {
            dph = interp_in(I, P.Pr, np_, k);
            d2ph = interp_in(I, P.Pr2, np_, k);
        }
        double pe;
        if (k == 0) pe = 1;
        else if (k == 1) { pe = 1.5 * cc2 - .5; ec1 = pe; }
        else { pe = evenleg_next(k, cc2, ec2, ec1); ec2 = ec1; ec1 = pe; }
        g1 += dph * pe;
        g2 += d2ph * pe;
    }
    d2 = g2;
    return g1;
}

// sum_k Phi_k(r) * dP_{2k}/dc and * d2P_{2k}/dc2 (dtheta / d2theta pieces, Potential.cpp:235-255)
FJ_HD void pot_theta_sums(const PotView &P, double r, double c, double &s1, double &s2)
{
    const int np_ = P.npoly, nr = P.nr;
    Interp I;
    interp_setup(P, (r >= P.ar[nr - 1]) ? r : dmax(r, P.ar[0]), I);
    const double x2 = I.ext ? I.x * I.x : 0.0;
    double xp = I.x, Pl_m1 = 0, Pl = 1;
    int nfull = 0;
    s1 = 0; s2 = 0;
    for (int k = 0; k < np_; k++) {
        double ph;
        if (I.ext) { ph = P.phil[(nr - 1) * np_ + k] * xp; xp *= x2; }
        else ph = interp_in(I, P.phil, np_, k);
        double d1 = 0, dd2 = 0;
        const int n = 2 * k;
        if (k > 0) {
            while (nfull < n) {
                const int i = nfull + 1;
                const double Pn = (i == 1) ? c : fullleg_next(i, c, Pl, Pl_m1);
                Pl_m1 = Pl; Pl = Pn; nfull = i;
            }
            d1 = (n * Pl_m1 - n * c * Pl) / (1 - c * c);
        }
        dd2 = (2 * c * d1 - n * (n + 1) * Pl) / (1. - c * c);
        s1 += ph * d1;
        s2 += ph * dd2;
    }
}

// epicycle frequencies getfreqs (pot/Potential.cpp:281-296)
FJ_HDNI void pot_freqs(const PotView &P, double R, double &kappa, double &nu, double &Omega)
{
    const double cth = 6.123233995736766e-17;  // cos(asin(1)) in double
    double d2, phi, dRv, dzv;
    pot_dr2(P, R, cth, d2);
    const double d2R = d2;
    const double g1 = pot_dr2(P, R, cth, d2);
    double s1, s2;
    pot_theta_sums(P, R, 0.0, s1, s2);
    const double dth = s1 * -sqrt(1 - 0.0 * 0.0);
    double d2th = s2 * (1 - 0.0 * 0.0);
    d2th += ((dth * 0.0) / sqrt(1 - 0.0 * 0.0));
    const double d2z = (1. / R) * g1 + (1. / (R * R)) * d2th;
    pot_grad(P, R, 0, phi, dRv, dzv);
    kappa = sqrt(d2R + 3 / R * dRv);
    nu = sqrt(d2z);
    Omega = sqrt(dRv / R);
}

// ----------------------------------------------------------------------------
// Brent root with the stopping rule of wrp_GSLroots (include/Utils.h:134-167)
// ----------------------------------------------------------------------------
FJ_HD bool same_sign(double x, double y) { return (x < 0 && y < 0) || (x > 0 && y > 0); }

// The iteration of brent_root as a state that is fed one function value at a time:
// x is the next abscissa, feed(f(x)) returns true when root (and fail) are final.
struct BrentState {
    double a, fa, b, fb, c, fc, d, e, x, root;
    int it;  // -2: f(lo) awaited, -1: f(hi), >= 0: iterations done
    unsigned fail;
    FJ_HD void begin(double lo, double hi)
    {
        a = x = lo; b = hi; it = -2; fail = 0;
        fa = fb = c = fc = d = e = root = 0;
    }
    FJ_HD bool feed(double f)
    {
        if (it == -2) {
            if (fabs(f) < 5e-4) { root = a; return true; }
            fa = f; x = b; it = -1;
            return false;
        }
        if (it == -1) {
            if (fabs(f) < 5e-4) { root = b; return true; }
            fb = f; c = b; fc = f; d = b - a; e = d;
            it = 0;
        } else {
            fb = f;
            const double cc = same_sign(fb, fc) ? a : c;
            const double xlo = b < cc ? b : cc, xhi = b < cc ? cc : b;
            const double alo = fabs(xlo), ahi = fabs(xhi);
            const double mn = ((xlo > 0 && xhi > 0) || (xlo < 0 && xhi < 0)) ? (alo < ahi ? alo : ahi) : 0.0;
            if (fabs(xhi - xlo) < 1e-8 + 1e-6 * mn && !(xhi - xlo > 1e-8)) { root = b; return true; }
            it++;
        }
        for (;;) {
            if (it >= kRootMaxIt) { root = b; fail = kFailRoot; return true; }
            bool secant = false;
            if (same_sign(fb, fc)) { secant = true; c = a; fc = fa; d = b - a; e = b - a; }
            if (fabs(fc) < fabs(fb)) { secant = true; a = b; b = c; c = a; fa = fb; fb = fc; fc = fa; }
            const double tol = 0.5 * DBL_EPSILON * fabs(b);
            const double m = 0.5 * (c - b);
            if (fb == 0) { root = b; return true; }
            if (fabs(m) <= tol) {  // no step left: the wrapper's test on [b, c], which only a huge b fails
                const double xlo = b < c ? b : c, xhi = b < c ? c : b, alo = fabs(xlo), ahi = fabs(xhi);
                const double mn = ((xlo > 0 && xhi > 0) || (xlo < 0 && xhi < 0)) ? (alo < ahi ? alo : ahi) : 0.0;
                if (fabs(xhi - xlo) < 1e-8 + 1e-6 * mn && !(xhi - xlo > 1e-8)) { root = b; return true; }
                it++;
                continue;
            }
            if (fabs(e) < tol || fabs(fa) <= fabs(fb)) { d = m; e = m; }
            else {
                const double sr = fb / fa;
                double pn, q;
                if (secant) { pn = 2 * m * sr; q = 1 - sr; }
                else {
                    q = fa / fc;
                    const double r = fb / fc;
                    pn = sr * (2 * m * q * (q - r) - (b - a) * (r - 1));
                    q = (q - 1) * (r - 1) * (sr - 1);
                }
                if (pn > 0) q = -q; else pn = -pn;
                const double lim1 = 3 * m * q - fabs(tol * q), lim2 = fabs(e * q);
                if (2 * pn < (lim1 < lim2 ? lim1 : lim2)) { e = d; d = pn / q; }
                else { d = m; e = m; }
            }
            a = b; fa = fb;
            if (fabs(d) > tol) b += d; else b += (m > 0 ? +tol : -tol);
            x = b;
            return false;
        }
    }
};

template <class F>
FJ_HDNI unsigned brent_root(F &f, double lo, double hi, double &root)
{
    BrentState s;
    s.begin(lo, hi);
    while (!s.feed(f(s.x))) {}
    root = s.root;
    return s.fail;
}

// ----------------------------------------------------------------------------
// QUADPACK QAGS (Piessens et al. 1983: DQAGSE, DQK21/DQK15): the panels and the
// decision on the first one.  The bisections (fj_group_qags.cuh) keep a list of
// kQagsCap intervals; a full list stops the refinement, keeps the current estimate
// and sets kFailQuad.
// ----------------------------------------------------------------------------
FJ_HD double rescale_err(double err, double resabs, double resasc)
{
    err = fabs(err);
    if (resasc != 0 && err != 0) {
#ifdef __CUDA_ARCH__
        const double ratio = 200 * err / resasc, scale = ratio * sqrt(ratio);  // an estimate: its last bit decides nothing
#else
        const double scale = pow(200 * err / resasc, 1.5);
#endif
        err = scale < 1 ? resasc * scale : resasc;
    }
    if (resabs > DBL_MIN / (50 * DBL_EPSILON)) {
        const double min_err = 50 * DBL_EPSILON * resabs;
        if (min_err > err) err = min_err;
    }
    return err;
}

// Gauss-Kronrod panels (DQK21, DQK15) as abscissas and sums, so that one
// lane or a whole warp can evaluate a panel's function values: the e-th
// abscissa (e < 2 nk - 1) in the evaluation order of the QUADPACK routine --
// the centre, then -/+ the Gauss-point offsets xgk[1], xgk[3], .., then -/+
// xgk[0], xgk[2], .. -- and the sums over the values in that order.
template <int RULE>
struct GKRule {
    static constexpr int nk = RULE == 21 ? 11 : 8;  // Kronrod abscissas in [0, 1]
    static constexpr int npts = 2 * nk - 1;         // function values per panel
    static constexpr int n1 = (nk - 1) / 2;         // Gauss-point pairs
};

FJ_HD double dmul_rn(double x, double y)
{
#ifdef __CUDA_ARCH__
    return __dmul_rn(x, y);
#else
    return x * y;
#endif
}
FJ_HD double dadd_rn(double x, double y)
{
#ifdef __CUDA_ARCH__
    return __dadd_rn(x, y);
#else
    return x + y;
#endif
}

template <int RULE>
FJ_HD void gk_tables(const double *&xgk, const double *&wgk, const double *&wg)
{
#ifdef __CUDA_ARCH__
    xgk = RULE == 21 ? fj_xgk21_d : fj_xgk15_d;
    wgk = RULE == 21 ? fj_wgk21_d : fj_wgk15_d;
    wg = RULE == 21 ? fj_wg10_d : fj_wg7_d;
#else
    xgk = RULE == 21 ? fj_xgk21 : fj_xgk15;
    wgk = RULE == 21 ? fj_wgk21 : fj_wgk15;
    wg = RULE == 21 ? fj_wg10 : fj_wg7;
#endif
}

template <int RULE>
FJ_HD double gk_abscissa(double a, double b, int e)
{
    using G = GKRule<RULE>;
    const double *xgk, *wgk, *wg;
    gk_tables<RULE>(xgk, wgk, wg);
    const double center = dmul_rn(0.5, dadd_rn(a, b)), half = dmul_rn(0.5, dadd_rn(b, -a));
    if (e == 0) return center;
    const int jj = e <= 2 * G::n1 ? 2 * ((e - 1) >> 1) + 1 : 2 * ((e - 1 - 2 * G::n1) >> 1);
    const double x = dmul_rn(half, xgk[jj]);
    return ((e - 1) & 1) ? dadd_rn(center, x) : dadd_rn(center, -x);
}

template <int RULE>
FJ_HD void gk_sum(double a, double b, const double *v, double &res, double &abserr, double &resabs, double &resasc)
{
    using G = GKRule<RULE>;
    constexpr int nk = G::nk, n1 = G::n1;
    const double *xgk, *wgk, *wg;
    gk_tables<RULE>(xgk, wgk, wg);
    const double half = dmul_rn(0.5, dadd_rn(b, -a)), ahalf = fabs(half);
    const double fc = v[0];
    double rg = 0, rk = fc * wgk[nk - 1], ra = fabs(rk);
    if (nk % 2 == 0) rg = fc * wg[nk / 2 - 1];
FJ_UNROLL
    for (int j = 0; j < n1; j++) {
        const int jj = 2 * j + 1;
        const double f1 = v[1 + 2 * j], f2 = v[2 + 2 * j];
        rg += wg[j] * (f1 + f2);
        rk += wgk[jj] * (f1 + f2);
        ra += wgk[jj] * (fabs(f1) + fabs(f2));
    }
FJ_UNROLL
    for (int j = 0; j < nk / 2; j++) {
        const int jj = 2 * j;
        const double f1 = v[1 + 2 * n1 + 2 * j], f2 = v[2 + 2 * n1 + 2 * j];
        rk += wgk[jj] * (f1 + f2);
        ra += wgk[jj] * (fabs(f1) + fabs(f2));
    }
    const double mean = 0.5 * rk;
    double rasc = wgk[nk - 1] * fabs(fc - mean);
FJ_UNROLL
    for (int jj = 0; jj < nk - 1; jj++) {
        const int em = (jj & 1) ? jj : 1 + 2 * n1 + jj;
        rasc += wgk[jj] * (fabs(v[em] - mean) + fabs(v[em + 1] - mean));
    }
    const double err = (rk - rg) * half;
    rk *= half; ra *= ahalf; rasc *= ahalf;
    res = rk; resabs = ra; resasc = rasc;
    abserr = rescale_err(err, ra, rasc);
}

// QAGS on [a,b] after its first panel: returns the QUADPACK error class of a call
// that the panel finishes (result and abserr set), or -1 when bisections follow
// (fj_group_qags.cuh).  limit is the reference's nominal limit.
FJ_HD int qags_head(double res0, double err0, double resabs0, double resasc0, double epsabs, double epsrel, int limit,
                    double &result, double &abserr)
{
    const double tol = epsabs > epsrel * fabs(res0) ? epsabs : epsrel * fabs(res0);
    if (err0 <= 100 * DBL_EPSILON * resabs0 && err0 > tol) { result = res0; abserr = err0; return 2; }
    if ((err0 <= tol && err0 != resasc0) || err0 == 0.0) { result = res0; abserr = err0; return 0; }
    if (limit == 1) { result = res0; abserr = err0; return 1; }
    return -1;
}

// ----------------------------------------------------------------------------
// Staeckel fudge (uvOrb/uvOrb.cpp, uvOrb/Uvpt.cpp) in FP64
// ----------------------------------------------------------------------------
struct Fudge {
    PotView P;
    double Delta, E, Er, Iv, Lzsq;
    double u, v, shu2, sv, cv, sv2;
    double sinv, cosv;     // sin(v), cos(v) as pt(Delta,u,v) recomputes them
    double sinhu, coshu;   // sinh(u), cosh(u) of the point
    double sh1sq, ch1sq, Phiu1, PhivPIH;
    double uinner, uouter, umid, vturn, ubar, Deltau;
    // what the u and v equations repeat at every evaluation (set by prepare)
    double LzD2, ish1, Erch, B0, C0, hL, DD, Dshu, Dchu;
    unsigned fail;

    FJ_HD void prepare()
    {
        DD = Delta * Delta;
        hL = .5 * Lzsq;
        LzD2 = hL / DD;
        ish1 = 1 / sh1sq;
        Erch = Er * ch1sq;
        B0 = (sh1sq + sv2) * Phiu1;
        C0 = (1 + shu2) * PhivPIH;
        Dshu = Delta * sinhu;
        Dchu = Delta * coshu;
    }

    FJ_HD double Phiu(double shu, double chu) const { return pot_phi(P, Delta * shu * sinv, Delta * chu * cosv); }
    FJ_HD double dU(double u_) const
    {
        const double shu = sinh(u_);
        return (shu * shu + sv2) * Phiu(shu, cosh(u_)) - (sh1sq + sv2) * Phiu1;
    }
    FJ_HD double Phiv(double sn, double cs) const { return pot_phi(P, Delta * sinhu * sn, Delta * coshu * cs); }
    FJ_HD double vturnfn(double v_) const
    {
        double sn, cs;
        sincos(v_, &sn, &cs);
        const double s2 = sn * sn;
        const double dV = C0 - (shu2 + s2) * pot_phi(P, Dshu * sn, Dchu * cs);
        return E * s2 + Iv + dV - hL / (DD * s2);
    }
    FJ_HD double uturnfn(double u_) const
    {
        const double shu = sinh(u_), chu = cosh(u_), s2 = shu * shu;
        const double dUv = (s2 + sv2) * Phiu(shu, chu) - B0;
        return E * (s2 - sh1sq) + Erch - dUv - LzD2 * (1 / s2 - ish1);
    }
    FJ_HD double duturnfn(double u_) const
    {
        const double shu = sinh(u_), chu = cosh(u_), s2 = shu * shu;
        double phi0, f0, f1;
        pot_grad(P, Delta * shu * sinv, Delta * chu * cosv, phi0, f0, f1);
        const double dPhidu = Delta * (f0 * chu * sv + f1 * shu * cv);
        return 2 * (E - phi0) * shu * chu - (s2 + sv2) * dPhidu + Lzsq * chu / (Delta * Delta * s2 * shu);
    }
};

struct UturnF { const Fudge *o; FJ_HD double operator()(double x) const { return o->uturnfn(x); } };
struct DuturnF { const Fudge *o; FJ_HD double operator()(double x) const { return o->duturnfn(x); } };
struct VturnF { const Fudge *o; FJ_HD double operator()(double x) const { return o->vturnfn(x); } };
// uvOrb::GetTurnu (uvOrb.cpp:131-201)
FJ_HDNI void get_turn_u(Fudge &o, double utry)
{
    UturnF U{&o};
    DuturnF D{&o};
    double u1 = utry, u2 = utry;
    double ut = U(utry), dut = D(utry), eps = .1;
    int it = 0;
    bool capped = false;
#define FJ_CAP()                                                        \
    if (++it > kLoopCap) { capped = true; break; }
    if (ut < 0) {
        if (dut > 0) {
            o.uinner = utry;
            while (!capped) {
                while (ut < 0 && dut > 0) {
                    o.uinner = utry; utry *= (1 + eps);
                    ut = U(utry); dut = D(utry);
                    FJ_CAP();
                }
                if (capped) break;
                if (ut >= 0) { u1 = utry; break; }
                utry /= (1 + eps); eps *= .2;
                if (eps < kTINY) { o.uinner = o.uouter = utry; return; }
                utry *= (1 + eps);
                ut = U(utry); dut = D(utry);
                FJ_CAP();
            }
            while (!capped && ut > 0) { u2 = utry; utry *= 1.1; ut = U(utry); FJ_CAP(); }
            o.uouter = utry;
        } else {
            while (!capped) {
                while (ut < 0 && dut < 0) {
                    o.uouter = utry; utry /= (1 + eps);
                    ut = U(utry); dut = D(utry);
                    FJ_CAP();
                }
                if (capped) break;
                if (ut >= 0) { u2 = utry; break; }
                utry *= (1 + eps); eps *= .2;
                if (eps < kTINY) { o.uinner = o.uouter = utry; return; }
                utry /= (1 + eps);
                ut = U(utry); dut = D(utry);
                FJ_CAP();
            }
            while (!capped && ut > 0) { u1 = utry; utry *= .9; ut = U(utry); FJ_CAP(); }
            o.uinner = utry;
        }
    } else {
        const double fu1 = ut;
        while (ut > 0) { u2 = utry; utry *= 1.1; ut = U(utry); FJ_CAP(); }
        o.uouter = utry;
        ut = fu1;
        while (!capped && ut > 0) { u1 = utry; utry *= .9; ut = U(utry); FJ_CAP(); }
        o.uinner = utry;
    }
#undef FJ_CAP
    if (capped) { o.fail |= kFailBracket; o.uinner = o.uouter = utry; return; }
    o.fail |= brent_root(U, o.uinner, u1, o.uinner);
    o.fail |= brent_root(U, u2, o.uouter, o.uouter);
}

// uvOrb::GetTurnv (uvOrb.cpp:203-224)
FJ_HDNI double get_turn_v(Fudge &o, double vtry)
{
    VturnF V{&o};
    double vtop = vtry, vbot = vtry;
    int it = 0;
    if (V(vtry) < 0) {
        while (V(vbot) < 0) {
            vbot = .5 * (kPIH + vbot);
            if (kPIH - vbot < kTINY) return kPIH;
            if (++it > kLoopCap) { o.fail |= kFailBracket; return kPIH; }
        }
    } else {
        while (V(vtop) > 0) {
            vtop *= .5;
            if (vtop < kTINY) return 0;
            if (++it > kLoopCap) { o.fail |= kFailBracket; return 0; }
        }
    }
    double r;
    if (!(vbot < vtop)) o.fail |= brent_root(V, vtop, vbot, r);
    else o.fail |= brent_root(V, vbot, vtop, r);
    return r;
}

// Momentum-integral rule: QAGS as wrp_GSLinteg (include/Utils.h:173-185) or fixed
// Gauss-Legendre.
struct GLRule {
    int n;              // 0 = QAGS
    const double *x01;  // nodes on (0,1)
    const double *w01;  // weights on (0,1)
};

// One phase-space point up to the reference point of the u-equation: uvOrb ctor
// (uvOrb.cpp:15-22), pt (Uvpt.cpp:11-24); pu2, pv2 the squared momenta.  Returns
// false for an unbound orbit.
FJ_HDNI bool fudge_point(const PotView &P, double Delta, double R, double z, double Phi, double pR, double vphi,
                         double pz, Fudge &o, double &pu2, double &pv2)
{
    o.P = P;
    o.fail = 0;
    o.Delta = Delta;
    const double Lz = R * vphi;
    o.Lzsq = Lz * Lz;
    const double Delta2 = Delta * Delta, R2 = R * R, z2 = z * z, r2 = R2 + z2;
    const double dmr = Delta2 - r2, dpr = Delta2 + r2;
    const double shu2 = .5 * (r2 - Delta2 + sqrt(dmr * dmr + 4 * Delta2 * R2)) / Delta2;
    const double shu = sqrt(shu2);
    o.u = asinh(shu);
    const double chu = sqrt(1 + shu2);
    const double cv2 = .5 * (r2 + Delta2 - sqrt(dpr * dpr - 4 * Delta2 * z2)) / Delta2;
    const double cv = z < 0 ? -sqrt(cv2) : sqrt(cv2);
    o.v = acos(cv);
    o.sv = sin(o.v);
    o.sv2 = 1 - cv2;
    o.shu2 = shu2;
    o.cv = cv;
    const double p2 = pR * pR + pz * pz;
    const double pu = Delta * (pR * chu * o.sv + pz * shu * cv);
    const double pv = Delta * (pR * shu * cv - pz * chu * o.sv);
    pu2 = pu * pu;
    pv2 = pv * pv;
    o.E = .5 * p2 + .5 * o.Lzsq / (R * R) + Phi;
    if (o.E >= 0 || isnan(o.E)) return false;
    sincos(o.v, &o.sinv, &o.cosv);
    o.sinhu = sinh(o.u);
    o.coshu = cosh(o.u);
    return true;
}

// The rest of the ctor (uvOrb.cpp:22-36) once o.umid is known: Er, Iv and what the
// equations repeat
FJ_HDNI void fudge_constants(Fudge &o, double pu2, double pv2)
{
    const double Delta2 = o.Delta * o.Delta, shu2 = o.shu2;
    {
        const double s = sinh(o.umid), c = cosh(o.umid);
        o.sh1sq = s * s; o.ch1sq = c * c;
        o.Phiu1 = o.Phiu(s, c);
    }
    o.PhivPIH = o.Phiv(sin(kPIH), cos(kPIH));
    o.Er = -o.E * (shu2 - o.sh1sq) / o.ch1sq + .5 * pu2 / (Delta2 * o.ch1sq) +
           .5 * o.Lzsq / (Delta2 * o.ch1sq) * (1 / shu2 - 1 / o.sh1sq) + o.dU(o.u) / o.ch1sq;
    {
        double sn, cs;
        sincos(o.v, &sn, &cs);
        const double dVv = (1 + o.shu2) * o.PhivPIH - (o.shu2 + sn * sn) * o.Phiv(sn, cs);
        o.Iv = .5 * pv2 / Delta2 - o.E * o.sv2 + .5 * o.Lzsq / (Delta2 * o.sv2) - dVv;
    }
    o.prepare();
}

constexpr double kUmidStart = 58;  // where getu0 starts (uvOrb.cpp:23)

// whether Ju and Jv vanish (uvOrb.cpp:226-229, 247-249), and their factors
// before the integrals (uvOrb.cpp:238, 256)
FJ_HD bool fudge_ju_zero(const Fudge &o) { return fabs(o.uouter - o.uinner) < kTINY; }
FJ_HD bool fudge_jv_zero(const Fudge &o) { return fabs(o.vturn - kPIH) < kTINY; }
FJ_HD double fudge_ju_factor(const Fudge &o) { return sqrt(2.0) * o.Delta * o.Deltau; }
FJ_HD double fudge_jv_factor(const Fudge &o) { return 2 * sqrt(2.0) * o.Delta * (kPIH - o.vturn); }

// ----------------------------------------------------------------------------
// focal distance and DF
// ----------------------------------------------------------------------------
// Deltafn (delta/tabulate.cpp:40-44) with linterp (Utils.h:122-128)
FJ_HD double deltafn(const double *Eg, const double *Dg, int n, double E)
{
    if (E < Eg[0]) return sqrt(dmax(.000001, Dg[0]));
    if (E < Eg[n - 1]) {
        double y;
        if (E <= Eg[0]) y = Dg[0];
        else {
            int top = 0, bot = 0;
            topbottom(Eg, n, E, bot, top);
            y = Dg[bot] + (E - Eg[bot]) / (Eg[top] - Eg[bot]) * (Dg[top] - Dg[bot]);
        }
        return sqrt(dmax(.000001, y));
    }
    return sqrt(dmax(.000001, Dg[n - 1]));
}

struct DFDev {
    int kind;
    double alpha, beta, J0, norm, tpi3, dphi_h, dz_h, dphi_g, dz_g, chi, k;
};

// GetRc (include/Utils.h:195-214): circular radius for Lz^2
FJ_HDNI double get_rc(const PotView &P, double Lzsq, double R, unsigned &fail)
{
    struct RcF {
        const PotView *P; double Lzsq;
        FJ_HD double operator()(double x) const
        {
            double phi, dR, dz;
            pot_grad(*P, x, 0, phi, dR, dz);
            return Lzsq / (x * x * x) - dR;
        }
    } f{&P, Lzsq};
    double Ri = R, Ro = R, dfRt = f(R);
    int it = 0;
    if (dfRt > 0) {
        while (dfRt > 0) { Ri = R; R *= 1.2; dfRt = f(R); if (++it > kLoopCap) { fail |= kFailBracket; break; } }
        Ro = R;
    } else {
        while (dfRt < 0) { Ro = R; R *= .8; dfRt = f(R); if (++it > kLoopCap) { fail |= kFailBracket; break; } }
        Ri = R;
    }
    double r;
    fail |= brent_root(f, Ri, Ro, r);
    return r;
}

// df() (df/DF.cpp:78-124) from the actions; NaN -> 0 as DF.cpp:105
FJ_HD double df_value(const DFDev &d, const PotView &P, double R, double Jr, double Jz, double Jphi,
                      unsigned &fail)
{
    double DF;
    if (d.kind == 1) {
        const double rc = get_rc(P, Jphi * Jphi, R, fail);
        double kappa, nu, Omega;
        pot_freqs(P, rc, kappa, nu, Omega);
        const double sigmar = exp(-rc / 2.) * 5.;
        const double sigmaz = exp(-rc / 4.) * .316;
        const double fr = Omega * 1e-1 * exp(-rc / 1.) / (kPI * sigmar * sigmar * kappa) * (1. + tanh(Jphi / .1)) *
                          exp(-kappa * Jr / (sigmar * sigmar));
        const double fz = nu / (2 * kPI * sigmaz * sigmaz) * exp(-2 * Jz / (sigmaz * sigmaz));
        DF = dmax(0., fr * fz);
    } else {
        const double h = Jr + d.dphi_h * fabs(Jphi) + d.dz_h * Jz;
        const double g = Jr + d.dphi_g * fabs(Jphi) + d.dz_g * Jz;
        const double DFeven = d.norm * dmax(0., pow(1. + d.J0 / h, d.alpha) / (pow(1. + g / d.J0, d.beta))) / d.tpi3;
        DF = d.chi == 0. ? DFeven : DFeven + d.k * tanh(d.chi * Jphi / d.J0) * DFeven;
    }
    if (isnan(DF)) return 0.;
    return DF;
}

}  // namespace fj
