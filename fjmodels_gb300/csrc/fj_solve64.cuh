// fj_solve64.cuh -- the plain FP64 action solves of a list of phase points by
// one block: turning points one point per thread, momentum integrals by groups
// of lanes (fj_group_qags.cuh).
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
// The values are those of fudge_actions, bit for bit up to div_by's rounding.
// Measured (GB300), one thread per orbit with in-place divisions before, this
// after: one iteration of a 16x6 model with 22^3 nodes 581 -> 230 ms, moments at
// 6 points 111 -> 22.6 ms, 40 line-profile values 181 -> 68.8 ms, 20 001 actions
// 34.8 -> 16.6 ms.
#pragma once

#include "fj_group_qags.cuh"

namespace fj {

constexpr int kSolveBlock = 128;                        // threads of a solving block
constexpr int kSolveLanes = 4;                          // lanes per momentum integral
constexpr int kSolveGroups = kSolveBlock / kSolveLanes;  // integrals in flight
constexpr int kTrigPanels = 1024;                       // bisection tree down to 1/512 of the range

// What a point's integrals need after its turning points, and its actions
struct OrbitRec {
    double E, Delta, sinv, cosv, sv2, sh1sq, Erch, B0, LzD2, ish1, ubar, Deltau;  // Ju
    double w, Dshu, Dchu, shu2, C0, Iv, hL, DD;                                   // Jv
    double fju, fjv;                                                              // factors of the integrals
    double Jr, Jz;                                                                // results
    unsigned fail, todo;      // kFail* bits of the turning points; 1: Ju to integrate, 2: Jv
    int more[2], full[2];     // Ju, Jv: goes on after its first panel; its list was full
    __device__ unsigned status() const { return fail | (full[0] | full[1] ? kFailQuad : 0u); }
};

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
    int next, nmore;                // list position; whether any integral goes on
};

__device__ __forceinline__ double orbit_integrand(const PotView &P, const OrbitRec &c, bool kv, double sn, double cs)
{
    double R, z, s2;
    if (!kv) {  // uvOrb.cpp:226-239
        const double u = c.ubar - c.Deltau * cs;
        const double shu = sinh(u), chu = cosh(u);
        s2 = shu * shu;
        R = c.Delta * shu * c.sinv;
        z = c.Delta * chu * c.cosv;
    } else {  // uvOrb.cpp:247-257
        double s, k;
        sincos(kPIH - c.w * cs, &s, &k);
        s2 = s * s;
        R = c.Dshu * s;
        z = c.Dchu * k;
    }
    const double phi = pot_phi(P, R, z);
    double f;
    if (!kv) {
        const double dUv = (s2 + c.sv2) * phi - c.B0;
        f = c.E * (s2 - c.sh1sq) + c.Erch - dUv - c.LzD2 * (1 / s2 - c.ish1);
    } else {
        const double dV = c.C0 - (c.shu2 + s2) * phi;
        f = c.E * s2 + c.Iv + dV - c.hL / (c.DD * s2);
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

// The actions of n phase points: load(q, Delta, R, z, Phi, vR, vphi, vz) gives
// point q (q < n <= chunk); results and status in S.rec[q].  All threads of a
// kSolveBlock-thread block call it; it ends with a __syncthreads().
template <class Load>
__device__ void solve_orbits64(const PotView &P, const GLRule &gl, const double2 *trig, int n, const SolveScratch &S,
                               SolveShared &sh, Load load)
{
    if (threadIdx.x == 0) { sh.next = kSolveBlock; sh.nmore = 0; }
    __syncthreads();
    // turning points, points taken as threads free up
    for (int q = threadIdx.x; q < n;) {
        double Delta, R, z, Phi, vR, vp, vz;
        load(q, Delta, R, z, Phi, vR, vp, vz);
        OrbitRec &r = S.rec[q];
        r.more[0] = r.more[1] = r.full[0] = r.full[1] = 0;
        Fudge o;
        if (!fudge_turning_points(P, Delta, R, z, Phi, vR, vp, vz, o)) {
            r.Jr = r.Jz = 1e31;
            r.fail = r.todo = 0;
        } else {
            r.E = o.E; r.Delta = Delta; r.sinv = o.sinv; r.cosv = o.cosv; r.sv2 = o.sv2; r.sh1sq = o.sh1sq;
            r.Erch = o.Erch; r.B0 = o.B0; r.LzD2 = o.LzD2; r.ish1 = o.ish1; r.ubar = o.ubar; r.Deltau = o.Deltau;
            r.w = kPIH - o.vturn; r.Dshu = o.Dshu; r.Dchu = o.Dchu; r.shu2 = o.shu2; r.C0 = o.C0; r.Iv = o.Iv;
            r.hL = o.hL; r.DD = o.DD;
            r.fju = fudge_ju_factor(o); r.fjv = fudge_jv_factor(o);
            r.Jr = r.Jz = 0;
            unsigned todo = (fudge_ju_zero(o) ? 0u : 1u) | (fudge_jv_zero(o) ? 0u : 2u);
            if (gl.n > 0) {  // fixed Gauss-Legendre integrals: on the spot
                JuIntF fju{&o};
                JvIntF fjv{&o};
                if (todo & 1u) r.Jr = r.fju * mom_integral(fju, kPI, gl, o.fail) / kPI;
                if (todo & 2u) r.Jz = r.fjv * mom_integral(fjv, kPIH, gl, o.fail) / kPI;
                todo = 0;
            }
            r.fail = o.fail;
            r.todo = todo;
        }
        q = atomicAdd(&sh.next, 1);
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
        const bool on = item < 2 * n && (S.rec[q].todo & (kv ? 2u : 1u));
        const double b = kv ? kPIH : kPI;
        if (on) {
            const OrbitRec &c = S.rec[q];
            for (int e = gi; e < 21; e += kSolveLanes) {
                double sn, cs;
                panel_sincos(trig, kv, 1u, 0., b, e, sn, cs);
                vals[e] = orbit_integrand(P, c, kv, sn, cs);
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
    if (threadIdx.x == 0) sh.next = 0;
    __syncthreads();
    if (sh.nmore > 0) {
        OrbitQags::List &L = S.lists[g];
        OrbitQags st;
        int item = -1;
        double a1 = 0, b2 = 0;
        unsigned heap = 0;
        for (;;) {
            if (gi == 0 && item < 0) {
                for (;;) {
                    item = atomicAdd(&sh.next, 1);
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
                    vals[e] = orbit_integrand(P, c, kv, sn, cs);
                }
            }
            __syncwarp();
            // the panels' sums on the group's first and third lanes
            double res = 0, err = 0, ra, rc = 0;
            if (on && (gi & 1) == 0)
                gk_sum<21>(gi ? b1 : a1, gi ? b2 : b1, vals + (gi ? 21 : 0), res, err, ra, rc);
            const double res2 = __shfl_sync(0xffffffffu, res, lead + 2), err2 = __shfl_sync(0xffffffffu, err, lead + 2),
                         rc2 = __shfl_sync(0xffffffffu, rc, lead + 2);
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
