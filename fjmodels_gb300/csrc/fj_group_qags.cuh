// fj_group_qags.cuh -- QUADPACK QAGS (DQAGSE) by a group of G lanes of a warp,
// 32 / G integrals at a time.
//
// One thread per integral leaves most of a warp idle: the number of panels per
// integral runs from 1 to over 100, so after a few bisections the lanes are at
// different places of different integrals.  Here the G lanes of a group share
// each panel's 21 function values, and all groups of a warp go through the same
// loop -- evaluate the 42 points of one bisection, sum, update -- each on its own
// integral; a group that finishes takes the next integral from the block's list.
// With G = 4 the 42 points are 11 rounds (95 % of the lanes busy), an integral's
// serial chain is a quarter as long, and a warp keeps 8 interval lists instead
// of 32.  The function values enter the same sums in the same order as in the
// one-thread form (qags_f), and the bookkeeping is its, statement by
// statement, so an integral has the same bits.
//
// The bookkeeping runs on the group's first lane only; the others receive the
// interval to bisect from it.
#pragma once

#include <cfloat>

#include "fj_device.cuh"

namespace fj {

template <class T> struct QagsNum;
template <> struct QagsNum<double> {
    static constexpr double eps = DBL_EPSILON, tiny = DBL_MIN, huge = DBL_MAX;
};
template <> struct QagsNum<float> {
    static constexpr float eps = FLT_EPSILON, tiny = FLT_MIN, huge = FLT_MAX;
};
__device__ __forceinline__ double qmax(double a, double b) { return a > b ? a : b; }
__device__ __forceinline__ float qmax(float a, float b) { return fmaxf(a, b); }
__device__ __forceinline__ double qabs(double a) { return fabs(a); }
__device__ __forceinline__ float qabs(float a) { return fabsf(a); }

template <class T> struct alignas(4 * sizeof(T)) QagsEntry { T a, b, r, e; };

// interval list, order and epsilon table of one group (in device memory, where
// the entries in use stay in L1)
template <class T, int CAP, bool HEAP = false>
struct QagsList {
    static constexpr bool kHeap = HEAP;  // whether the intervals carry their number in the bisection tree
    QagsEntry<T> iv[CAP];
    T eps[52], res3[3];
    unsigned heap[HEAP ? CAP : 1];  // root 1, halves of h: 2h and 2h + 1; 0 beyond 2^30
    unsigned char iord[CAP];
};

// Wynn epsilon step (DQELG; tab[0..n-1] with room for n+2; the result count advances
// only on completed updates, as in GSL), as qelg_f
template <class T>
__device__ __noinline__ void group_qelg(T *tab, int &n_io, T *res3, int &nres, T &result, T &abserr)
{
    constexpr T EPS = QagsNum<T>::eps, HUGE_ = QagsNum<T>::huge;
    const int n = n_io - 1;
    const T current = tab[n];
    result = current;
    abserr = HUGE_;
    if (n < 2) return;
    tab[n + 2] = tab[n];
    tab[n] = HUGE_;
    const int newelm = n / 2;
    int n_final = n;
    for (int i = 0; i < newelm; i++) {
        T res = tab[n - 2 * i + 2];
        const T e0 = tab[n - 2 * i - 2], e1 = tab[n - 2 * i - 1], e2 = res;
        const T e1abs = qabs(e1);
        const T delta2 = e2 - e1, err2 = qabs(delta2);
        const T tol2 = qmax(qabs(e2), e1abs) * EPS;
        const T delta3 = e1 - e0, err3 = qabs(delta3);
        const T tol3 = qmax(e1abs, qabs(e0)) * EPS;
        if (err2 <= tol2 && err3 <= tol3) {
            const T rel = 5 * EPS * qabs(res);
            result = res;
            abserr = qmax(err2 + err3, rel);
            return;
        }
        const T e3 = tab[n - 2 * i];
        tab[n - 2 * i] = e1;
        const T delta1 = e1 - e3, err1 = qabs(delta1);
        const T tol1 = qmax(e1abs, qabs(e3)) * EPS;
        if (err1 <= tol1 || err2 <= tol2 || err3 <= tol3) { n_final = 2 * i; break; }
        const T ss = (1 / delta1 + 1 / delta2) - 1 / delta3;
        if (qabs(ss * e1) <= T(0.0001)) { n_final = 2 * i; break; }
        res = e1 + 1 / ss;
        tab[n - 2 * i] = res;
        const T error = err2 + qabs(res - e2) + err3;
        if (error <= abserr) { abserr = error; result = res; }
    }
    if (n_final == 49) n_final = 48;
    if (n % 2 == 1) { for (int i = 0; i <= newelm; i++) tab[1 + 2 * i] = tab[2 * i + 3]; }
    else { for (int i = 0; i <= newelm; i++) tab[2 * i] = tab[2 * i + 2]; }
    if (n != n_final) for (int i = 0; i <= n_final; i++) tab[i] = tab[n - n_final + i];
    n_io = n_final + 1;
    if (nres < 3) { res3[nres] = result; abserr = HUGE_; }
    else {
        abserr = qabs(result - res3[2]) + qabs(result - res3[1]) + qabs(result - res3[0]);
        res3[0] = res3[1]; res3[1] = res3[2]; res3[2] = result;
    }
    nres += 1;
    abserr = qmax(5 * EPS * qabs(result), abserr);
}

// The state of one integral after its first panel (the first lane's registers)
// IER: also the QUADPACK error class of a finished integral (ier)
template <class T, int CAP, bool HEAP = false, bool IER = false>
struct GroupQags {
    using List = QagsList<T, CAP, HEAP>;
    int ier_class;
    T res0_, resabs;
    T area, errsum, errmax, res_ext, err_ext, correc, ertest, erlarg, small, len;
    int maxerr, nrmax, last, numrl2, nres, ktmin, ierro, iroff1, iroff2, iroff3;
    bool extrap, noext;

    // res0, err0: the first panel on [a, b], which did not finish the integral
    __device__ void begin(List &L, T a, T b, T res0, T err0, T resabs0 = 0)
    {
        if (IER) { res0_ = res0; resabs = resabs0; ier_class = 0; }
        L.iv[0] = QagsEntry<T>{a, b, res0, err0};
        if (HEAP) L.heap[0] = 1;
        L.iord[0] = 0;
        L.eps[0] = res0;
        area = res0; errsum = err0; errmax = err0;
        res_ext = res0; err_ext = QagsNum<T>::huge;
        correc = ertest = erlarg = small = 0;
        len = qabs(b - a);
        maxerr = nrmax = 0; last = 1; numrl2 = 1; nres = 0;
        ktmin = ierro = iroff1 = iroff2 = iroff3 = 0;
        extrap = noext = false;
    }

    __device__ T list_sum(const List &L, int n) const
    {
        T s = 0;
        for (int k = 0; k <= n; k++) s += L.iv[k].r;
        return s;
    }

    // The two half panels [a1, b1], [b1, b2] of interval maxerr: results, errors
    // and their resasc.  Returns true when the integral is finished (result, and
    // full if the list had no room left), else maxerr is the next interval.
    __device__ bool update(List &L, T area1, T error1, T rasc1, T area2, T error2, T rasc2, T epsabs,
                           T epsrel, T &result, bool &full)
    {
        constexpr T EPS = QagsNum<T>::eps, TINY_ = QagsNum<T>::tiny, HUGE_ = QagsNum<T>::huge;
        const QagsEntry<T> top = L.iv[maxerr];
        const T a1 = top.a, b1 = T(0.5) * (top.a + top.b), a2 = b1, b2 = top.b;
        const unsigned h = HEAP ? L.heap[maxerr] : 0u, h1 = h < (1u << 30) ? 2 * h : 0u, h2 = h1 ? h1 + 1u : 0u;
        const T erlast = errmax;
        const T area12 = area1 + area2, erro12 = error1 + error2;
        int ier = 0;  // a class set in one bisection always ends the loop there
        errsum = errsum + erro12 - errmax;
        area = area + area12 - top.r;
        if (!(rasc1 == error1 || rasc2 == error2)) {
            if (qabs(top.r - area12) <= T(1e-5) * qabs(area12) && erro12 >= T(0.99) * errmax) {
                if (extrap) iroff2++; else iroff1++;
            }
            if (last > 9 && erro12 > errmax) iroff3++;
        }
        const T errbnd = qmax(epsabs, epsrel * qabs(area));
        if (iroff1 + iroff2 >= 10 || iroff3 >= 20) ier = 2;
        if (iroff2 >= 5) ierro = 3;
        if (qmax(qabs(a1), qabs(b2)) <= (1 + 100 * EPS) * (qabs(a2) + 1000 * TINY_)) ier = 4;
        if (!(error2 > error1)) {
            L.iv[maxerr] = QagsEntry<T>{a1, b1, area1, error1};
            L.iv[last] = QagsEntry<T>{a2, b2, area2, error2};
            if (HEAP) { L.heap[maxerr] = h1; L.heap[last] = h2; }
        } else {
            L.iv[maxerr] = QagsEntry<T>{a2, b2, area2, error2};
            L.iv[last] = QagsEntry<T>{a1, b1, area1, error1};
            if (HEAP) { L.heap[maxerr] = h2; L.heap[last] = h1; }
        }
        {   // DQPSRT with 1-based positions
            unsigned char *iord = L.iord;
            const int N = last + 1;
            if (N <= 2) { iord[0] = 0; iord[1] = 1; }
            else {
                const T em = L.iv[maxerr].e;
                int nr1 = nrmax + 1;
                if (nr1 != 1) {
                    const int ido = nr1 - 1;
                    for (int i = 1; i <= ido; i++) {
                        const int isucc = iord[nr1 - 2];
                        if (em <= L.iv[isucc].e) break;
                        iord[nr1 - 1] = (unsigned char)isucc;
                        nr1--;
                    }
                }
                const int jupbn = N, jbnd = jupbn - 1, ibeg = nr1 + 1;
                const T errmin = L.iv[N - 1].e;
                int i = ibeg;
                bool found = false;
                if (ibeg <= jbnd) {
                    for (i = ibeg; i <= jbnd; i++) {
                        const int isucc = iord[i - 1];
                        if (em >= L.iv[isucc].e) { found = true; break; }
                        iord[i - 2] = (unsigned char)isucc;
                    }
                }
                if (!found) { iord[jbnd - 1] = (unsigned char)maxerr; iord[jupbn - 1] = (unsigned char)(N - 1); }
                else {
                    iord[i - 2] = (unsigned char)maxerr;
                    int k = jbnd;
                    bool ins = false;
                    for (int j = i; j <= jbnd; j++) {
                        const int isucc = iord[k - 1];
                        if (errmin < L.iv[isucc].e) { iord[k] = (unsigned char)(N - 1); ins = true; break; }
                        iord[k] = (unsigned char)isucc;
                        k--;
                    }
                    if (!ins) iord[i - 1] = (unsigned char)(N - 1);
                }
                nrmax = nr1 - 1;
            }
            maxerr = iord[nrmax];
            errmax = L.iv[maxerr].e;
        }
        bool stop = false;  // the loop ends here
        if (errsum <= errbnd) {
            if (IER) ier_class = ier > 2 ? ier - 1 : ier;
            result = list_sum(L, last);
            return true;
        }
        if (ier) stop = true;
        else if (last == 1) {
            small = len * T(0.375);
            erlarg = errsum;
            ertest = errbnd;
            L.eps[1] = area; numrl2 = 2;
        } else if (!noext) {
            erlarg -= erlast;
            if (qabs(b1 - a1) > small) erlarg += erro12;
            bool go = true;
            if (!extrap) {
                if (qabs(L.iv[maxerr].b - L.iv[maxerr].a) > small) go = false;
                else { extrap = true; nrmax = 1; }
            }
            if (go && !(ierro == 3 || erlarg <= ertest)) {
                for (int k = nrmax + 1; k <= last + 1; k++) {
                    maxerr = L.iord[nrmax];
                    errmax = L.iv[maxerr].e;
                    if (qabs(L.iv[maxerr].b - L.iv[maxerr].a) > small) { go = false; break; }
                    nrmax++;
                }
            }
            if (go) {
                L.eps[numrl2] = area; numrl2++;
                T reseps, abseps;
                group_qelg<T>(L.eps, numrl2, L.res3, nres, reseps, abseps);
                ktmin++;
                if (ktmin > 5 && err_ext < T(1e-3) * errsum) ier = 5;
                if (abseps < err_ext) {
                    ktmin = 0;
                    err_ext = abseps;
                    res_ext = reseps;
                    correc = erlarg;
                    ertest = qmax(epsabs, epsrel * qabs(reseps));
                    if (err_ext <= ertest) stop = true;
                }
                if (!stop) {
                    if (numrl2 == 1) noext = true;
                    if (ier == 5) stop = true;
                    else {
                        maxerr = L.iord[0];
                        errmax = L.iv[maxerr].e;
                        nrmax = 0;
                        extrap = false;
                        small *= T(0.5);
                        erlarg = errsum;
                    }
                }
            }
        }
        if (!stop) {
            last++;
            if (last < CAP) return false;
            full = true;  // no room for another interval: the estimate so far
            result = list_sum(L, CAP - 1);
            return true;
        }
        bool take_sum = false;
        if (err_ext == HUGE_) take_sum = true;
        else if (ier + ierro != 0) {
            if (ierro == 3) err_ext += correc;
            if (res_ext != 0 && area != 0) {
                if (err_ext / qabs(res_ext) > errsum / qabs(area)) take_sum = true;
            } else if (err_ext > errsum) take_sum = true;
        }
        if (IER) {
            bool skip_div = false;
            if (err_ext != HUGE_ && ier + ierro != 0) {
                if (ier == 0) ier = 3;
                if (!(res_ext != 0 && area != 0) && !take_sum && area == 0) skip_div = true;
            }
            if (!take_sum && !skip_div) {
                const int ksgn = qabs(res0_) >= (1 - 50 * EPS) * resabs ? 1 : -1;
                if (!(ksgn == -1 && qmax(qabs(res_ext), qabs(area)) <= resabs * T(0.01))) {
                    const T ratio = res_ext / area;
                    if (ratio < T(0.01) || ratio > 100 || errsum > qabs(area)) ier = 6;
                }
            }
            ier_class = ier > 2 ? ier - 1 : ier;
        }
        result = take_sum ? list_sum(L, last) : res_ext;
        return true;
    }
};

}  // namespace fj
