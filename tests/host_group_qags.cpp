// Host build of the kernels' QAGS (fjmodels_gb300/csrc/fj_group_qags.cuh: the bookkeeping of one
// group's first lane, in FP64 and FP32) and of the one-thread FP32 form (fj_mixed.cuh).  Test
// infrastructure for tests/test_group_qags_host.py.
#define __constant__
#define __device__
#define __noinline__
#define __forceinline__ inline
#include <cmath>
using std::isfinite;
using std::isnan;
#include <cstdio>
#include <cstring>

#include "fj_group_qags.cuh"
#include "fj_mixed.cuh"

using namespace fj;

namespace {
using F64 = double (*)(double);
using F32 = float (*)(float);

template <int RULE>
int run64(F64 f, double a, double b, double epsabs, double epsrel, double *result, int *full)
{
    constexpr int N = GKRule<RULE>::npts;
    double v[N], res, err, ra, rc, ae;
    for (int e = 0; e < N; e++) v[e] = f(gk_abscissa<RULE>(a, b, e));
    gk_sum<RULE>(a, b, v, res, err, ra, rc);
    *full = 0;
    const int h = qags_head(res, err, ra, rc, epsabs, epsrel, 1000, *result, ae);
    if (h >= 0) return h;
    using Q = GroupQags<double, 256, true, true>;
    static Q::List L;
    Q st;
    st.begin(L, a, b, res, err, ra);
    for (;;) {
        const QagsEntry<double> top = L.iv[st.maxerr];
        const unsigned heap = L.heap[st.maxerr];  // the interval's place in the tree gives its ends
        if (heap) {
            double x = a, y = b;
            for (int bit = 30 - __builtin_clz(heap); bit >= 0; bit--) {
                const double m = 0.5 * (x + y);
                if ((heap >> bit) & 1u) x = m; else y = m;
            }
            if (x != top.a || y != top.b) return -1;
        }
        const double m = 0.5 * (top.a + top.b);
        double r2, e2, c2;
        for (int e = 0; e < N; e++) v[e] = f(gk_abscissa<RULE>(top.a, m, e));
        gk_sum<RULE>(top.a, m, v, res, err, ra, rc);
        for (int e = 0; e < N; e++) v[e] = f(gk_abscissa<RULE>(m, top.b, e));
        gk_sum<RULE>(m, top.b, v, r2, e2, ra, c2);
        bool fl = false;
        if (st.update(L, res, err, rc, r2, e2, c2, epsabs, epsrel, *result, fl)) {
            *full = fl;
            return st.ier_class;
        }
    }
}

GK21f rule21f()
{
    GK21f K;
    for (int i = 0; i < 11; i++) {
        K.xgk[i] = (float)fj_xgk21[i];
        K.wgk[i] = (float)fj_wgk21[i];
        if (i < 5) K.wg[i] = (float)fj_wg10[i];
    }
    return K;
}
}  // namespace

extern "C" int group64(F64 f, int rule, double a, double b, double epsabs, double epsrel, double *result, int *full)
{
    return rule == 21 ? run64<21>(f, a, b, epsabs, epsrel, result, full)
                      : run64<15>(f, a, b, epsabs, epsrel, result, full);
}

extern "C" float group32(F32 f, float a, float b, float epsabs, float epsrel, int *full)
{
    const GK21f K = rule21f();
    float v[21], res, err, ra, rc;
    for (int e = 0; e < 21; e++) v[e] = f(gk21_abscissa(K, a, b, e));
    gk21_sum(K, a, b, v, res, err, ra, rc);
    *full = 0;
    const float tol = fmaxf(epsabs, epsrel * fabsf(res));  // the exits on the first panel, as the kernel has them
    if ((err <= 100 * FLT_EPSILON * ra && err > tol) || (err <= tol && err != rc) || err == 0.0f) return res;
    using Q = GroupQags<float, kQagsCapF>;
    static Q::List L;
    Q st;
    st.begin(L, a, b, res, err);
    for (;;) {
        const QagsEntry<float> top = L.iv[st.maxerr];
        const float m = 0.5f * (top.a + top.b);
        float r2, e2, c2, r;
        for (int e = 0; e < 21; e++) v[e] = f(gk21_abscissa(K, top.a, m, e));
        gk21_sum(K, top.a, m, v, res, err, ra, rc);
        for (int e = 0; e < 21; e++) v[e] = f(gk21_abscissa(K, m, top.b, e));
        gk21_sum(K, m, top.b, v, r2, e2, ra, c2);
        bool fl = false;
        if (st.update(L, res, err, rc, r2, e2, c2, epsabs, epsrel, r, fl)) {
            *full = fl;
            return r;
        }
    }
}

extern "C" float one_thread32(F32 f, float a, float b, float epsabs, float epsrel, int *full)
{
    unsigned fail = 0;
    const float r = qags_f(f, rule21f(), a, b, epsabs, epsrel, fail);
    *full = (fail & kFailQuad) ? 1 : 0;
    return r;
}
