// Host build of the mixed form's evaluator (pot_dphi_f of fjmodels_gb300/csrc/fj_mixed.cuh) with the
// tables that the kernels give it (evaluator_tables_f) and its multipole loop unrolled, against the
// form without either.  Test infrastructure for tests/test_evaluator_host.py.
//   input (stdin, text): nr npoly, ar[nr], phil[nr*npoly], n, then n lines "R z R' z'" (grid point, position)
//   output: n lines of three values in hexadecimal: plain, with tables, with tables and unrolled
#define __constant__
#include <cmath>
using std::isfinite;
using std::isnan;
#include <cstdio>
#include <cstring>
#include <vector>

#include "fj_mixed.cuh"

using namespace fj;

template <int NP>
float unrolled(int np, const PotViewF &P, float R, float z, float rpt, float dr2, float dc2, float Phipt)
{
    if constexpr (NP > 8) return pot_dphi_f<0>(P, R, z, rpt, dr2, dc2, Phipt);
    else return np == NP ? pot_dphi_f<NP>(P, R, z, rpt, dr2, dc2, Phipt)
                         : unrolled<NP + 1>(np, P, R, z, rpt, dr2, dc2, Phipt);
}

int main()
{
    int nr, np, n;
    if (scanf("%d %d", &nr, &np) != 2) return 1;
    std::vector<double> ar(nr), phil((size_t)nr * np);
    for (auto *v : {&ar, &phil})
        for (double &x : *v)
            if (scanf("%lf", &x) != 1) return 1;
    if (scanf("%d", &n) != 1) return 1;
    const PotView P{nr, np, ar.data(), phil.data(), phil.data(), phil.data()};
    std::vector<float> far(nr), fphil((size_t)nr * np), fPr((size_t)nr * np), ih(nr), qc(4 * kQuadIntervals), pyl(np),
        pd(2 * (size_t)nr * np), pe(2 * kQuadIntervals * (size_t)np);
    for (int i = 0; i < n; i++) {
        double R, z, x, y;
        if (scanf("%lf %lf %lf %lf", &R, &z, &x, &y) != 4) return 1;
        const double Phi = pot_phi(P, R, z);
        mixed_tables_f(nr, np, ar.data(), phil.data(), phil.data(), Phi, R, z, far.data(), fphil.data(), fPr.data(),
                       ih.data(), qc.data(), pyl.data(), 0, 1);
        PotViewF V = mixed_view_f(nr, np, ar.data(), phil.data(), Phi, R, z, far.data(), fphil.data(), fPr.data(),
                                  ih.data(), qc.data(), pyl.data());
        const float Phipt = pot_phi_f(V, (float)R, (float)z), rpt = (float)sqrt(R * R + z * z);
        const float dr2 = (float)(x * x + y * y - R * R - z * z),
                    dc2 = (float)(y * y / (x * x + y * y) - z * z / (R * R + z * z));
        float v[3];
        v[0] = pot_dphi_f<0>(V, (float)x, (float)y, rpt, dr2, dc2, Phipt);
        evaluator_tables_f(V, phil.data(), Phi, pd.data(), pe.data(), 0, 1);
        V.pd = pd.data();
        V.pe = pe.data();
        v[1] = pot_dphi_f<0>(V, (float)x, (float)y, rpt, dr2, dc2, Phipt);
        v[2] = unrolled<3>(np, V, (float)x, (float)y, rpt, dr2, dc2, Phipt);
        unsigned u[3];
        memcpy(u, v, sizeof u);
        printf("%08x %08x %08x %.9g %.17g\n", u[0], u[1], u[2], v[0], pot_phi(P, x, y) - Phi);
    }
    return 0;
}
