// Host build of bracket_near (fjmodels_gb300/csrc/fj_device.cuh): for every radius x and guess of the
// input the interval found and the number of reads of the grid.  Test infrastructure for
// tests/test_bracket_host.py.
//   input (stdin, text): nr, ar[nr], n, then n pairs (x, guess); output: n lines "interval reads"
#define __constant__
#include <cmath>
using std::isfinite;
using std::isnan;
#include <cstdio>
#include <vector>

#include "fj_device.cuh"

int main()
{
    int nr, n;
    if (scanf("%d", &nr) != 1) return 1;
    std::vector<double> ar(nr);
    for (double &r : ar)
        if (scanf("%lf", &r) != 1) return 1;
    if (scanf("%d", &n) != 1) return 1;
    for (int k = 0; k < n; k++) {
        double x;
        int guess, reads = 0;
        if (scanf("%lf %d", &x, &guess) != 2) return 1;
        const int b = fj::bracket_near([&](int i) { reads++; return ar.at(i); }, nr, x, guess);
        printf("%d %d\n", b, reads);
    }
    return 0;
}
