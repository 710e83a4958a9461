// The integer reconstructions of csrc/weno_fixed.cuh beside jumps, on the host against long double.
// Prints one line a check; see test_weno_jumps.py.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <random>

#include "../2dense_gb300/csrc/weno_fixed.cuh"

typedef long double ld;
namespace fx = dense::fx;

static double draw(std::mt19937_64& r) { return std::uniform_real_distribution<double>(-1, 1)(r); }

// what a reconstruction adds to its centre value, from the first differences
template <bool Z> ld correction(const double g[4]) {
    const ld ss = (double)1.0e-6f, cs[3] = {1, 6, 3};
    const ld A[3] = {(ld)g[0] - g[1], (ld)g[1] - g[2], (ld)g[2] - g[3]};
    const ld B[3] = {g[0] - 3 * (ld)g[1], (ld)g[1] + g[2], 3 * (ld)g[2] - g[3]};
    const ld q[3] = {(2 * (ld)g[0] - 5 * (ld)g[1]) / 6, (-(ld)g[1] - 2 * (ld)g[2]) / 6, ((ld)g[3] - 4 * (ld)g[2]) / 6};
    ld d[3], num = 0, den = 0;
    for (int k = 0; k < 3; ++k) d[k] = ss + 13 * A[k] * A[k] / 12 + B[k] * B[k] / 4;
    const ld tau = d[2] - d[0];
    for (int k = 0; k < 3; ++k) {
        const ld w = Z ? cs[k] * (1 + tau / d[k] * (tau / d[k])) : cs[k] / (d[k] * d[k]);
        num += w * q[k];
        den += w;
    }
    return num / den;
}

// two jumps, one at each end of the stencil, a power of two apart, the middle smooth: the error in
// units of the largest value, and what AdaWENO's switch (delta 1/2) takes for smooth
template <bool Z> void between() {
    std::mt19937_64 r(71);
    double worst = 0;
    int smooth = 0;
    for (int t = 0; t < 20000; ++t) {
        const double level = std::pow(10.0, 2 * draw(r)), jump = 1e3 * level * std::pow(10.0, 4 * std::fabs(draw(r))) + 300.0;
        const double rest = level * std::pow(10.0, -3 + 3 * draw(r)), one = std::ldexp(jump, 1 + (int)(r() % 4));
        const double mid = r() & 1 ? rest : 0.0;
        const double g[4] = {r() & 1 ? jump : -jump, mid * draw(r), mid * draw(r), r() & 1 ? one : -one}, flat[4] = {0, 0, 0, 0};
        const double h = fx::pair<Z>(level, g, 0.0, flat);
        worst = std::max(worst, (double)(fabsl(h - (level + correction<Z>(g))) / one));
        fx::u64 a, b;
        smooth += fx::surrogate(g, 0.5, a, b);
    }
    printf("between %d %.17g %d\n", (int)Z, worst, smooth);
}

int main() {
    between<false>();
    between<true>();
}
