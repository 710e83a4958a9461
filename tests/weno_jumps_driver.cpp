// The integer reconstructions of csrc/weno_fixed.cuh beside jumps, on the host against long double.
// Prints one line a check; see test_weno_jumps.py.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <random>

#include "../2dense_gb300/csrc/weno_fixed.cuh"

#define __device__
#define __forceinline__ inline
namespace fx = dense::fx;
#include "../2dense_gb300/csrc/weno_fast.cuh"
#include "../2dense_gb300/csrc/weno_value.cuh"

typedef long double ld;

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

// fx::pair's value in FP64, as the sweeps form it
template <bool Z> double pair_fp64(double lp, const double gp[4], double lm, const double gm[4]) {
    return about_fp64(lp, lm, correction_fp64<Z>(gp) - correction_fp64<Z>(gm));
}
struct Errors {
    double sum = 0, sum64 = 0, worst = 0, worst64 = 0;
    int n = 0;
    void add(double e, double e64) {
        sum += e * e; sum64 += e64 * e64;
        worst = std::max(worst, e); worst64 = std::max(worst64, e64);
        ++n;
    }
    void print() const { printf("%.17g %.17g %.17g %.17g\n", std::sqrt(sum / n), std::sqrt(sum64 / n), worst, worst64); }
};

// a face's value as the component-wise sweeps form it, on the small side of a jump of 10^decades times
// the level (in both stencils, or in one), relative to the centre values and corrections there. kind 0:
// centre values of the level; 1: centre values zero, as where a transverse flux changes sign
template <bool Z> void sided(int kind, int decades) {
    std::mt19937_64 r(81 + 100 * kind + decades);
    Errors err;
    for (int t = 0; t < 20000; ++t) {
        const double level = std::pow(10.0, 3 * draw(r)), amp = level * std::pow(10.0, -2 + 2 * draw(r));
        const double lp = kind ? 0.0 : level * (1 + 0.3 * draw(r)), lm = kind ? 0.0 : -0.7 * level * (1 + 0.3 * draw(r));
        double gp[4], gm[4], rm[4];
        for (double* g : {gp, gm}) {
            const double a = draw(r), b = 0.3 * draw(r);
            const int j = (int)(r() % 4);
            const double jump = level * std::pow(10.0, decades) * (1 + 0.5 * draw(r)) * (r() & 1 ? 1 : -1);
            for (int m = 0; m < 4; ++m) g[m] = amp * (a + b * (m - 1.5)) + (m == j && (g == gp || t & 1) ? jump : 0.0);
        }
        for (int m = 0; m < 4; ++m) rm[m] = -gm[m];
        const ld cp = correction<Z>(gp), cm = correction<Z>(gm), want = cp + cm + lp + lm;
        bool fp64;
        double h = fx::pair<Z>(lp, gp, lm, rm, &fp64);
        if (fp64) h = pair_fp64<Z>(lp, gp, lm, rm);
        const double h64 = (lp + correction_fp64<Z>(gp)) + (lm + correction_fp64<Z>(gm));
        const double size = std::max(std::fabs(lp), std::fabs(lm)) + (double)(fabsl(cp) + fabsl(cm));
        err.add((double)fabsl(h - want) / size, (double)fabsl(h64 - want) / size);
    }
    printf("sided %d %d %d ", (int)Z, kind, decades);
    err.print();
}
// the forms of pair, through either arithmetic: odd, the same in either order; zeros
template <bool Z> void value_forms() {
    std::mt19937_64 r(91);
    int odd = 0, swap = 0, flat = 0, fp64s = 0;
    auto value = [&](double lp, const double gp[4], double lm, const double gm[4]) {
        bool fp64;
        const double h = fx::pair<Z>(lp, gp, lm, gm, &fp64);
        fp64s += fp64;
        return fp64 ? pair_fp64<Z>(lp, gp, lm, gm) : h;
    };
    for (int t = 0; t < 20000; ++t) {
        double gp[4], gm[4], np[4], nm[4];
        const double lp = draw(r), lm = draw(r);
        for (int m = 0; m < 4; ++m) {
            gp[m] = draw(r) * std::pow(10.0, 3 * draw(r));
            gm[m] = draw(r) * std::pow(10.0, 3 * draw(r));
            np[m] = -gp[m]; nm[m] = -gm[m];
        }
        const double h = value(lp, gp, lm, gm);
        odd += value(-lp, np, -lm, nm) != -h;
        swap += value(lm, nm, lp, np) != h;
        const double zero[4] = {0, -0.0, 0, 0};
        flat += value(lp, zero, lm, zero) != lp + lm;
        flat += value(0.0, zero, 0.0, zero) != 0.0;
    }
    printf("forms %d %d %d %d %d\n", (int)Z, odd, swap, flat, fp64s);
}

int main() {
    for (int kind = 0; kind < 2; ++kind)
        for (int decades : {-3, 0, 1, 2, 4, 6, 10, 14}) { sided<false>(kind, decades); sided<true>(kind, decades); }
    value_forms<false>();
    value_forms<true>();
    between<false>();
    between<true>();
}
