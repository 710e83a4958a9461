// The integer reconstructions of csrc/weno_fixed.cuh beside jumps, on the host against long double.
// Prints one line a check; see test_weno_jumps.py.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <limits>
#include <random>

#include "../2dense_gb300/csrc/weno_fixed.cuh"

#define __device__
#define __forceinline__ inline
namespace fx = dense::fx;
#include "../2dense_gb300/csrc/weno_fast.cuh"
#include "../2dense_gb300/csrc/weno_value.cuh"
#include "../2dense_gb300/csrc/char_fast.cuh"

typedef long double ld;

static double draw(std::mt19937_64& r) { return std::uniform_real_distribution<double>(-1, 1)(r); }

// what a reconstruction adds to its centre value, from the first differences
template <bool Z, typename T> ld correction_of(const T g[4]) {
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

template <bool Z> ld correction(const double g[4]) { return correction_of<Z>(g); }

// the weights over the linear ones, from the first differences
static void weights_of(const double g[4], ld w[3]) {
    const ld ss = (double)1.0e-6f, cs[3] = {0.1L, 0.6L, 0.3L};
    const ld A[3] = {(ld)g[0] - g[1], (ld)g[1] - g[2], (ld)g[2] - g[3]};
    const ld B[3] = {g[0] - 3 * (ld)g[1], (ld)g[1] + g[2], 3 * (ld)g[2] - g[3]};
    ld d[3], sum = 0;
    for (int k = 0; k < 3; ++k) d[k] = ss + 13 * A[k] * A[k] / 12 + B[k] * B[k] / 4;
    for (int k = 0; k < 3; ++k) sum += w[k] = cs[k] * (1 + (d[2] - d[0]) / d[k] * ((d[2] - d[0]) / d[k]));
    for (int k = 0; k < 3; ++k) w[k] /= sum;
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

// A face's four fluxes of the characteristic schemes beside a jump of about `ratio` times the level in
// density, pressure and velocities (the tangential one zero on the small side now and then), with the
// Roe state as given: char_fields and char_field_fp64 as the sweeps put them together, and an FP64
// reconstruction of the fields' values, centre included. Errors relative to each flux's centre values and itself.
void fields(double ratio) {
    std::mt19937_64 r((unsigned)(500 + 10 * std::log10(ratio)));
    const double g = 1.4;
    Errors err[4];
    for (int t = 0; t < 10000; ++t) {
        const int j = 1 + (int)(r() % 5);
        const bool left = r() & 1;
        const double jr = 1 + ratio * (0.5 + std::fabs(draw(r))), jp = 1 + ratio * (0.5 + 3 * std::fabs(draw(r)));
        const double amp = std::pow(10.0, -3 + 2 * draw(r)), p0 = 0.1 + std::fabs(draw(r)), u0 = 2 * draw(r);
        const double v0 = r() % 3 ? draw(r) : 0.0, du = 2 * draw(r), dv = r() % 3 ? 2 * draw(r) : 0.0;
        double F[2][6][4], cell[6][4], lam = 0;
        for (int m = 0; m < 6; ++m) {
            const bool big = left ? m < j : m >= j;
            const double x = m - 2.5;
            cell[m][0] = (1 + amp * (0.1 * draw(r) + 0.1 * x)) * (big ? jr : 1);
            cell[m][1] = u0 + amp * (0.1 * draw(r) + 0.2 * x) + (big ? du : 0);
            cell[m][2] = (v0 != 0 ? v0 + amp * (0.1 * draw(r) - 0.1 * x) : 0.0) + (big ? dv : 0);
            cell[m][3] = p0 * (1 + amp * (0.1 * draw(r) + 0.1 * x)) * (big ? jp : 1);
            lam = std::max(lam, std::fabs(cell[m][1]) + std::sqrt(g * cell[m][3] / cell[m][0]));
        }
        lam *= 1 + 0.5 * std::fabs(draw(r));
        for (int m = 0; m < 6; ++m) {
            const double *c = cell[m], E = c[3] / (g - 1) + 0.5 * c[0] * (c[1] * c[1] + c[2] * c[2]);
            const double U[4] = {c[0], c[0] * c[1], c[0] * c[2], E};
            const double f[4] = {U[1], U[1] * c[1] + c[3], U[1] * c[2], c[1] * (E + c[3])};
            for (int k = 0; k < 4; ++k) { F[0][m][k] = 0.5 * (f[k] + lam * U[k]); F[1][m][k] = 0.5 * (f[k] - lam * U[k]); }
        }
        EigFast e;
        const double *L = cell[2], *R = cell[3];
        auto H = [&](const double* c) { return g / (g - 1) * c[3] / c[0] + 0.5 * (c[1] * c[1] + c[2] * c[2]); };
        roe_eig_fast<0>(g - 1, std::sqrt(L[0]), std::sqrt(R[0]), L[1], R[1], L[2], R[2], H(L), H(R), e);
        ld cq[4] = {0, 0, 0, 0}, zq[4] = {0, 0, 0, 0};
        double c6[4] = {0, 0, 0, 0}, w6[4] = {0, 0, 0, 0}, centre[4] = {0, 0, 0, 0}, size[4] = {0, 0, 0, 0};
        for (int s = 0; s < 2; ++s) {
            double d[4][4], gk[4][4], lc[4], cs[4];
            for (int m = 0; m < 4; ++m)
                for (int c = 0; c < 4; ++c) d[m][c] = F[s][s ? 5 - m : m][c] - F[s][s ? 4 - m : m + 1][c];
            auto dF = [&](int m, double f[4]) { for (int c = 0; c < 4; ++c) f[c] = d[m][c]; };
            const double* C = F[s][s ? 3 : 2];
            const unsigned redo = char_fields<0>(e, dF, C[0], C[2], cs);
            for (int k = 0; k < 4; ++k) c6[k] += redo >> k & 1 ? char_field_fp64<0>(e, dF, k) : cs[k];
            for (int m = 0; m < 4; ++m) {
                double l[4];
                project_fast<0>(e, d[m], l);
                for (int k = 0; k < 4; ++k) gk[k][m] = l[k];
            }
            project_fast<0>(e, C, lc);
            for (int k = 0; k < 4; ++k) {
                w6[k] += 6 * (lc[k] + correction_fp64<true>(gk[k]));
                // the exact differences' exact fields
                ld gq[4];
                for (int m = 0; m < 4; ++m) {
                    const double *a = F[s][s ? 5 - m : m], *b = F[s][s ? 4 - m : m + 1];
                    const ld f0 = (ld)a[0] - b[0], w = ((ld)a[1] - b[1]) - e.un0 * f0, qt = ((ld)a[2] - b[2]) - e.ut0 * f0;
                    const ld z = ((ld)a[3] - b[3]) - e.uu0 * f0 - e.un0 * w - e.ut0 * qt;
                    gq[m] = k == 0 ? e.ih * z - e.ia5 * w : k == 1 ? f0 - e.ihh * z : k == 2 ? qt : e.ih * z + e.ia5 * w;
                }
                cq[k] += correction_of<true>(gq);
                zq[k] += C[k];
                centre[k] += C[k];
                size[k] = std::max(size[k], std::fabs(C[k]));
            }
        }
        const ld s = cq[0] + cq[1] + cq[3], dd = cq[3] - cq[0];
        const ld want[4] = {zq[0] + s, zq[1] + e.un0 * s + e.a0 * dd, zq[2] + e.ut0 * s + cq[2],
                            zq[3] + e.h0 * (cq[0] + cq[3]) + e.a0 * e.un0 * dd + e.uu0 * cq[1] + e.ut0 * cq[2]};
        double h[4], h64[4];
        const double zero[4] = {0, 0, 0, 0};
        back_project_fast<0>(e, c6, centre, h);
        back_project_fast<0>(e, w6, zero, h64);
        for (int k = 0; k < 4; ++k) {
            // (a transverse flux beside a larger normal one is not held to its own smallness)
            const double sz = std::max(size[k] + (double)fabsl(want[k]), k == 2 ? 1e-3 * size[1] : 0.0);
            err[k].add((double)fabsl(h[k] - want[k]) / sz, (double)fabsl(h64[k] - want[k]) / sz);
        }
    }
    for (int k = 0; k < 4; ++k) { printf("fields %g %d ", ratio, k); err[k].print(); }
}

// AdaWENO's smooth branch: a component beside a jump of 10^decades times its level, reconstructed with
// the weights of a surrogate that is smooth for the given delta, relative to the centre values and
// corrections; FP64's from the same weights. few: surrogates with a jump among them (delta 0: always smooth)
void borrowed(double delta, int decades) {
    std::mt19937_64 r((unsigned)(900 + 10 * decades + (int)(100 * delta)));
    const double k = std::sqrt(delta / (1.0 - delta)), theta_c = k / (1.0 + k);
    Errors err;
    for (int t = 0; t < 200000 && err.n < 20000; ++t) {
        const double level = std::pow(10.0, 3 * draw(r)), amp = std::pow(10.0, -2 + 2 * draw(r)), half = r() & 1 ? 0.0 : 1.0;
        double gs[2][4], g[2][4];
        ld c[2];
        double c64[2];
        fx::u64 f0[2], f2[2];
        bool ok = true, rough = false;
        for (int s = 0; s < 2; ++s) {
            const double a = draw(r), b = 0.3 * draw(r), js = std::pow(10.0, 3 * draw(r)) * draw(r);
            const int j = (int)(r() % 4), i = (int)(r() % 4);
            for (int m = 0; m < 4; ++m) {
                gs[s][m] = 0.1 * (a + b * (m - 1.5)) + (delta == 0.0 && m == i && r() & 1 ? js : 0.0);
                g[s][m] = level * (amp * (a + draw(r) * 0.3) + (m == j ? std::pow(10.0, decades) * (1 + 0.5 * draw(r)) : 0.0));
            }
            ok = fx::surrogate(gs[s], theta_c, f0[s], f2[s]) && ok;
            rough = fx::rough(gs[s]) || rough;
        }
        if (!ok) continue;
        const double lp = half * level * (1 + 0.3 * draw(r)), lm = -0.7 * half * level * (1 + 0.3 * draw(r));
        for (int s = 0; s < 2; ++s) {
            ld w[3];
            double u[3];
            weights_of(gs[s], w);
            c[s] = (w[0] * (2 * (ld)g[s][0] - 5 * (ld)g[s][1]) + w[1] * (-(ld)g[s][1] - 2 * (ld)g[s][2]) +
                    w[2] * ((ld)g[s][3] - 4 * (ld)g[s][2])) / 6;
            weights_fp64<true>(gs[s], u);
            c64[s] = correction_by_fp64(g[s], u);
        }
        const fx::u32 top = fx::umax(fx::exponent_of(g[0]), fx::exponent_of(g[1])), eh = fx::umax(top, fx::kExpMin);
        const double c6 = fx::to_double(fx::correction6_by(g[0], eh, f0[0], f2[0]) + fx::correction6_by(g[1], eh, f0[1], f2[1]), eh, top);
        double h = fx::about(lp, lm, c6);
        if (fx::far_weights(theta_c) && (rough || fx::coarse_by(top, lp, lm, c6))) h = about_fp64(lp, lm, c64[0] + c64[1]);
        const ld want = c[0] + c[1] + lp + lm;
        const double size = std::max(std::fabs(lp), std::fabs(lm)) + (double)(fabsl(c[0]) + fabsl(c[1]));
        err.add((double)fabsl(h - want) / size, (double)fabsl((lp + c64[0]) + (lm + c64[1]) - want) / size);
    }
    printf("borrowed %g %d ", delta, decades);
    err.print();
}

// the update's flux change with the directions' fluxes and differences orders apart, relative to the larger
// product; FP64's beside it. kind 0: both; 1: large eta fluxes that cancel; 2: large xi fluxes that
// cancel; 3: dt/dx and dt/dy up to 1e9 apart
void change(int kind) {
    std::mt19937_64 r(131 + kind);
    Errors err;
    int odd = 0;
    for (int t = 0; t < 50000; ++t) {
        double h[4];
        for (int d = 0; d < 2; ++d) {
            const double size = std::pow(10.0, 12 * draw(r)), small = std::pow(10.0, -12 * std::fabs(draw(r))), base = draw(r);
            for (int k = 0; k < 2; ++k) h[2 * d + k] = size * (base + small * draw(r));
        }
        if (kind == 1) { h[2] = h[3] = 1e3 * std::fabs(h[2]); }
        if (kind == 2) { h[0] = h[1] = 1e3 * std::fabs(h[0]); }
        const double dtdx = std::pow(10.0, -3 + 3 * draw(r)), dtdy = dtdx * std::pow(10.0, kind == 3 ? 9 * draw(r) : draw(r));
        const fx::Rates q = fx::rates_of(dtdx, dtdy);
        const ld x = (ld)dtdx * ((ld)h[1] - h[0]), y = (ld)dtdy * ((ld)h[3] - h[2]);
        const double size = (double)std::max(fabsl(x), fabsl(y)), got = fx::flux_change(h[0], h[1], h[2], h[3], q);
        odd += fx::flux_change(h[1], h[0], h[3], h[2], q) != -got || fx::flux_change(-h[0], -h[1], -h[2], -h[3], q) != -got;
        if (size == 0.0) continue;
        err.add((double)fabsl(got - (x + y)) / size, (double)fabsl(fma(dtdx, h[1] - h[0], dtdy * (h[3] - h[2])) - (x + y)) / size);
    }
    // the ends of the range
    const double inf = std::numeric_limits<double>::infinity();
    odd += fx::flux_change(-4e307, 4e307, 0.0, 0.0, fx::rates_of(1.0, 1.0)) != 8e307;
    odd += fx::flux_change(-1e200, 1e200, 0.0, 0.0, fx::rates_of(1e200, 1.0)) != inf;
    odd += fx::flux_change(1e200, -1e200, 0.0, 0.0, fx::rates_of(1e200, 1.0)) != -inf;
    odd += fx::flux_change(1.0, 2.0, 5.0, 5.0, fx::rates_of(0x1p-600, 1.0)) != 0x1p-600;
    printf("change %d %d ", kind, odd);
    err.print();
}

// dW/dlf[m] from the first differences, written out (the five sum to one)
template <bool Z> void gradient_of(const double g[4], ld G[5]) {
    const ld ss = (double)1.0e-6f, cs[3] = {0.1L, 0.6L, 0.3L};
    const ld A[3] = {(ld)g[0] - g[1], (ld)g[1] - g[2], (ld)g[2] - g[3]};
    const ld B[3] = {g[0] - 3 * (ld)g[1], (ld)g[1] + g[2], 3 * (ld)g[2] - g[3]};
    const ld q[3] = {(2 * (ld)g[0] - 5 * (ld)g[1]) / 6, (-(ld)g[1] - 2 * (ld)g[2]) / 6, ((ld)g[3] - 4 * (ld)g[2]) / 6};
    const ld a[3][5] = {{1 / 3.L, -7 / 6.L, 11 / 6.L, 0, 0}, {0, -1 / 6.L, 5 / 6.L, 1 / 3.L, 0}, {0, 0, 1 / 3.L, 5 / 6.L, -1 / 6.L}};
    const ld dA[3][5] = {{1, -2, 1, 0, 0}, {0, 1, -2, 1, 0}, {0, 0, 1, -2, 1}};
    const ld dB[3][5] = {{1, -4, 3, 0, 0}, {0, 1, 0, -1, 0}, {0, 0, 3, -4, 1}};
    ld be[3], d[3], al[3], db[3], S = 0, W = 0, st = 0;
    for (int k = 0; k < 3; ++k) { be[k] = 13 * A[k] * A[k] / 12 + B[k] * B[k] / 4; d[k] = ss + be[k]; }
    const ld tau = fabsl(be[2] - be[0]);
    for (int k = 0; k < 3; ++k) { al[k] = Z ? cs[k] * (1 + tau * tau / (d[k] * d[k])) : cs[k] / (d[k] * d[k]); S += al[k]; }
    for (int k = 0; k < 3; ++k) W += al[k] * q[k] / S;
    for (int k = 0; k < 3; ++k) {
        const ld e = (q[k] - W) / S;
        db[k] = Z ? -2 * e * cs[k] * tau * tau / (d[k] * d[k] * d[k]) : -2 * e * al[k] / d[k];
        if (Z) st += 2 * e * cs[k] * tau / (d[k] * d[k]);
    }
    if (be[2] >= be[0]) { db[2] += st; db[0] -= st; } else { db[2] -= st; db[0] += st; }
    for (int m = 0; m < 5; ++m) {
        G[m] = 0;
        for (int k = 0; k < 3; ++k) G[m] += al[k] / S * a[k][m] + db[k] * (13 * A[k] * dA[k][m] / 6 + B[k] * dB[k][m] / 2);
    }
}
// the taped gradient of a stencil as the component-wise sweeps form it, on the exponent it shares with its
// partner, beside weno_grad's. kind 0: both smooth; 1: a jump of 10^decades times the level in this one;
// 2: in the partner; 3: both rough
template <bool Z> void taped(int kind, int decades) {
    std::mt19937_64 r(171 + 10 * kind + decades);
    Errors err;
    for (int t = 0; t < 20000; ++t) {
        const double level = std::pow(10.0, 2 * draw(r)), amp = level * std::pow(10.0, -1.5 + 1.5 * draw(r));
        double g[2][4], G[5], G64[5];
        for (int s = 0; s < 2; ++s) {
            const double a = draw(r), b = 0.3 * draw(r), c = 0.1 * draw(r), jump = level * std::pow(10.0, decades) * (1 + 0.5 * draw(r));
            const int j = (int)(r() % 4);
            for (int m = 0; m < 4; ++m)
                g[s][m] = (kind == 3 ? level * draw(r) : amp * (a + b * (m - 1.5) + c * (m - 1.5) * (m - 1.5))) +
                          (kind == 1 + s && m == j ? jump : 0.0);
        }
        fx::u32 top = 0;
        const fx::u32 e0 = fx::scale_of(g[0], top), eh = fx::umax(e0, fx::scale_of(g[1], top));
        fx::Gradient q;
        fx::correction6_taped<Z>(g[0], eh, q);
        weno_grad_of<Z>(g[0], G64);
        if (fx::rough<Z>(g[0], eh)) weno_grad_of<Z>(g[0], G);
        else fx::gradient_out(q, top, G);
        ld want[5];
        gradient_of<Z>(g[0], want);
        double e = 0, e64 = 0;
        for (int m = 0; m < 5; ++m) {
            e = std::max(e, (double)fabsl(G[m] - want[m]));
            e64 = std::max(e64, (double)fabsl(G64[m] - want[m]));
        }
        err.add(e, e64);
    }
    printf("taped %d %d %d ", (int)Z, kind, decades);
    err.print();
}

// the Roe means of two cells whose densities are up to 10^decades apart, the enthalpies the other way
// round: relative to the weighted mean of the magnitudes, in units of 2^-53
void means(int decades) {
    std::mt19937_64 r(211 + decades);
    double worst = 0;
    for (int t = 0; t < 20000; ++t) {
        const double f = std::pow(10.0, decades * draw(r)), sl = std::sqrt(1 + std::fabs(draw(r))), sr = std::sqrt(f * (1 + std::fabs(draw(r))));
        const double ul = draw(r) * std::pow(10.0, 3 * draw(r)), ur = draw(r) * std::pow(10.0, 3 * draw(r));
        const double hl = 20 + 1e6 * f, hr = 20 + 1e6;  // (above the velocities' squares over two)
        EigFast e;
        roe_eig_fast<0>(0.4, sl, sr, ul, ur, 0.5 * ur, 0.5 * ul, hl + ul * ul + ur * ur, hr + ul * ul + ur * ur, e);
        const ld HL = hl + ul * ul + ur * ur, HR = hr + ul * ul + ur * ur;
        auto mean = [&](ld l, ld x) { return (sl * l + sr * x) / ((ld)sl + sr); };
        worst = std::max(worst, (double)(fabsl(e.un0 - mean(ul, ur)) / mean(std::fabs(ul), std::fabs(ur)) / 0x1p-53L));
        worst = std::max(worst, (double)(fabsl(e.ut0 - mean(0.5 * ur, 0.5 * ul)) / mean(0.5 * std::fabs(ur), 0.5 * std::fabs(ul)) / 0x1p-53L));
        worst = std::max(worst, (double)(fabsl(e.h0 - mean((double)HL, (double)HR)) / mean((double)HL, (double)HR) / 0x1p-53L));
    }
    printf("means %d %.17g\n", decades, worst);
}

int main() {
    for (int decades : {0, 2, 4, 8}) means(decades);
    for (int kind = 0; kind < 4; ++kind)
        for (int decades : {-2, -1, 0, 1, 4}) { taped<false>(kind, decades); taped<true>(kind, decades); }
    for (int kind = 0; kind < 4; ++kind) change(kind);
    for (double delta : {0.0, 0.001, 0.01, 0.5, 0.9})
        for (int decades : {-3, 0, 2, 6, 10}) borrowed(delta, decades);
    for (double ratio : {0.1, 2.0, 8.0, 100.0, 1e4, 1e8}) fields(ratio);
    for (int kind = 0; kind < 2; ++kind)
        for (int decades : {-3, 0, 1, 2, 4, 6, 10, 14}) { sided<false>(kind, decades); sided<true>(kind, decades); }
    value_forms<false>();
    value_forms<true>();
    between<false>();
    between<true>();
}
