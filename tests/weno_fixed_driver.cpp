// The integer reconstructions of csrc/weno_fixed.cuh on the host, beside the FP64 form of
// csrc/weno_fast.cuh, both against long double. Prints one line a check; see test_weno_fixed.py.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <limits>
#include <random>

#include "../2dense_gb300/csrc/weno_fixed.cuh"

#define __device__
#define __forceinline__ inline
namespace f64 {
namespace fx {  // the FP64 form with an IEEE reciprocal
static double rcp(double d) { return 1.0 / d; }
}
#include "../2dense_gb300/csrc/weno_fast.cuh"
template <bool Z> double recon(double lf2, const double g[4]) {
    double d0, d1, d2, B[3];
    betas_g(g, d0, d1, d2, B);
    WenoTerms t;
    weno_terms<Z>(g, d0, d1, d2, t);
    return fma(weno_num(t), fx::rcp(t.N), lf2);
}
}  // namespace f64

typedef long double ld;

// the reconstruction as weno_mod.f90 writes it
template <bool Z> ld exact(const double f[5]) {
    const ld a = f[0], b = f[1], c = f[2], d = f[3], e = f[4], ss = (double)1.0e-6f;
    const ld is[3] = {13 * (a - 2 * b + c) * (a - 2 * b + c) / 12 + (a - 4 * b + 3 * c) * (a - 4 * b + 3 * c) / 4,
                      13 * (b - 2 * c + d) * (b - 2 * c + d) / 12 + (b - d) * (b - d) / 4,
                      13 * (c - 2 * d + e) * (c - 2 * d + e) / 12 + (3 * c - 4 * d + e) * (3 * c - 4 * d + e) / 4};
    const ld q[3] = {(2 * a - 7 * b + 11 * c) / 6, (-b + 5 * c + 2 * d) / 6, (2 * c + 5 * d - e) / 6};
    const ld cs[3] = {1, 6, 3}, tau = is[2] - is[0];
    ld num = 0, den = 0;
    for (int k = 0; k < 3; ++k) {
        const ld s = (ss + is[k]) * (ss + is[k]), w = Z ? cs[k] * (1 + tau * tau / s) : cs[k] / s;
        num += w * q[k];
        den += w;
    }
    return num / den;
}

struct Stencils {
    double fp[5], fm[5], gp[4], gm[4];
    double rm[4];  // the second's differences with the opposite sign, as fx::pair takes them
    void differences() {
        for (int m = 0; m < 4; ++m) { gp[m] = fp[m] - fp[m + 1]; gm[m] = fm[m] - fm[m + 1]; rm[m] = -gm[m]; }
    }
    double size() const {
        double s = 0;
        for (int m = 0; m < 5; ++m) s = std::max(s, std::max(std::fabs(fp[m]), std::fabs(fm[m])));
        return s;
    }
};

// kind 0 smooth, 1 one jump of 0.03 to 30 times the level, 2 rough, 3 a flat side beside a jump of up
// to 3e4 times the level, 4 the same beside 1e12 times the level
Stencils draw(std::mt19937_64& r, int kind) {
    std::uniform_real_distribution<double> u(-1, 1);
    Stencils s;
    const double level = std::pow(10.0, 2 * u(r)), amp = level * std::pow(10.0, -4 + 4 * u(r));
    for (double* f : {s.fp, s.fm}) {
        const double a = u(r), b = u(r), c = u(r), jump = level * std::pow(10.0, 1.5 * u(r));
        const int j = 1 + (int)(r() % 4);
        for (int m = 0; m < 5; ++m) {
            const double x = m - 2.0;
            f[m] = level * (f == s.fp ? 1.0 : -0.7) + amp * (a * x + 0.3 * b * x * x + 0.1 * c * x * x * x);
            if (kind == 1 && m >= j) f[m] += jump;
            if (kind == 2) f[m] += level * u(r);
            if (kind >= 3) f[m] = m < j ? level : f[m] + jump * (kind == 3 ? 1e3 * u(r) : 1e12);
        }
    }
    s.differences();
    return s;
}

template <bool Z> void accuracy(int kind) {
    std::mt19937_64 r(11 + kind);
    double worst = 0, worst64 = 0, sum = 0, sum64 = 0;
    const int n = 100000;
    for (int t = 0; t < n; ++t) {
        const Stencils s = draw(r, kind);
        const ld ref = exact<Z>(s.fp) + exact<Z>(s.fm);
        const double h = dense::fx::pair<Z>(s.fp[2], s.gp, s.fm[2], s.rm);
        const double h64 = f64::recon<Z>(s.fp[2], s.gp) + f64::recon<Z>(s.fm[2], s.gm);
        const double e = (double)fabsl(h - ref) / s.size(), e64 = (double)fabsl(h64 - ref) / s.size();
        worst = std::max(worst, e); worst64 = std::max(worst64, e64);
        sum += e * e; sum64 += e64 * e64;
    }
    printf("accuracy %d %d %.17g %.17g %.17g %.17g\n", (int)Z, kind, worst, std::sqrt(sum / n), worst64, std::sqrt(sum64 / n));
}

template <bool Z> void forms() {
    std::mt19937_64 r(5);
    int odd = 0, swap = 0, flat = 0, bad = 0, n = 0;
    double scale_err = 0;
    for (int t = 0; t < 20000; ++t) {
        Stencils s = draw(r, t % 5);
        const double cp = s.fp[2], cm = s.fm[2], h = dense::fx::pair<Z>(cp, s.gp, cm, s.rm);
        double np[4], nm[4];
        for (int m = 0; m < 4; ++m) { np[m] = -s.gp[m]; nm[m] = -s.rm[m]; }
        odd += dense::fx::pair<Z>(-cp, np, -cm, nm) != -h;
        swap += dense::fx::pair<Z>(cm, s.gm, cp, np) != h;
        const double zero[4] = {0, -0.0, 0, 0};
        flat += dense::fx::pair<Z>(cp, zero, cm, zero) != cp + cm;
        for (double x : {std::numeric_limits<double>::quiet_NaN(), std::numeric_limits<double>::infinity(),
                         -std::numeric_limits<double>::infinity()}) {
            Stencils b = s;
            (t & 1 ? b.gp : b.rm)[(t >> 1) & 3] = x;
            bad += !std::isnan(dense::fx::pair<Z>(cp, b.gp, cm, b.rm));
        }
        // the same differences at any scale: far above ss the weights do not depend on it, far below
        // they are the linear ones
        if (t % 5 == 0) {
            const double p = std::ldexp(1.0, (int)(r() % 900) - 700);
            Stencils b;
            for (int m = 0; m < 5; ++m) { b.fp[m] = s.fp[m] * p; b.fm[m] = s.fm[m] * p; }
            if (b.size() < 1e90 && b.size() > 1e-180) {
                b.differences();
                double g = 0;
                for (int m = 0; m < 4; ++m) g = std::max(g, std::max(std::fabs(b.gp[m]), std::fabs(b.gm[m])));
                const ld ref = (exact<Z>(b.fp) - b.fp[2]) + (exact<Z>(b.fm) - b.fm[2]);
                // the differences themselves carry the rounding of their level
                const double tol = 64 * (std::ldexp(b.size(), -53) + std::ldexp(g, -53));
                scale_err = std::max(scale_err, (double)(fabsl(dense::fx::pair<Z>(0.0, b.gp, 0.0, b.rm) - ref) / tol));
                ++n;
            }
        }
    }
    printf("forms %d %d %d %d %d %d %.17g\n", (int)Z, odd, swap, flat, bad, n, scale_err);
}

// AdaWENO's surrogate: its switch against theta > delta, and another stencil reconstructed with its
// weights against long double
void adaptive() {
    std::mt19937_64 r(9);
    std::uniform_real_distribution<double> u(0, 1);
    int wrong = 0, near = 0, ends = 0, smooth = 0, nans = 0;
    double worst = 0;
    const int n = 50000;
    for (int t = 0; t < n; ++t) {
        const Stencils s = draw(r, t % 4);
        const double delta = t % 3 ? u(r) : 0.5, k = std::sqrt(delta / (1.0 - delta)), theta_c = k / (1.0 + k);
        const ld a = s.fp[0], b = s.fp[1], c = s.fp[2], d = s.fp[3], e = s.fp[4], ss = (double)1.0e-6f;
        const ld is[3] = {13 * (a - 2 * b + c) * (a - 2 * b + c) / 12 + (a - 4 * b + 3 * c) * (a - 4 * b + 3 * c) / 4,
                          13 * (b - 2 * c + d) * (b - 2 * c + d) / 12 + (b - d) * (b - d) / 4,
                          13 * (c - 2 * d + e) * (c - 2 * d + e) / 12 + (3 * c - 4 * d + e) * (3 * c - 4 * d + e) / 4};
        ld al[3], sum = 0;
        const ld tau = is[2] - is[0], cs[3] = {0.1L, 0.6L, 0.3L};
        for (int i = 0; i < 3; ++i) { al[i] = cs[i] * (1 + tau * tau / ((ss + is[i]) * (ss + is[i]))); sum += al[i]; }
        const ld theta = 1 / (1 + (sum - 1) * (sum - 1));
        dense::fx::u64 f0, f2;
        const bool got = dense::fx::surrogate(s.gp, theta_c, f0, f2);
        smooth += got;
        // the surrogate's differences carry the rounding of its values: 2^-53 of them, amplified by the
        // indicators' sensitivity to the smallest difference (or sqrt(ss))
        ld small = std::sqrt((double)ss);
        ld sens = 64 * s.size() * 0x1p-53L;
        for (int m = 0; m < 4; ++m) if (s.gp[m] != 0) small = std::min(small, (ld)std::fabs(s.gp[m]));
        if (fabsl(theta - delta) <= 1e-9L + sens / small) ++near;
        else wrong += got != (theta > delta);
        ends += !dense::fx::surrogate(s.gp, 0.0, f0, f2) || dense::fx::surrogate(s.gp, 1.0, f0, f2);
        double bad[4] = {s.gp[0], s.gp[1], s.gp[2], s.gp[3]};
        bad[t & 3] = t & 4 ? std::numeric_limits<double>::quiet_NaN() : std::numeric_limits<double>::infinity();
        dense::fx::u64 x, y;
        nans += dense::fx::surrogate(bad, 0.0, x, y);
        // the other stencil (s.fm) with these weights: the weights are taken as they are (an error of
        // theirs counts with the third differences), the arithmetic is compared
        const ld w0 = ldexpl((ld)f0, -63), w2 = ldexpl((ld)f2, -62), w1 = 1 - w0 - w2;
        const ld q0 = (2 * (ld)s.fm[0] - 7 * (ld)s.fm[1] + 11 * (ld)s.fm[2]) / 6, q1 = (-(ld)s.fm[1] + 5 * (ld)s.fm[2] + 2 * (ld)s.fm[3]) / 6,
                 q2 = (2 * (ld)s.fm[2] + 5 * (ld)s.fm[3] - (ld)s.fm[4]) / 6;
        const dense::fx::u32 eh = dense::fx::umax(dense::fx::exponent_of(s.gm), dense::fx::kExpMin);
        const double h = dense::fx::about(s.fm[2], 0.0, dense::fx::to_double(dense::fx::correction6_by(s.gm, eh, f0, f2), eh, eh));
        worst = std::max(worst, (double)(fabsl(h - (w0 * q0 + w1 * q1 + w2 * q2)) / s.size()));
        // and the weights
        worst = std::max(worst, (double)(fabsl(w0 - al[0] / sum) > 1e-9L + sens / small));
    }
    printf("adaptive %d %d %d %d %d %d %.17g\n", n, wrong, near, ends, nans, smooth, worst);
}

// rcp, rsqrt and sqrt_normal: the largest error in ulp over mantissas and exponents, and the arguments
// outside their range
void roots() {
    std::mt19937_64 r(21);
    double worst[3] = {0, 0, 0};
    for (int t = 0; t < 1000000; ++t) {
        double x;
        if (t < 1000) x = 1.0 + t * 0x1p-52;
        else if (t < 2000) x = 2.0 - (t - 999) * 0x1p-52;
        else if (t < 3000) x = 4.0 - (t - 1999) * 0x1p-51;
        else x = std::ldexp(1.0 + (double)(r() >> 12) * 0x1p-52, (int)(r() % 2000) - 1000);
        const ld want[3] = {1.0L / x, 1.0L / sqrtl(x), sqrtl(x)};
        const double got[3] = {dense::fx::rcp(x), dense::fx::rsqrt(x), dense::fx::sqrt_normal(x)};
        for (int k = 0; k < 3; ++k) {
            const double w = (double)want[k], ulp = std::nextafter(w, 1e308) - w;
            worst[k] = std::max(worst[k], (double)(fabsl(got[k] - want[k]) / ulp));
        }
    }
    int bad = dense::fx::rcp(-8.0) != -0.125;
    const double inf = std::numeric_limits<double>::infinity(), nan = std::numeric_limits<double>::quiet_NaN();
    for (double x : {0.0, -0.0, inf, -inf, nan, 1e-310}) bad += !std::isnan(dense::fx::rcp(x));
    for (double x : {0.0, -1.0, inf, nan, 1e-310})
        bad += !std::isnan(dense::fx::rsqrt(x)) + !std::isnan(dense::fx::sqrt_normal(x));
    printf("roots %.17g %.17g %.17g %d\n", worst[0], worst[1], worst[2], bad);
}

// the update's flux change against long double, in units of 2^-53 of the largest flux times the larger
// rate; its oddness; what is not finite
void change() {
    std::mt19937_64 r(31);
    std::uniform_real_distribution<double> u(-1, 1);
    double worst = 0;
    int odd = 0, bad = 0;
    const double inf = std::numeric_limits<double>::infinity(), nan = std::numeric_limits<double>::quiet_NaN();
    for (int t = 0; t < 200000; ++t) {
        const double size = std::pow(10.0, 6 * u(r)), small = std::pow(10.0, -8 * std::fabs(u(r)));
        double h[4];
        const double bx = u(r), by = u(r);
        for (int k = 0; k < 4; ++k) h[k] = size * ((k < 2 ? bx : by) + small * u(r));
        const double dtdx = std::pow(10.0, -2 + 2 * u(r)), dtdy = dtdx * std::pow(10.0, 3 * u(r)), sg = t & 1 ? -1.0 : 1.0;
        const dense::fx::Rates q = dense::fx::rates_of(sg * dtdx, sg * dtdy);
        const ld want = (ld)(sg * dtdx) * ((ld)h[1] - h[0]) + (ld)(sg * dtdy) * ((ld)h[3] - h[2]);
        const double got = dense::fx::flux_change(h[0], h[1], h[2], h[3], q);
        double big = 0;
        for (double x : h) big = std::max(big, std::fabs(x));
        worst = std::max(worst, (double)(fabsl(got - want) / (0x1p-53L * (big * std::max(dtdx, dtdy) + fabsl(want)))));
        odd += dense::fx::flux_change(-h[0], -h[1], -h[2], -h[3], q) != -got;
        odd += dense::fx::flux_change(h[1], h[0], h[3], h[2], q) != -got;
        const double x = t % 3 == 0 ? nan : t % 3 == 1 ? inf : -inf, keep = h[t & 3];
        h[t & 3] = x;
        bad += !std::isnan(dense::fx::flux_change(h[0], h[1], h[2], h[3], q));
        h[t & 3] = keep;
        bad += !std::isnan(dense::fx::flux_change(h[0], h[1], h[2], h[3], dense::fx::rates_of(x, dtdy)));
        bad += !std::isnan(dense::fx::flux_change(h[0], h[1], h[2], h[3], dense::fx::rates_of(dtdx, x)));
        bad += dense::fx::flux_change(h[0], h[1], h[2], h[3], dense::fx::rates_of(0.0, 0.0)) != 0.0;
        bad += dense::fx::flux_change(h[0], h[0], h[2], h[2], q) != 0.0;
    }
    printf("change %.17g %d %d\n", worst, odd, bad);
}

// to_double against the host's own rounding of an integer: every width, and the values that round up
// to the next power of two
void conversion() {
    std::mt19937_64 r(41);
    int bad = 0;
    for (int k = 1; k < 63; ++k)
        for (int t = 0; t < 4000; ++t) {
            dense::fx::i64 c = (dense::fx::i64)(t < 2100 ? (1ull << k) - (unsigned long long)t : r() >> (64 - k));
            if (c <= 0) continue;
            if (t & 1) c = -c;
            const double want = std::ldexp((double)c, 3), got = dense::fx::to_double(c, 1083u << 20, 0);
            // halves go away from zero here, to even there
            if (got != want && std::fabs((double)((ld)got / 8 - c)) > std::fabs((double)((ld)want / 8 - c))) ++bad;
        }
    printf("conversion %d\n", bad);
}

// the gradient dW/dlf[m] of the reconstruction, written out
template <bool Z> void exact_gradient(const double f[5], ld G[5]) {
    const ld ss = (double)1.0e-6f, cs[3] = {0.1L, 0.6L, 0.3L};
    ld g[4], be[3], d[3], al[3], db[3], S = 0, W = 0, st = 0;
    for (int m = 0; m < 4; ++m) g[m] = (ld)f[m] - f[m + 1];
    const ld A[3] = {g[0] - g[1], g[1] - g[2], g[2] - g[3]}, B[3] = {g[0] - 3 * g[1], g[1] + g[2], 3 * g[2] - g[3]};
    const ld q[3] = {(2 * g[0] - 5 * g[1]) / 6, (-g[1] - 2 * g[2]) / 6, (g[3] - 4 * g[2]) / 6};  // about lf2
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
    const ld a[3][5] = {{1 / 3.L, -7 / 6.L, 11 / 6.L, 0, 0}, {0, -1 / 6.L, 5 / 6.L, 1 / 3.L, 0}, {0, 0, 1 / 3.L, 5 / 6.L, -1 / 6.L}};
    const ld dA[3][5] = {{1, -2, 1, 0, 0}, {0, 1, -2, 1, 0}, {0, 0, 1, -2, 1}};
    const ld dB[3][5] = {{1, -4, 3, 0, 0}, {0, 1, 0, -1, 0}, {0, 0, 3, -4, 1}};
    for (int m = 0; m < 5; ++m) {
        G[m] = 0;
        for (int k = 0; k < 3; ++k) G[m] += al[k] / S * a[k][m] + db[k] * (13 * A[k] * dA[k][m] / 6 + B[k] * dB[k][m] / 2);
    }
}
// the taped reconstruction: its gradient (weno_grad's where the stencil is rough) and weno_grad's everywhere
// against long double, its value against the plain one, and a change of sign of the differences
template <bool Z> void gradient(int kind) {
    std::mt19937_64 r(61 + kind);
    double sum = 0, sum64 = 0, worst = 0;
    int bits = 0, even = 0;
    const int n = 50000;
    for (int t = 0; t < n; ++t) {
        const Stencils s = draw(r, kind);
        ld G[5];
        exact_gradient<Z>(s.fp, G);
        double g[5], g64[5], ne[4], ge[5];
        dense::fx::u32 top = 0;
        const dense::fx::u32 eh = dense::fx::scale_of(s.gp, top);
        dense::fx::Gradient q, qe;
        bits += dense::fx::correction6_taped<Z>(s.gp, eh, q) != dense::fx::correction6<Z>(s.gp, eh);
        for (int m = 0; m < 4; ++m) ne[m] = -s.gp[m];
        dense::fx::correction6_taped<Z>(ne, eh, qe);
        for (int m = 0; m < 5; ++m) even += qe.g[m] != q.g[m];
        f64::weno_grad_of<Z>(s.gp, g64);
        dense::fx::gradient_out(q, top, g);
        dense::fx::gradient_out(q, dense::fx::kExpMax, ge);
        even += !std::isnan(ge[t % 5]);
        double e = 0, e64 = 0;
        for (int m = 0; m < 5; ++m) {
            if (dense::fx::rough(s.gp)) g[m] = g64[m];
            e = std::max(e, (double)fabsl(g[m] - G[m]));
            e64 = std::max(e64, (double)fabsl(g64[m] - G[m]));
        }
        sum += e * e; sum64 += e64 * e64; worst = std::max(worst, e);
    }
    printf("gradient %d %d %.17g %.17g %.17g %d %d\n", (int)Z, kind, std::sqrt(sum / n), std::sqrt(sum64 / n), worst, bits, even);
}

int main() {
    conversion();
    roots();
    change();
    std::mt19937_64 r(3);
    double worst = 0;
    for (int t = 0; t < 2000000; ++t) {
        dense::fx::u64 n = (r() >> 2) | (1ull << 62);
        if (t < 64) n = (1ull << 62) + (dense::fx::u64)t;
        else if (t < 128) n = (1ull << 63) - 1 - (dense::fx::u64)t;
        const ld e = (ld)dense::fx::reciprocal(n) * (ld)n / ((ld)(1ull << 62) * (ld)(1ull << 63)) - 1;
        worst = std::max(worst, (double)fabsl(e));
    }
    printf("reciprocal %.17g\n", worst);
    for (int k = 0; k < 5; ++k) { accuracy<false>(k); accuracy<true>(k); }
    forms<false>();
    forms<true>();
    adaptive();
    for (int k = 0; k < 5; ++k) { gradient<false>(k); gradient<true>(k); }
}
