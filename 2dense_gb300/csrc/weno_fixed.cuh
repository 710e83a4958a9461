// weno_fixed.cuh -- WENO-JS5 / WENO-Z5 reconstructions on the integer pipes, for the fast sweeps.
//
// GB300 issues an FP64 instruction of a warp every 16 cycles of an SM, and in that time up to 64
// others: measured per warp and SM, DFMA 16.9 cycles, against 0.6 for a 32-bit IMAD or LOP, 1.0 for a
// 32x32+64-bit IMAD.WIDE, 0.6 for a 64-bit shift and 4.5 for the upper half of a 64x64-bit
// product. A reconstruction in FP64 is about 34 instructions, 556 (JS) to 668 (Z) cycles with the
// integer pipes idle; the same value in 64-bit integers takes 172 and 205, and leaves the FP64 pipe
// to the split fluxes of other warps. The component-wise xi sweep of a 2048 x 2048 LLF stage went
// from 2.414 to 0.684 ms (JS) and from 2.773 to 0.780 ms (Z), the eta sweep from 2.301 to 0.655 and
// from 2.657 to 0.754 ms; what bounds them now is the integer ALU (71 % busy) and issue. A word
// carries 57 to 64 significant bits where a double carries 53, but they count from a stencil's largest
// difference; on the small side of a jump, where that says too little, FP64 takes over (enough,
// weno_value.cuh): 1 % of these sweeps for the test alone, 2 to 4 % of the time of the steps of a
// captured shock.
//
// The value. With g_m = lf_m - lf_(m+1), A_k = g_k - g_(k+1), B_0 = A_0 - 2 g_1, B_1 = g_1 + g_2,
// B_2 = A_2 + 2 g_2 and d_k = 4 (ss + beta_k) = 4 ss + 13/3 A_k^2 + B_k^2 (weno_fast.cuh), the
// candidates differ by third differences, so that with weights of sum one
//   6 (h - lf_2) = -(g_1 + 2 g_2) + 2 w_0 (A_0 - A_1) + w_2 (A_1 - A_2).
// The representation:
//  * the first differences become fixed-point integers of one exponent for the stencils of a face
//    value, that of the largest one, below 2^58: their sums and differences are exact (a large
//    difference cannot be clipped: two clipped ones would look alike to WENO-Z's tau);
//  * the indicators 3 d_k = 12 ss + 13 A_k^2 + 3 B_k^2 and everything made of them are positive
//    floating-point numbers of a 64-bit mantissa and an integer exponent, whose products need
//    no normalising between them; the weights' common denominators are those of weno_terms;
//  * the weights v_k are aligned to the largest (what they lose is below 2^-54 of their sum), and
//    the quotient by their sum is one 62-bit reciprocal, a hardware single-precision seed with one
//    third-order step;
//  * every rounding is a truncation of magnitudes, so a change of sign of the data changes the
//    sign of the result and nothing else: mirror-symmetric flows stay so bit for bit.
// A NaN or infinity among the differences, or a difference from 2^977 on, gives NaN (in FP64 the
// indicators' products overflow from 2^75 on). Against long double over random smooth,
// discontinuous and rough stencils the error's rms is 0.57 to 0.86 of the FP64 form's, its maximum
// 0.58 to 1.0; relative to the small side of a jump, where FP64 takes over, 0.6 to 1.0 and 0.6 to 1.1.
//
// The functions compile for the host too, where the tests compare them with long double.
#pragma once
#include "fastmath.cuh"

namespace dense {
namespace fx {

// Exponents of doubles in place (bits 20..30 of the upper word).
constexpr u32 kExpMask = 0x7ff00000u;
constexpr u32 kExpMin = 200u << 20;   // differences below 2^-882 count as zero
constexpr u32 kExpSS = 1014u << 20;   // of sqrt(4 ss) = 2^-9
constexpr u32 kExpMax = 2000u << 20;  // NaN, infinity, or so large that the result is NaN too
DENSE_FX u32 exponent(double g) { return hi32(bits(g)) & kExpMask; }
// The largest exponent of a stencil's differences.
DENSE_FX u32 exponent_of(const double g[4]) {
    return umax(umax(exponent(g[0]), exponent(g[1])), umax(exponent(g[2]), exponent(g[3])));
}
// The largest exponent of its smoothest substencil's two.
DENSE_FX u32 smoothest_of(const double g[4]) {
    const u32 e1 = exponent(g[1]), e2 = exponent(g[2]);
    return umin(umin(umax(exponent(g[0]), e1), umax(e1, e2)), umax(e2, exponent(g[3])));
}
// The exponent of what the rounding of a sum of two reconstructions is relative to (enough).
DENSE_FX u32 size_of(double lp, const double gp[4], double lm, const double gm[4]) {
    return umax(umax(exponent(lp), exponent(lm)), umax(smoothest_of(gp), smoothest_of(gm)) + (1u << 20));
}
// The fixed-point exponent E, in place, of a stencil's differences; top: at least the largest one's.
DENSE_FX u32 scale_of(const double g[4], u32& top) {
    const u32 most = exponent_of(g);
    top = umax(top, most);
    return umax(most, kExpMin);
}

// A double as a fixed-point integer in units of 2^(E - 1080) (E in place in eh, at least the
// double's): below 2^58, truncated. (A larger one comes out clipped.)
DENSE_FX i64 to_fixed(double g, u32 eh) {
    const u64 b = bits(g);
    const u32 h = hi32(b);
    const int sh = (int)(eh - (h & kExpMask)) >> 20;
    // 1.m in [2^62, 2^63); where the exponent is zero the shift leaves nothing of it
    const u64 m = ((u64)((((h << 10) | ((u32)b >> 22)) & 0x3fffffffu) | 0x40000000u) << 32) | (u32)((u32)b << 10);
    const u64 a = shr(m, (u32)imax(sh, 0) + 5);
    const u64 s = (u64)(i64)((int)h >> 31);
    return (i64)((a ^ s) - s);
}
// c 2^(E - 1080) rounded to nearest, |c| below 2^63; NaN for top from kExpMax on
DENSE_FX double to_double(i64 c, u32 eh, u32 top) {
    const u64 a = abs64(c);
    const int n = clz64(a) & 63;
    u64 r = ((u64)c & 0x8000000000000000ull) | (((u64)((eh >> 20) + 5 - n) << 52) + ((((a << n) >> 10) + 1) >> 1));
    if (a == 0) r = 0;
    if (top >= kExpMax) r = 0x7ff8000000000000ull;
    return from_bits(r);
}

// a^2 / 2^64 for a below 2^61, at most 2 below its floor
DENSE_FX u64 sq61(u64 a) { return wide(hi32(a), hi32(a)) + hi32(wide(2 * hi32(a), (u32)a)); }
// 3 d_k = 12 ss + 13 A^2 + 3 B^2 as M 2^x (up to a power of two common to all), M with its top
// bit set; |A| and |B| at most 2^60. A and B are scaled up by 2^n first, so that a small
// indicator keeps its bits, but not past the unit of 12 ss, where nothing is left to keep: the
// squares' unit is then 2^up of it (or, where all differences are that small, 2^-down).
struct Indicator {
    u64 M;     // the mantissa
    int x;     // its exponent
    u64 a, b;  // |A| 2^n and |B| 2^n, the larger in [2^60, 2^61) unless n is capped
    u32 n;
};
DENSE_FX void indicator(i64 A, i64 B, u32 nmax, u32 down, Indicator& d) {
    constexpr u64 kS = (u64)(12.0 * (double)1.0e-6f * 302231454903657293676544.0);  // 12 ss 2^78
    d.a = abs64(A);
    d.b = abs64(B);
    d.n = umin((u32)clz64(d.a | d.b) - 3u, nmax);
    const u32 up = 2 * (nmax - d.n);
    d.a <<= d.n;
    d.b <<= d.n;
    const u64 q = shr(13 * sq61(d.a) + 3 * sq61(d.b), down) + shr(kS, up);  // below 2^63, at least 2^57
    const int z = clz32(hi32(q));
    d.x = (int)up - z;
    d.M = q << z;
}
// The three of a stencil. A square's unit is 2^(2 (E - 1080 - n) + 64), that of 12 ss 2^-78.
struct Stencil {
    i64 G1, G2, A0, A1, A2, B0, B1, B2;
    Indicator d[3];
};
DENSE_FX void stencil_of(const double g[4], u32 eh, Stencil& s) {
    s.G1 = to_fixed(g[1], eh);
    s.G2 = to_fixed(g[2], eh);
    s.A0 = to_fixed(g[0], eh) - s.G1;
    s.A1 = s.G1 - s.G2;
    s.A2 = s.G2 - to_fixed(g[3], eh);
    s.B0 = s.A0 - 2 * s.G1;
    s.B1 = s.G1 + s.G2;
    s.B2 = s.A2 + 2 * s.G2;
    const int e = (int)(eh >> 20) - 1009;
    const u32 nmax = (u32)imax(e, 0), down = (u32)imax(-2 * e, 0);
    indicator(s.A0, s.B0, nmax, down, s.d[0]);
    indicator(s.A1, s.B1, nmax, down, s.d[1]);
    indicator(s.A2, s.B2, nmax, down, s.d[2]);
}

// The weights' shares 2 w_0 and w_2 and their sum n = sum of all c_k v_k, from the indicators:
// u0/n = 2 w_0, u2/n = w_2, n in [2^62, 2^63). JS: v_k = P_k, the product of the other two
// squares; Z: v_k = D + tau^2 P_k (weno_terms), and lin = 10 D on the scale of n. The linear
// weights are 1, 6 and 3 tenths. The rest is for the gradient (correction6_taped).
struct Weights {
    u64 u0, u2, n, lin;
    u64 P[3];       // d_k^2 P_k is common to all: P[k] 2^(-a[k])
    int a[3], am;   // 2 x_k, the smallest
    u64 t[3];       // Z: c_k tau^2 P_k on the scale of n
    u64 tau;        // Z: |d_2 - d_0| = tau 2^xt
    int xt, shift;  // Z: 10 N = n 2^(shift + sum of a + 320), with P[k] 2^(-a[k]) = P_k 2^(-sum of a - 192)
};
template <bool Z>
DENSE_FX void weights(const Indicator d[3], Weights& w) {
    const int a0 = 2 * d[0].x, a1 = 2 * d[1].x, a2 = 2 * d[2].x, am = imin(imin(a0, a1), a2);
    const u64 q0 = sqhi(d[0].M), q1 = sqhi(d[1].M), q2 = sqhi(d[2].M);     // at least 2^62
    const u64 P0 = mulhi(q1, q2), P1 = mulhi(q0, q2), P2 = mulhi(q0, q1);  // at least 2^60 - 2
    w.P[0] = P0; w.P[1] = P1; w.P[2] = P2;
    w.a[0] = a0; w.a[1] = a1; w.a[2] = a2; w.am = am;
    u64 v0, v1, v2, t0 = 0, t1 = 0, t2 = 0, ds = 0;
    int X = 0;
    // v_k below 2^59 (10 x 2^59 < 2^63), the largest at least 2^54 (JS) or 2^57 (Z)
    if (!Z) {
        v0 = shr(P0, a0 - am + 5);
        v1 = shr(P1, a1 - am + 5);
        v2 = shr(P2, a2 - am + 5);
    } else {
        const int xm = imax(d[0].x, d[2].x);
        const u64 dd = abs64((i64)(shr(d[2].M, xm - d[2].x + 1) - shr(d[0].M, xm - d[0].x + 1)));
        const int c = clz64(dd) & 63;
        const int at = dd ? 2 * (xm + 1 - c) : -100000;  // tau = 0 leaves every v_k = D
        w.tau = dd << c;
        w.xt = xm + 1 - c;
        const u64 T = sqhi(w.tau);
        const u64 D = mulhi(q0, P0);
        t0 = mulhi(T, P0);
        t1 = mulhi(T, P1);
        t2 = mulhi(T, P2);
        // all below 2^(64 - z), z at most 6: the alignment shifts by that much less
        X = imax(0, at - am) + 6 - clz32(hi32(D | t0 | t1 | t2));
        ds = shr(D, X);
        t0 = shr(t0, X - (at - a0));
        t1 = shr(t1, X - (at - a1));
        t2 = shr(t2, X - (at - a2));
        v0 = ds + t0;
        v1 = ds + t1;
        v2 = ds + t2;
    }
    v2 *= 3;
    w.n = v0 + 6 * v1 + v2;
    const int c = clz32(hi32(w.n)) - 1;
    w.u0 = v0 << (c + 1);
    w.u2 = v2 << c;
    w.n <<= c;
    w.lin = (10 * ds) << c;
    w.t[0] = t0 << c;
    w.t[1] = (6 * t1) << c;
    w.t[2] = (3 * t2) << c;
    w.shift = X - c;
}

// u C / 2^64, truncated towards zero
DENSE_FX i64 scaled(u64 u, i64 C) {
    const u64 s = (u64)(C >> 63);
    return (i64)((mulhi(u, ((u64)C ^ s) - s) ^ s) - s);
}
// (u0 C0 + u2 C2) / n, |C| below 2^62, r = reciprocal(n)
DENSE_FX i64 weighted(const Weights& w, u64 r, i64 C0, i64 C2) {
    const i64 t = scaled(w.u0, C0) + scaled(w.u2, C2);
    const u64 s = (u64)(t >> 63);
    const u64 q = mulhi63((((u64)t ^ s) - s) << 1, r) << 2;
    return (i64)((q ^ s) - s);
}

// 6 (h - lf_2) of one stencil in units of 2^(E - 1080), from its first differences
template <bool Z>
DENSE_FX i64 correction6(const double g[4], u32 eh) {
    Stencil s;
    Weights w;
    stencil_of(g, eh, s);
    weights<Z>(s.d, w);
    return weighted(w, reciprocal(w.n), s.A0 - s.A1, s.A1 - s.A2) - s.G1 - 2 * s.G2;
}

// The same with the gradient 6 dh/dlf[m] in units of 2^-55, for the adjoint's tape: with W = h,
// r_k = -1/2 dW/dbeta_k and dbeta_k/dlf = 13/6 A_k dA_k/dlf + 1/2 B_k dB_k/dlf (weno_grad),
//   6 g_0 = 2 w_0 - 2 r_0 (13 A_0 + 3 B_0),
//   6 g_1 = -7 w_0 - w_1 + 2 r_0 (26 A_0 + 12 B_0) - 2 r_1 (13 A_1 + 3 B_1),
//   6 g_3 = 2 w_1 + 5 w_2 - 2 r_1 (13 A_1 - 3 B_1) + 2 r_2 (26 A_2 + 12 B_2),
//   6 g_4 = -w_2 - 2 r_2 (13 A_2 + 3 B_2),
// and the five sum to one. JS: r_k = 4 w_k (q_k - W)/d_k; Z: the same with the part of w_k that is
// not linear, and r_0, r_2 +- dW/dtau = 4 sum_k (q_k - W) c_k tau P_k / N. The r_k are floating-point
// (62 bits and an exponent), the products fixed-point: entries are of order one, their errors a
// few units of 2^-58, the truncations above all, where FP64 rounds each of a dozen sums.
struct Gradient {
    i64 g[5];
};
DENSE_FX i64 with_sign(u64 a, u64 s) { return (i64)((a ^ s) - s); }
// 2 r U L 2^(n - 4) in units of 2^-55: r an integer times U 2^e, U = 2^(E - 1080); down = the shift
DENSE_FX i64 share(i64 r, i64 L, int down) {
    const u64 p = mulhi(abs64(r), abs64(L)) << 2;  // below 2^63
    const u64 v = shr(p, (u32)imax(down + 2, 0)) << imin(imax(-down - 2, 0), 63);
    return with_sign(v, (u64)((r ^ L) >> 63));
}
template <bool Z>
DENSE_FX i64 correction6_taped(const double g[4], u32 eh, Gradient& out) {
    Stencil s;
    Weights w;
    stencil_of(g, eh, s);
    weights<Z>(s.d, w);
    const u64 rn = reciprocal(w.n);
    const i64 c6 = weighted(w, rn, s.A0 - s.A1, s.A1 - s.A2) - s.G1 - 2 * s.G2;
    const int E2 = 2 * (int)(eh >> 20);
    // 6 (q_k - W), below 2^62
    const i64 Q[3] = {2 * s.G1 + 2 * s.A0 - 5 * s.G1 - c6, -s.G1 - 2 * s.G2 - c6, s.G2 - s.A2 - 4 * s.G2 - c6};
    // the weights, and JS's r_k's, as fractions of 2^62
    const u64 f0 = mulhi63(w.u0 >> 1, rn) << 1, f2 = mulhi63(w.u2, rn) << 1;
    const u64 f1 = mulhi63(w.n - (w.u0 >> 1) - w.u2, rn) << 1;
    const u64 f[3] = {Z ? mulhi63(w.t[0], rn) << 1 : f0, Z ? mulhi63(w.t[1], rn) << 1 : f1,
                      Z ? mulhi63(w.t[2], rn) << 1 : f2};
    i64 r[3];  // times U 2^x[k]
    int x[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const u64 q = abs64(Q[k]);
        const int m = imax(clz64(q | 1) - 2, 0);
        const u64 t = mulhi(f[k], q << m) << 3;                         // below 2^63
        r[k] = with_sign(mulhi63(t, reciprocal(s.d[k].M >> 1)), (u64)(Q[k] >> 63));  // below 2^62
        x[k] = 16 - m - s.d[k].x;
    }
    if (Z) {
        // dW/dtau: the sum's terms c_k P_k (q_k - W) on one exponent
        const u64 o = abs64(Q[0]) | abs64(Q[1]) | abs64(Q[2]);
        const int m = imax(clz64(o | 1) - 3, 0);                           // Q 2^m below 2^61
        u64 p0 = shr(w.P[0], w.a[0] - w.am + 3), p1 = 6 * shr(w.P[1], w.a[1] - w.am + 3),
            p2 = 3 * shr(w.P[2], w.a[2] - w.am + 3);
        const int up = clz32(hi32(p0 | p1 | p2));
        p0 <<= up;
        p1 <<= up;
        p2 <<= up;
        const i64 y = scaled(p0, Q[0] * ((i64)1 << m)) + scaled(p1, Q[1] * ((i64)1 << m)) + scaled(p2, Q[2] * ((i64)1 << m));
        const u64 z = mulhi(mulhi63(rn, w.tau >> 1) << 1, abs64(y) << 1);  // |y| below 2^63
        const u64 same = (u64)(y >> 63);
        // d_2 >= d_0: r_0 gains it, r_2 loses it
        const bool ge = s.d[2].x > s.d[0].x || (s.d[2].x == s.d[0].x && s.d[2].M >= s.d[0].M);
        const int xz = 20 - m - up + w.xt - w.am - w.shift;
        const bool some = w.tau != 0;
#pragma unroll
        for (int k = 0; k < 3; k += 2) {
            const i64 v = some ? with_sign(z, same ^ ((k == 0) == ge ? 0ull : ~0ull)) : 0;
            // the two parts on the larger exponent of those that are not zero, two bits down
            const int xr = r[k] ? x[k] : -1000000, xv = v ? xz : -1000000, xm = imax(imax(xr, xv), -900000);
            const u64 a = shr(abs64(r[k]), (u32)imin(xm - xr, 64) + 1), b = shr(abs64(v), (u32)imin(xm - xv, 64) + 1);
            r[k] = with_sign(a, (u64)(r[k] >> 63)) + with_sign(b, (u64)(v >> 63));
            x[k] = xm + 1;
        }
    }
    i64 L[3], K[3];
    int down[3];
    const i64 As[3] = {s.A0, s.A1, s.A2}, Bs[3] = {s.B0, s.B1, s.B2};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const i64 A = with_sign(s.d[k].a >> 4, (u64)(As[k] >> 63)), B = with_sign(s.d[k].b >> 4, (u64)(Bs[k] >> 63));
        L[k] = 13 * A + 3 * B;                               // below 2^62
        K[k] = k == 1 ? 13 * A - 3 * B : 2 * L[k] + 6 * B;
        down[k] = imin(imax(2036 - E2 - x[k] + (int)s.d[k].n, -200), 200);
    }
    const i64 h0 = (i64)(f0 >> 4), h1 = (i64)(f1 >> 4), h2 = (i64)(f2 >> 4);  // units of 2^-58
    out.g[0] = ((2 * h0) / 8) - share(r[0], L[0], down[0]);
    out.g[1] = -((7 * h0 + h1) / 8) + share(r[0], K[0], down[0]) - share(r[1], L[1], down[1]);
    out.g[3] = (2 * h1 + 5 * h2) / 8 - share(r[1], K[1], down[1]) + share(r[2], K[2], down[2]);
    out.g[4] = -(h2 / 8) - share(r[2], L[2], down[2]);
    out.g[2] = ((i64)6 << 55) - out.g[0] - out.g[1] - out.g[3] - out.g[4];
    return c6;
}
// The entries of a gradient (NaN where top says so).
DENSE_FX void gradient_out(const Gradient& q, u32 top, double g[5]) {
#pragma unroll
    for (int m = 0; m < 5; ++m) g[m] = to_double(q.g[m], 1025u << 20, top) * (1.0 / 6.0);
}

// Whether lp is the smaller one in magnitude (of two opposite ones, the positive).
DENSE_FX bool smaller(double lp, double lm) {
    const u64 ap = bits(lp) << 1, am = bits(lm) << 1;          // (an FP64 absolute value would take that pipe)
    return ap < am || (ap == am && (i64)bits(lp) >= 0);
}
// lp + lm + c/6, c on the smaller one first: the two FP64 roundings are no larger than those of two
// values and their sum, and the same in either order.
DENSE_FX double about(double lp, double lm, double c) {
    const bool first = smaller(lp, lm);
    return fma(c, 1.0 / 6.0, first ? lp : lm) + (first ? lm : lp);
}
// Whether about(lp, lm, c) is to be computed in FP64 instead: the exponent, in place, that c has to reach
// for the integer form, 0 where any will do. top is the largest exponent of the differences, size
// that of what the value's rounding is relative to: lp, lm and twice the smoothest substencil
// (size_of). Past the value's own rounding the integer form is good to a few of its units, which are
// 2^-57 of the largest difference, FP64 to 2^-53 of the values and of the corrections, which are
// no smaller than the smoothest substencils' differences but by chance. So where the largest
// difference is of a higher binade than all of these -- on the small side of a jump, of either
// stencil -- FP64 is more exact. (Above 2^72 its products would overflow; from kExpMax on the
// result is NaN.)
constexpr u32 kExpFP64 = 1095u << 20;
DENSE_FX u32 enough(u32 top, u32 size) {
    u32 n = top > size && top <= kExpFP64 ? top : 0u;
#ifdef __CUDA_ARCH__
    asm volatile("" : "+r"(n));  // formed here, not after the corrections with its inputs kept in registers
#endif
    return n;
}
// The sum of two reconstructions about lp and lm, whose corrections share their exponent and the
// conversion back. gm: the second's differences with the opposite sign, as a sweep has them (a
// correction is odd in its differences, to the bit; negating doubles would take the FP64 pipe). fp64:
// takes whether it is to be computed in FP64 instead.
template <bool Z>
DENSE_FX double pair(double lp, const double gp[4], double lm, const double gm[4], bool* fp64 = nullptr) {
    u32 top = 0;
    const u32 ep = scale_of(gp, top), eh = umax(ep, scale_of(gm, top));
    const u32 need = fp64 ? enough(top, size_of(lp, gp, lm, gm)) : 0u;
    const double c = to_double(correction6<Z>(gp, eh) - correction6<Z>(gm, eh), eh, top);
    if (fp64) *fp64 = exponent(c) < need;
    return about(lp, lm, c);
}
// Whether the unit eh of a stencil's differences lies more than two binades (JS; Z: one) above its smoothest
// substencil (or sqrt(ss)), by a difference of its own or of the stencil it shares the unit with: the
// gradient's terms are relative to the smoothest substencil, and the fixed-point differences then know
// it less well than FP64 does. Such stencils, beside extrema and jumps, take weno_grad's gradient.
// Against long double the rms error is 0.56 to 1.0 of weno_grad's; with two binades Z's would be 1.1
// beside jumps, and told by a stencil's own differences alone 9 to 11 where the partner has the jump.
// (JS with one: 256 x 256 adjoint 7.61 ms instead of 7.30.)
template <bool Z>
DENSE_FX bool rough(const double g[4], u32 eh) {
    return eh > umax(smoothest_of(g), kExpSS) + ((Z ? 1u : 2u) << 20);
}
DENSE_FX bool rough(const double g[4]) { return rough<false>(g, exponent_of(g)); }
// 6 (h - lf_2) of one reconstruction.
template <bool Z>
DENSE_FX double correction(const double g[4]) {
    u32 top = 0;
    const u32 eh = scale_of(g, top);
    return to_double(correction6<Z>(g, eh), eh, top);
}

// AdaWENO: the WENO-Z weights of a scalar surrogate, from its first differences, as fractions
// 2 w_0 = f0/2^62 and w_2 = f2/2^62, and its switch theta > delta, which is 10 D > theta_c n
// (Params::theta_c; 0 always, 1 never). A NaN or infinity is not smooth.
DENSE_FX bool surrogate(const double g[4], double theta_c, u64& f0, u64& f2) {
    u32 top = 0;
    const u32 eh = scale_of(g, top);
    Stencil s;
    Weights w;
    stencil_of(g, eh, s);
    weights<true>(s.d, w);
    const u64 r = reciprocal(w.n);
    f0 = mulhi63(w.u0 >> 1, r) << 2;
    f2 = mulhi63(w.u2, r) << 1;
    const u64 tb = bits(theta_c);
    const u32 te = (u32)(tb >> 52);  // theta_c in [0, 1]: its exponent field is at most 1023
    const u64 tc = shr((tb << 11) | 0x8000000000000000ull, 1022u - te);
    const bool smooth = te == 0 || (te < 1023u && w.lin > mulhi(w.n, tc));
    return smooth && top < kExpMax;
}
// 6 (h - lf_2) of another stencil by a surrogate's weights, in units of 2^(E - 1080), E at least
// the exponent of its differences.
DENSE_FX i64 correction6_by(const double g[4], u32 eh, u64 f0, u64 f2) {
    const i64 G1 = to_fixed(g[1], eh), G2 = to_fixed(g[2], eh);
    const i64 A0 = to_fixed(g[0], eh) - G1, A1 = G1 - G2, A2 = G2 - to_fixed(g[3], eh);
    return scaled(f0, (A0 - A1) * 4) + scaled(f2, (A1 - A2) * 4) - G1 - 2 * G2;
}

// Whether the smooth branch may meet weights far from the linear ones: down to delta = 0.01 a smooth
// surrogate's are within a factor of 11 (sum alpha - 1 <= 10) and its differences alike, so that a jump
// of a component counts in its value, and the integer form's rms error is 0.6 to 0.75 of FP64's beside
// jumps of any size. theta_c = k/(1 + k), k = sqrt(delta/(1 - delta)).
DENSE_FX bool far_weights(double theta_c) { return theta_c < 0.0913; }
// Where it may: whether about(lp, lm, c6) of such corrections is to be computed in FP64 instead (enough; the
// sum's rounding is relative to a few binades more than it, and a surrogate that is rough is never left
// to integers).
DENSE_FX bool coarse_by(u32 top, double lp, double lm, double c6) {
    return exponent(c6) + (3u << 20) < enough(top, umax(exponent(lp), exponent(lm)));
}

// dt/dx and dt/dy, each m 2^(e - 1086) with the top bit of m set, 0 for a zero rate, and dt's sign; e kNoRate
// where one is not finite.
constexpr int kNoRate = 1 << 20;
struct Rate {
    u64 m;
    int e;
};
struct Rates {
    Rate x, y;
    u32 sign;  // 0 or the sign bit of an upper word
};
DENSE_FX Rate rate_of(u64 b) {
    const int e = (int)((b >> 52) & 0x7ff);
    Rate r;
    r.m = e ? (b << 11) | 0x8000000000000000ull : 0;
    r.e = e == 0x7ff ? kNoRate : e;
    return r;
}
DENSE_FX Rates rates_of(double dtdx, double dtdy) {
    Rates r;
    r.x = rate_of(bits(dtdx));
    r.y = rate_of(bits(dtdy));
    r.sign = hi32(bits(dtdx)) & 0x80000000u;
    return r;
}
// A rate times the difference of two fluxes: sign (all ones or zero) and m 2^(e - 1080), m below 2^63 and not below
// 2^61 (or 0). The fluxes are fixed-point integers of their own exponent, 2^-57 of the larger one, so
// that their difference is exact unless one of them is 2^5 times the other, and good to 2^-57 then.
struct Change {
    u64 m, sign;
    int e;
};
DENSE_FX Change change_of(double l, double r, const Rate& q, u32& top) {
    const u32 t = umax(exponent(l), exponent(r)), eh = umax(t, 64u << 20);
    top = umax(top, t);
    const i64 d = to_fixed(r, eh) - to_fixed(l, eh);  // below 2^59
    const u64 a = abs64(d);
    const int n = clz64(a) & 63;
    Change c;
    c.m = mulhi(a << n, q.m) >> 1;
    c.sign = (u64)(d >> 63);
    c.e = c.m ? (int)(eh >> 20) - n + q.e - 1021 : -10000;
    return c;
}
// dt/dx (xr - xl) + dt/dy (yr - yl): each direction's difference exact or good to 2^-57 of itself, its
// product with the rate truncated below 2^-60, the smaller product to the larger one's unit, their sum
// rounded once. Below 2^-950 the result is 0; NaN for what is not finite.
DENSE_FX double flux_change(double xl, double xr, double yl, double yr, const Rates& q) {
    u32 top = 0;
    const Change x = change_of(xl, xr, q.x, top), y = change_of(yl, yr, q.y, top);
    const int e = imax(x.e, y.e);
    const u64 a = shr(x.m, (u32)(e - x.e) + 1), b = shr(y.m, (u32)(e - y.e) + 1);
    const i64 t = (i64)((a ^ x.sign) - x.sign) + (i64)((b ^ y.sign) - y.sign);   // below 2^63
    const u64 m = abs64(t);
    const int n = clz64(m) & 63;
    // (as to_double, with an infinity from 2^1024 on: a product in its place would take the FP64 pipe)
    u64 r = ((u64)(imin(e, 3000) + 6 - n) << 52) + ((((m << n) >> 10) + 1) >> 1);
    if (r >= 0x7ff0000000000000ull) r = 0x7ff0000000000000ull;
    r |= (u64)t & 0x8000000000000000ull;
    if (e + 1 < 64 || m == 0) r = 0;
    if (top >= 0x7ff00000u || umax((u32)q.x.e, (u32)q.y.e) == (u32)kNoRate) r = 0x7ff8000000000000ull;
    return from_bits(r ^ ((u64)q.sign << 32));
}

}  // namespace fx
}  // namespace dense
