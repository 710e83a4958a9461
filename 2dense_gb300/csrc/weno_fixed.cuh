// weno_fixed.cuh -- WENO-JS5 / WENO-Z5 reconstructions on the integer pipes, for the fast sweeps.
//
// GB300 issues an FP64 instruction of a warp every 16 cycles of an SM, and in that time up to 64
// others: measured per warp and SM, DFMA 16.9 cycles, against 0.6 for a 32-bit IMAD or LOP, 1.0 for a
// 32x32+64-bit IMAD.WIDE, 0.6 for a 64-bit shift and 4.5 for the upper half of a 64x64-bit
// product. A reconstruction in FP64 is about 34 instructions, 556 (JS) to 668 (Z) cycles with the
// integer pipes idle; the same value in 64-bit integers takes 172 and 205, and leaves the FP64 pipe
// to the split fluxes of other warps. The component-wise xi sweep of a 2048 x 2048 LLF stage went
// from 2.414 to 0.684 ms (JS) and from 2.773 to 0.778 ms (Z), the eta sweep from 2.301 to 0.663 and
// from 2.657 to 0.772 ms; what bounds them now is the integer ALU (72 % busy, 340 instructions a
// reconstruction before its last trimming). Nothing is computed in fewer bits than before: the
// words carry 57 to 64 significant bits where a double carries 53.
//
// The value. With g_m = lf_m - lf_(m+1), A_k = g_k - g_(k+1), B_0 = A_0 - 2 g_1, B_1 = g_1 + g_2,
// B_2 = A_2 + 2 g_2 and d_k = 4 (ss + beta_k) = 4 ss + 13/3 A_k^2 + B_k^2 (weno_fast.cuh), the
// candidates differ by third differences, so that with weights of sum one
//   6 (h - lf_2) = -(g_1 + 2 g_2) + 2 w_0 (A_0 - A_1) + w_2 (A_1 - A_2).
// The representation:
//  * the first differences become fixed-point integers of one exponent for the stencils of a face
//    value, below 2^58: their sums and differences are exact. The exponent is the largest
//    difference's, but at most kCap above that of the smoothest substencil (of sqrt(ss), where that
//    is more): past a jump of 2^kCap times the rest, the weights leave 2^-3kCap of the rest to the
//    substencils that contain it, whatever it is, so it may as well be clipped, and the rest keeps
//    57 - kCap bits or more beside any jump;
//  * the indicators 3 d_k = 12 ss + 13 A_k^2 + 3 B_k^2 and everything made of them are positive
//    floating-point numbers of a 64-bit mantissa and an integer exponent, whose products need
//    no normalising between them; the weights' common denominators are those of weno_terms;
//  * the weights v_k are aligned to the largest (what they lose is below 2^-54 of their sum), and
//    the quotient by their sum is one 62-bit reciprocal, a hardware single-precision seed with one
//    third-order step;
//  * every rounding is a truncation of magnitudes, so a change of sign of the data changes the
//    sign of the result and nothing else: mirror-symmetric flows stay so bit for bit.
// A NaN or infinity among the differences gives NaN. Against long double over random smooth,
// discontinuous and rough stencils the error's rms is 0.57 to 0.86 of the FP64 form's, its maximum
// 0.58 to 1.0.
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
constexpr u32 kCap = 15u;
DENSE_FX u32 exponent(double g) { return hi32(bits(g)) & kExpMask; }
// The fixed-point exponent E, in place, of a stencil's differences; top: at least the largest one's.
DENSE_FX u32 scale_of(const double g[4], u32& top) {
    const u32 e1 = exponent(g[1]), e2 = exponent(g[2]);
    const u32 m0 = umax(exponent(g[0]), e1), m1 = umax(e1, e2), m2 = umax(e2, exponent(g[3]));
    const u32 most = umax(m0, m2), least = umin(umin(m0, m1), m2);
    top = umax(top, most);
    return umax(umin(most, umax(least, kExpSS) + (kCap << 20)), kExpMin);
}

// A double as a fixed-point integer in units of 2^(E - 1080) (E in place in eh): below 2^58,
// truncated; a larger one clipped to E.
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
DENSE_FX u64 indicator(i64 A, i64 B, u32 nmax, u32 down, int& x) {
    constexpr u64 kS = (u64)(12.0 * (double)1.0e-6f * 302231454903657293676544.0);  // 12 ss 2^78
    u64 a = abs64(A), b = abs64(B);
    const u32 n = umin((u32)clz64(a | b) - 3u, nmax), up = 2 * (nmax - n);
    a <<= n;
    b <<= n;
    const u64 d = shr(13 * sq61(a) + 3 * sq61(b), down) + shr(kS, up);  // below 2^63, at least 2^57
    const int z = clz32(hi32(d));
    x = (int)up - z;
    return d << z;
}
// The three of a stencil. A square's unit is 2^(2 (E - 1080 - n) + 64), that of 12 ss 2^-78.
DENSE_FX void indicators(i64 A0, i64 A1, i64 A2, i64 G1, i64 G2, u32 eh, u64 M[3], int x[3]) {
    const int e = (int)(eh >> 20) - 1009;
    const u32 nmax = (u32)imax(e, 0), down = (u32)imax(-2 * e, 0);
    M[0] = indicator(A0, A0 - 2 * G1, nmax, down, x[0]);
    M[1] = indicator(A1, G1 + G2, nmax, down, x[1]);
    M[2] = indicator(A2, A2 + 2 * G2, nmax, down, x[2]);
}

// The weights' shares 2 w_0 and w_2 and their sum n = sum of all c_k v_k, from the indicators:
// u0/n = 2 w_0, u2/n = w_2, n in [2^62, 2^63). JS: v_k = P_k, the product of the other two
// squares; Z: v_k = D + tau^2 P_k (weno_terms), and lin = 10 D on the scale of n. The linear
// weights are 1, 6 and 3 tenths.
template <bool Z>
DENSE_FX void weights(const u64 M[3], const int x[3], u64& u0, u64& u2, u64& n, u64& lin) {
    const int a0 = 2 * x[0], a1 = 2 * x[1], a2 = 2 * x[2], am = imin(imin(a0, a1), a2);
    const u64 q0 = sqhi(M[0]), q1 = sqhi(M[1]), q2 = sqhi(M[2]);           // at least 2^62
    const u64 P0 = mulhi(q1, q2), P1 = mulhi(q0, q2), P2 = mulhi(q0, q1);  // at least 2^60 - 2
    u64 v0, v1, v2;
    lin = 0;
    // v_k below 2^59 (10 x 2^59 < 2^63), the largest at least 2^54 (JS) or 2^57 (Z)
    if (!Z) {
        v0 = shr(P0, a0 - am + 5);
        v1 = shr(P1, a1 - am + 5);
        v2 = shr(P2, a2 - am + 5);
    } else {
        const int xm = imax(x[0], x[2]);
        const u64 dd = abs64((i64)(shr(M[2], xm - x[2] + 1) - shr(M[0], xm - x[0] + 1)));
        const int c = clz64(dd) & 63;
        const int at = dd ? 2 * (xm + 1 - c) : -100000;  // tau = 0 leaves every v_k = D
        const u64 T = sqhi(dd << c);
        const u64 D = mulhi(q0, P0), t0 = mulhi(T, P0), t1 = mulhi(T, P1), t2 = mulhi(T, P2);
        // all below 2^(64 - z), z at most 6: the alignment shifts by that much less
        const int X = imax(0, at - am) + 6 - clz32(hi32(D | t0 | t1 | t2));
        const u64 ds = shr(D, X);
        lin = 10 * ds;
        v0 = ds + shr(t0, X - (at - a0));
        v1 = ds + shr(t1, X - (at - a1));
        v2 = ds + shr(t2, X - (at - a2));
    }
    v2 *= 3;
    n = v0 + 6 * v1 + v2;
    const int c = clz32(hi32(n)) - 1;
    u0 = v0 << (c + 1);
    u2 = v2 << c;
    n <<= c;
    lin <<= c;
}

// u C / 2^64, truncated towards zero
DENSE_FX i64 scaled(u64 u, i64 C) {
    const u64 s = (u64)(C >> 63);
    return (i64)((mulhi(u, ((u64)C ^ s) - s) ^ s) - s);
}
// (u0 C0 + u2 C2) / n, |C| below 2^62
DENSE_FX i64 weighted(u64 u0, u64 u2, u64 n, i64 C0, i64 C2) {
    const i64 t = scaled(u0, C0) + scaled(u2, C2);
    const u64 s = (u64)(t >> 63);
    const u64 q = mulhi63((((u64)t ^ s) - s) << 1, reciprocal(n)) << 2;
    return (i64)((q ^ s) - s);
}

// 6 (h - lf_2) of one stencil in units of 2^(E - 1080), from its first differences
template <bool Z>
DENSE_FX i64 correction6(const double g[4], u32 eh) {
    const i64 G1 = to_fixed(g[1], eh), G2 = to_fixed(g[2], eh);
    const i64 A0 = to_fixed(g[0], eh) - G1, A1 = G1 - G2, A2 = G2 - to_fixed(g[3], eh);
    u64 M[3], u0, u2, n, lin;
    int x[3];
    indicators(A0, A1, A2, G1, G2, eh, M, x);
    weights<Z>(M, x, u0, u2, n, lin);
    return weighted(u0, u2, n, A0 - A1, A1 - A2) - G1 - 2 * G2;
}

// lp + lm + c/6, c on the smaller one first: the two FP64 roundings are no larger than those of two
// values and their sum, and the same in either order.
DENSE_FX double about(double lp, double lm, double c) {
    const u64 ap = bits(lp) << 1, am = bits(lm) << 1;          // (an FP64 absolute value would take that pipe)
    const bool first = ap < am || (ap == am && (i64)bits(lp) >= 0);  // of two opposite ones, the positive
    return fma(c, 1.0 / 6.0, first ? lp : lm) + (first ? lm : lp);
}
// The sum of two reconstructions about lp and lm, whose corrections share their exponent and the
// conversion back. gm: the second's differences with the opposite sign, as a sweep has them (a
// correction is odd in its differences, to the bit; negating doubles would take the FP64 pipe).
template <bool Z>
DENSE_FX double pair(double lp, const double gp[4], double lm, const double gm[4]) {
    u32 top = 0;
    const u32 ep = scale_of(gp, top), eh = umax(ep, scale_of(gm, top));
    const double c = to_double(correction6<Z>(gp, eh) - correction6<Z>(gm, eh), eh, top);
    return about(lp, lm, c);
}
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
    const i64 G1 = to_fixed(g[1], eh), G2 = to_fixed(g[2], eh);
    const i64 A0 = to_fixed(g[0], eh) - G1, A1 = G1 - G2, A2 = G2 - to_fixed(g[3], eh);
    u64 M[3], u0, u2, n, lin;
    int x[3];
    indicators(A0, A1, A2, G1, G2, eh, M, x);
    weights<true>(M, x, u0, u2, n, lin);
    const u64 r = reciprocal(n);
    f0 = mulhi63(u0 >> 1, r) << 2;
    f2 = mulhi63(u2, r) << 1;
    const u64 tb = bits(theta_c);
    const u32 te = (u32)(tb >> 52);  // theta_c in [0, 1]: its exponent field is at most 1023
    const u64 tc = shr((tb << 11) | 0x8000000000000000ull, 1022u - te);
    const bool smooth = te == 0 || (te < 1023u && lin > mulhi(n, tc));
    return smooth && top < kExpMax;
}
// 6 (h - lf_2) of another stencil by a surrogate's weights, in units of 2^(E - 1080), E at least
// the exponent of its differences (the weights are not its own: nothing is clipped).
DENSE_FX i64 correction6_by(const double g[4], u32 eh, u64 f0, u64 f2) {
    const i64 G1 = to_fixed(g[1], eh), G2 = to_fixed(g[2], eh);
    const i64 A0 = to_fixed(g[0], eh) - G1, A1 = G1 - G2, A2 = G2 - to_fixed(g[3], eh);
    return scaled(f0, (A0 - A1) * 4) + scaled(f2, (A1 - A2) * 4) - G1 - 2 * G2;
}
// The largest exponent of a stencil's differences.
DENSE_FX u32 exponent_of(const double g[4]) {
    return umax(umax(exponent(g[0]), exponent(g[1])), umax(exponent(g[2]), exponent(g[3])));
}

// dt/dx and dt/dy as fixed-point factors of one exponent, below 2^62 (in units of 2^-shift), and
// dt's sign; shift kNoShift where one is not finite.
constexpr int kNoShift = 1 << 20;
struct Rates {
    u64 x, y;
    int shift;
    u32 sign;  // 0 or the sign bit of an upper word
};
DENSE_FX Rates rates_of(double dtdx, double dtdy) {
    const u64 bx = bits(dtdx), by = bits(dtdy), top = 0x2000000000000000ull;
    const u32 ex = (hi32(bx) >> 20) & 0x7ffu, ey = (hi32(by) >> 20) & 0x7ffu, e = umax(ex, ey);
    Rates r;
    r.x = shr(((bx << 9) & (top - 1)) | top, e - ex);
    r.y = shr(((by << 9) & (top - 1)) | top, e - ey);
    r.shift = e == 0x7ffu ? kNoShift : 61 + 1023 - (int)e;
    r.sign = hi32(bx) & 0x80000000u;
    return r;
}
// dt/dx (xr - xl) + dt/dy (yr - yl): the differences exact in fixed point, their products with the rates
// and the sum truncated below 2^-57 of the largest flux times the larger rate, rounded once.
DENSE_FX double flux_change(double xl, double xr, double yl, double yr, const Rates& r) {
    const u32 top = umax(umax(exponent(xl), exponent(xr)), umax(exponent(yl), exponent(yr)));
    const u32 eh = umax(top, kExpMin);
    const i64 X = to_fixed(xr, eh) - to_fixed(xl, eh), Y = to_fixed(yr, eh) - to_fixed(yl, eh);  // below 2^59
    const i64 t = scaled(r.x, X * 8) + scaled(r.y, Y * 8);     // 2^(shift - 61) of the sum, below 2^61
    const int e = (int)(eh >> 20) + 61 - r.shift;
    double d = to_double(t, (u32)imax(e, 64) << 20, top);
    if (e < 64) d = 0.0;                                       // below 2^-950: also where a rate is 0
    if (r.shift == kNoShift) d = from_bits(0x7ff8000000000000ull);
    return from_bits(bits(d) ^ ((u64)r.sign << 32));
}

}  // namespace fx
}  // namespace dense
