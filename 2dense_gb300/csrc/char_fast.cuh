// char_fast.cuh -- characteristic-wise WENO-Z of the fast kernels (104 and AdaWENO's characteristic
// branch): Roe state, projection, corrections of the fields, back-projection. Included inside the
// sweeps' own namespace, after weno_value.cuh.
#pragma once

// The Roe state of the two cells next to an interface from
// their sqrt(rho) and total enthalpy H = gamma/(gamma-1) p/rho + |u|^2/2 (staged once per cell),
// with one reciprocal for the three weighted means and one inverse square root giving both
// alpha0 and 1/alpha0; 1/hh0 = (gamma-1)/alpha0^2. With n the normal and t the tangential momentum
// component, the projection on the left eigenvectors of get_l_r_vec_xi/_eta
// (scheme_weno5th_SC.f90:277-328, 607-658) is
//   w = f_n - u_n0 f_0,  q = f_t - u_t0 f_0,  z = f_3 - uu0 f_0 - u_n0 w - u_t0 q,
//   l_0 = z/(2 hh0) - w/(2 a0),  l_1 = f_0 - z/hh0,  l_2 = q,  l_3 = z/(2 hh0) + w/(2 a0)
// (9 operations where the rows' products take 13), and the back-projection
//   h_0 = c0 + c1 + c3,  h_n = u_n0 h_0 + a0 (c3 - c0),  h_t = u_t0 h_0 + c2,
//   h_3 = H0 (c0 + c3) + a0 u_n0 (c3 - c0) + uu0 c1 + u_t0 c2.
struct EigFast {
    double un0, ut0, a0, h0, uu0;
    double ia5, ih, ihh;  // 1/(2 a0), 1/(2 hh0), 1/hh0
};

template <int DIR>
__device__ __forceinline__ bool roe_eig_fast(double g1, double sl, double sr, double ul, double ur,
                                             double vl, double vr, double hl, double hr, EigFast& e) {
    // (each mean as one sum: about either side's value it would keep that value's rounding, which the other
    // side's weight may dwarf -- of an enthalpy 1e8 times the other's at that density ratio, 1e-12 of the mean)
    const double r = fx::rcp(sl + sr);
    const double u0 = fma(sr, ur, sl * ul) * r;
    const double v0 = fma(sr, vr, sl * vl) * r;
    e.h0 = fma(sr, hr, sl * hl) * r;
    e.uu0 = 0.5 * fma(u0, u0, v0 * v0);
    const double c2 = g1 * (e.h0 - e.uu0);
    const double ia = fx::rsqrt(c2);
    e.a0 = c2 * ia;
    e.ia5 = 0.5 * ia;
    e.ih = g1 * ia * e.ia5;
    e.ihh = 2.0 * e.ih;
    e.un0 = DIR == 0 ? u0 : v0;
    e.ut0 = DIR == 0 ? v0 : u0;
    return c2 > 0.0;
}

// Characteristic fields of a flux (or flux difference) f.
template <int DIR>
__device__ __forceinline__ void project_fast(const EigFast& e, const double f[4], double l[4]) {
    const double w = fma(-e.un0, f[0], f[1 + DIR]), q = fma(-e.ut0, f[0], f[2 - DIR]);
    const double z = fma(-e.ut0, q, fma(-e.un0, w, fma(-e.uu0, f[0], f[3])));
    const double m = e.ia5 * w;
    l[0] = fma(e.ih, z, -m);
    l[1] = fma(-e.ihh, z, f[0]);
    l[2] = q;
    l[3] = fma(e.ih, z, m);
}

// Characteristic-wise WENO-Z. The projection is linear, so a field's first differences are the
// projected differences of the split flux; and the projected centre value, projected back, is the
// centre flux itself, so that only the reconstructions' corrections pass through the fields:
//   h = F+(centre) + F-(centre) + sum_k r_k (c_k+ + c_k-),
// one back-projection for both signs and none of the centres' projections.
//
// cs[k]: 6 c_k of one sign from its differences dF(m, f); returns the fields (bits) that FP64 is to do
// instead (char_field_fp64). A field's rounding is relative to the centre's share of the fields,
// which the back-projection adds up: f0, the centre's first component, for the fields 0, 1 and 3, its
// tangential momentum ft and u_t f0 for the second. Where 16 times that and the correction itself
// are of lower binades than the largest difference, FP64 takes the field (fx::enough). 16: beside
// jumps of 0.1 to 1e8 times the level the rms error of the fluxes is 0.05 to 0.85 of that of an
// FP64 reconstruction of the fields' values, which projects the centre too.
template <int DIR, typename Diff>
__device__ __forceinline__ unsigned char_fields(const EigFast& e, Diff dF, double f0, double ft, double cs[4]) {
    double g[4][4];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        double f[4], l[4];
        dF(m, f);
        project_fast<DIR>(e, f, l);
#pragma unroll
        for (int k = 0; k < 4; ++k) g[k][m] = l[k];
    }
    constexpr fx::u32 k16 = 4u << 20;
    const fx::u32 s0 = fx::exponent(f0) + k16;
    const fx::u32 s2 = fx::umax(fx::exponent(ft) + k16, (fx::u32)fx::imax((int)(fx::exponent(e.ut0) + s0) - (1023 << 20), 0));
    unsigned redo = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        fx::u32 top = 0;
        const fx::u32 eh = fx::scale_of(g[k], top);
        const fx::u32 need = fx::enough(top, k == 2 ? s2 : s0);
        cs[k] = fx::to_double(fx::correction6<true>(g[k], eh), eh, top);
        if (fx::exponent(cs[k]) < need) redo |= 1u << k;
    }
    return redo;
}
// 6 c_k of field k in FP64
template <int DIR, typename Diff>
__device__ __forceinline__ double char_field_fp64(const EigFast& e, Diff dF, int k) {
    double g[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        double f[4], l[4];
        dF(m, f);
        project_fast<DIR>(e, f, l);
        g[m] = k == 0 ? l[0] : k == 1 ? l[1] : k == 2 ? l[2] : l[3];
    }
    return product(6.0, correction_fp64<true>(g));
}
template <int DIR>
__device__ __forceinline__ void back_project_fast(const EigFast& e, const double c[4], const double centre[4],
                                                  double h[4]) {
    const double s = c[0] + c[3], d = c[3] - c[0], h0 = s + c[1], ad = e.a0 * d;
    const double hn = fma(e.un0, h0, ad), ht = fma(e.ut0, h0, c[2]);
    const double h3 = fma(e.h0, s, fma(e.un0, ad, fma(e.uu0, c[1], e.ut0 * c[2])));
    h[0] = fma(1.0 / 6.0, h0, centre[0]);
    h[1 + DIR] = fma(1.0 / 6.0, hn, centre[1 + DIR]);
    h[2 - DIR] = fma(1.0 / 6.0, ht, centre[2 - DIR]);
    h[3] = fma(1.0 / 6.0, h3, centre[3]);
}
