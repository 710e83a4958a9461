// weno_value.cuh -- a face's value in FP64, for the stencils that the integer form (weno_fixed.cuh)
// leaves to it: its unit is 2^-57 of a stencil's largest difference, which beside a jump says too
// little about a value on the small side (fx::enough). Included inside the sweeps' own namespace, after
// weno_fast.cuh.
#pragma once

// a b, not to be contracted with what it is added to: the plain and taping sweeps round alike
__device__ __forceinline__ double product(double a, double b) {
#ifdef __CUDA_ARCH__
    return __dmul_rn(a, b);
#else
    return a * b;
#endif
}
// h - lf_2 of one stencil, from its first differences
template <bool Z>
__device__ __forceinline__ double correction_fp64(const double g[4]) {
    double d0, d1, d2, B[3];
    betas_g(g, d0, d1, d2, B);
    WenoTerms t;
    weno_terms<Z>(g, d0, d1, d2, t);
    return product(weno_num(t), fx::rcp(t.N));
}
// fx::about of a sum c of corrections that is not six times over
__device__ __forceinline__ double about_fp64(double lp, double lm, double c) {
    const bool first = fx::smaller(lp, lm);
    return ((first ? lp : lm) + c) + (first ? lm : lp);
}
// The weights of a stencil over the linear ones, w_k / c_k, from its first differences, and what a
// reconstruction with such weights adds to the centre of another stencil (AdaWENO's smooth branch)
template <bool Z>
__device__ __forceinline__ void weights_fp64(const double g[4], double u[3]) {
    double d0, d1, d2, B[3];
    betas_g(g, d0, d1, d2, B);
    WenoTerms t;
    weno_terms<Z>(g, d0, d1, d2, t);
    const double iN = fx::rcp(t.N);
#pragma unroll
    for (int k = 0; k < 3; ++k) u[k] = t.v[k] * iN;
}
__device__ __forceinline__ double correction_by_fp64(const double g[4], const double u[3]) {
    const double r0 = fma(c30 / 3.0, g[0], (-5.0 * c30 / 6.0) * g[1]);
    const double r1 = fma(-c31 / 3.0, g[2], (-c31 / 6.0) * g[1]);
    const double r2 = fma(c32 / 6.0, g[3], (-2.0 * c32 / 3.0) * g[2]);
    return fma(u[2], r2, fma(u[1], r1, u[0] * r0));
}
