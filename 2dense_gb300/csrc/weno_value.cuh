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
