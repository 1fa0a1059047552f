// Refined FP64 reciprocals and roots of the pair and triplet kernels (included by
// d3_engine.cu; checked against CUDA's double functions by k_selftest_math).

__device__ __forceinline__ double rsqrt_nr(double x) {
    // x^(-1/2): the hardware's double-precision approximation (relative error ~2^-20,
    // no conversions) and one third-order step, y (1 + e/2 + 3/8 e^2) with e = 1 - x y^2
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x * y, y, 1.0);
    return fma(y * e, fma(0.375, e, 0.5), y);
}

__device__ __forceinline__ double rcp_nr(double x) {
    // 1/x: hardware approximation and one third-order step, y (1 + e + e^2), e = 1 - x y
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

__device__ __forceinline__ double rcbrt_nr(double x) {
    // x^(-1/3): float seed 2^(-log2(x)/3), one Newton step z + z e / 3, e = 1 - x z^3
    const double z = (double)sfu_exp2(sfu_log2((float)x) * (-1.0f / 3.0f));
    const double e = fma(-x * z, z * z, 1.0);
    return fma(z * e, 1.0 / 3.0, z);
}

// two steps: the per-entry set-up
__device__ __forceinline__ double rsqrt_nr2(double x) {
    const double y = rsqrt_nr(x);
    return y * fma(-0.5 * x * y, y, 1.5);
}

__device__ __forceinline__ double rcp_nr2(double x) {
    const double y = rcp_nr(x);
    return fma(fma(-x, y, 1.0), y, y);
}

__device__ __forceinline__ double rcbrt_nr2(double x) {
    const double z = rcbrt_nr(x);
    return fma(z * fma(-x * z, z * z, 1.0), 1.0 / 3.0, z);
}
