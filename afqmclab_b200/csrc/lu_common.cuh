// Device helpers shared by the LU kernels (walker_kernels.cu, lu_block.cu).
#pragma once
#include <math_constants.h>

#include "walker_kernels.cuh"

// A rank that orders candidates like the pivot search: for values >= +0 the
// IEEE bits are monotonic; NaN ranks as infinity; ineligible rows rank 0.
__device__ __forceinline__ unsigned long long gr_rank(zd a0, bool eligible)
{
    double v = zcabs1(a0);
    if (!(v == v)) v = CUDART_INF;
    return eligible ? (unsigned long long)__double_as_longlong(v) + 1ull : 0ull;
}

// 1 / b without a division, so that it schedules between other arithmetic:
// b is scaled by a power of two (exact) so that max(|re|, |im|) lies in
// [1, 2), the real reciprocal y of d = |b|^2 in [1, 8) starts from the
// single-precision approximation and takes two Newton-Raphson steps
// y <- y + y (1 - d y), each of which doubles the correct bits (about 21 ->
// 42 -> full precision), and 1/b = s conj(b s) y.  Within a few ulp of the
// rounded quotient; a NaN or infinite b gives NaN (callers test zero first).
__device__ __forceinline__ zd zrcp_nr(zd b)
{
    const double m = fmax(fabs(b.x), fabs(b.y));
    const long long e = (__double_as_longlong(m) >> 52) & 0x7ff;
    const double s = __longlong_as_double((2046 - e) << 52);   // 2^(1023 - e)
    const double xs = b.x * s, ys = b.y * s;
    const double d = fma(xs, xs, ys * ys);
    double y = (double)__fdividef(1.0f, (float)d);
    y = fma(y, fma(-d, y, 1.0), y);
    y = fma(y, fma(-d, y, 1.0), y);
    const double t = y * s;
    return make_double2(xs * t, -ys * t);
}

// Position of the warp's best candidate: largest rank, then lowest position.
__device__ __forceinline__ int gr_warp_best(unsigned long long u, int pos)
{
    const unsigned hi = (unsigned)(u >> 32), lo = (unsigned)u;
    const unsigned mhi = __reduce_max_sync(0xffffffffu, hi);
    const unsigned mlo = __reduce_max_sync(0xffffffffu, hi == mhi ? lo : 0u);
    const unsigned key = (hi == mhi && lo == mlo) ? (unsigned)pos : 0xffffffffu;
    return (int)__reduce_min_sync(0xffffffffu, key);
}

// Per-walker finish of the block log-determinants: the overlap's log and,
// by mode, the constraint or the population weight.  ldB/sgB hold the
// walker's nb block log-determinants and singular flags.
__device__ __forceinline__ void lu_walker_finish(int w, bool act, int nb, int mult, const zd *ldB, const int *sgB,
                                 const zd *logw, zd logwAdd, zd logwT, zd *logov, int *alive, int *surv,
                                 zd *logwOut, double *weight, int *status, int mode)
{
    if (!act) {
        if (mode == LU_PROJECT) surv[w] = 0;
        if (mode == LU_POPWEIGHT) { weight[w] = 0.0; alive[w] = 1; }
        return;
    }
    bool singular = false;
    zd logdetSum = make_double2(0.0, 0.0);
    // a singular block adds lognorm -1e300 with phase 1
    // (lognormPhaseDeterminant, tensor_2d_common_fun.cpp:75-84)
    for (int t = 0; t < nb; ++t) {
        const bool sb = sgB[t] != 0;
        singular = singular || sb;
        logdetSum = zadd(logdetSum, sb ? make_double2(-1e300, 0.0) : ldB[t]);
    }
    const zd lwR = zadd(logwAdd, logw[w]);
    if (mult == 2) logdetSum = zadd(logdetSum, logdetSum);
    const zd lo = zadd(zadd(zconj(logwT), lwR), logdetSum);
    logov[w] = lo;
    if (singular && status) atomicOr(status + w, (int)ST_SINGULAR);
    if (!(isfinite(lo.x) && isfinite(lo.y)) && status && !singular) atomicOr(status + w, (int)ST_NONFINITE);
    if (mode == LU_PROJECT) {
        const double ph = lo.y;
        const double c = cos(ph);
        if (c <= 0.0) {
            alive[w] = 0; surv[w] = 0;
        } else {
            logwOut[w] = zadd(logw[w], make_double2(log(c), -ph));
            surv[w] = 1;
        }
    } else if (mode == LU_POPWEIGHT) {
        const zd e = zexp(lo);
        if (e.x <= 0.0) {
            weight[w] = 0.0;
        } else {
            weight[w] = e.x;
            logwOut[w] = zsub(logw[w], lo);
        }
        alive[w] = 1;
    }
}
