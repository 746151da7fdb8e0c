// Device helpers shared by the LU kernels (walker_kernels.cu, lu_block.cu).
#pragma once
#include <math_constants.h>

#include "walker_kernels.cuh"

// A 32-bit rank for the pivot search, one warp reduction wide: the leading 25
// bits of |re| + |im| (11 of exponent, 14 of mantissa; NaN ranks as infinity),
// then the lower position.  Ineligible rows rank 0.  Where a row ties with the
// chosen one in the leading bits (lb_rival), which the kernels test beside other
// work, the choice is made again by all 64 bits (lb_exact).
__device__ __forceinline__ unsigned lb_rank(zd a, int pos, bool eligible)
{
    const unsigned hi = min((unsigned)__double2hiint(zcabs1(a)) & 0x7fffffffu, 0x7ff00000u);   // a NaN as infinity
    return eligible ? (((hi >> 6) + 1u) << 7) | (unsigned)(127 - pos) : 0u;
}

__device__ __forceinline__ bool lb_tied(unsigned u, unsigned v) { return (u >> 7) == (v >> 7); }
// Whether a row of rank u ties with the chosen one of rank `best` (and is not it).
__device__ __forceinline__ bool lb_rival(unsigned u, unsigned best) { return (u ^ best) - 1u < 127u; }

// The bits of |re| + |im|, monotonic in the value; NaN as infinity.
__device__ __forceinline__ unsigned long long lb_bits(zd a)
{
    const unsigned long long v = (unsigned long long)__double_as_longlong(zcabs1(a));
    return min(v, 0x7ff0000000000000ull);
}

// The rank of the warp's pivot among the ties with `best` by zgetf2's rule: the
// first position of the largest |re| + |im|.  u: this lane's lb_rank of a.
__device__ __forceinline__ unsigned lb_exact(zd a, unsigned u, unsigned best)
{
    const unsigned long long v = lb_bits(a);
    bool in = lb_tied(u, best);
    const unsigned hi = in ? (unsigned)(v >> 32) : 0u;
    const unsigned mhi = __reduce_max_sync(0xffffffffu, hi);
    in = in && hi == mhi;
    const unsigned lo = in ? (unsigned)v : 0u;
    const unsigned mlo = __reduce_max_sync(0xffffffffu, lo);
    in = in && lo == mlo;
    return __reduce_max_sync(0xffffffffu, in ? u : 0u);
}

// 1 / b: conj(b) / |b|^2 with the reciprocal of d = |b|^2 from the hardware's
// approximation (20 bits) and two Newton-Raphson steps.  Good while d is
// within 1e-280 .. 1e280; lb_rcp_any covers the rest (zero gives zero).
__device__ __forceinline__ zd lb_rcp(zd b, double &d)
{
    d = fma(b.x, b.x, b.y * b.y);
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
    y = fma(y, fma(-d, y, 1.0), y);
    y = fma(y, fma(-d, y, 1.0), y);
    return make_double2(b.x * y, -b.y * y);
}
static __device__ __noinline__ zd lb_rcp_any(zd b)
{
    return zeq0(b) ? make_double2(0.0, 0.0) : zdiv(make_double2(1.0, 0.0), b);
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
