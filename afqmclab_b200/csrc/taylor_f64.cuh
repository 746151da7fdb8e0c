// exp(M) phi per walker in FP64 as one kernel (see taylor_f64.cu).
#pragma once
#include "common.cuh"

struct TaylorF64 {
    int n = 0, N = 0, W = 0;           // walkers are n x N, wsize = n N
    const zd *M = nullptr;             // n x n per walker (Mstride apart; 0: shared)
    long long Mstride = 0;
    bool packed = false;               // M symmetric, stored in panels (taylor_panel_at)
    const zd *src = nullptr;
    zd *dst = nullptr;                 // may be src
    const int *mask = nullptr;         // walkers with mask[w] == 0 are left alone
    int *order = nullptr, *status = nullptr;
    int kmax = 0, checkFrom = 0;       // series cap; first order at which convergence is tested
    double acc = 0.0;                  // converged when max |term| <= acc
    // dst = post * exp(M) src where given: an n x n matrix, complex or real
    const zd *postZ = nullptr;
    const double *postR = nullptr;
};

// Panel storage of a symmetric n x n matrix: 8 columns per panel, each with
// the rows from the panel's first one down to n rounded up to a multiple of 8
// (entries beyond n are zero).  Entry (r, c) with r >= c rounded down to its
// panel's start; taylor_panel_size entries in all.
HD long long taylor_panel_at(long long n, long long r, long long c)
{
    const long long n8 = (n + 7) / 8 * 8, c0 = c / 8 * 8;
    return c0 * n8 - c0 * (c0 - 8) / 2 + (c - c0) * (n8 - c0) + (r - c0);
}
HD long long taylor_panel_size(long long n)
{
    const long long n8 = (n + 7) / 8 * 8;
    return n8 * n8 - n8 * (n8 - 8) / 2;
}

// Whether the kernel takes this shape.
bool taylor_f64_supported(int n, int N);
cudaError_t taylor_f64(const TaylorF64 &a, cudaStream_t s);
