// exp(M) phi per walker in FP64 as one kernel (see taylor_f64.cu).
#pragma once
#include "common.cuh"

struct TaylorF64 {
    int n = 0, N = 0, W = 0;           // walkers are n x N, wsize = n N
    const zd *M = nullptr;             // n x n per walker (Mstride apart; 0: shared)
    long long Mstride = 0;
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

// Whether the kernel takes this shape.
bool taylor_f64_supported(int n, int N);
cudaError_t taylor_f64(const TaylorF64 &a, cudaStream_t s);
