// Blocked Gauss-Jordan of the overlap blocks on the FP64 matrix instruction
// (see lu_block.cu); same arguments as launch_lu_logdet_inverse32.
#pragma once
#include "walker_kernels.cuh"

// One block of up to 128 columns, or two of up to 64.
bool lu_block_supported(const Blocks &bl);
cudaError_t lu_block(int W, const Blocks &bl, const zd *S, zd *Sinv, float *Sinv32, const int *active, const zd *logw,
                     zd logwAdd, zd logwT, zd *logov, int *alive, int *surv, zd *logwOut, double *weight, int *status,
                     int mode, bool wantInverse, cudaStream_t s);
