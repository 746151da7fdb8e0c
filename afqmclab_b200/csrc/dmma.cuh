// The FP64 matrix instruction and the asynchronous element copies that feed
// it, shared by the FP64 kernels (zgemm.cu, taylor_f64.cu).
#pragma once
#include "common.cuh"

// c += a b on an 8 x 8 block of C with 4 contraction indices.  Lane t holds
// a = A(t / 4, t % 4), b = B(t % 4, t / 4), c = C(t / 4, 2 (t % 4) + {0, 1}).
__device__ __forceinline__ void dmma(double &c0, double &c1, double a, double b)
{
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
                 : "+d"(c0), "+d"(c1)
                 : "d"(a), "d"(b));
}

// asynchronous copy of one element (16 bytes complex, 8 bytes real) into
// shared memory; an element outside the operand is filled with zeros
template <int BYTES>
__device__ __forceinline__ void cp_async_elem(unsigned dst, const void *src, bool valid)
{
    const int n = valid ? BYTES : 0;
    if (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(n) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait()
{
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}
