// One-time set-up per device.
//
// Kernel attributes such as the dynamic shared-memory limit belong to the
// context of the device that is current when they are set, so a process that
// launches on several devices has to set them on each one.  first_on_device
// returns true the first time it is called for `flags` with a given device
// current (devices 0..63), false afterwards.
//
// each_device_once runs `set` until it has succeeded once on the current
// device; a second thread that arrives meanwhile runs it too, so nobody
// launches before the attribute is set.
#pragma once
#include <atomic>
#include <cuda_runtime.h>

inline bool first_on_device(std::atomic<unsigned long long> &flags)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return true;
    const unsigned long long bit = 1ull << dev;
    return (flags.fetch_or(bit) & bit) == 0;
}

template <class F>
inline cudaError_t each_device_once(std::atomic<unsigned long long> &flags, F set)
{
    int dev = 0;
    cudaError_t r = cudaGetDevice(&dev);
    if (r != cudaSuccess) return r;
    const unsigned long long bit = dev >= 0 && dev < 64 ? 1ull << dev : 0ull;
    if (bit && (flags.load() & bit)) return cudaSuccess;
    r = set();
    if (r == cudaSuccess) flags.fetch_or(bit);
    return r;
}
