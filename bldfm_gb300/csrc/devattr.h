// Once-per-device guard for kernel attributes (cudaFuncSetAttribute applies
// to the current device's context): a call site keeps one flag word and
// sets its attributes when first_on_device() says the current device has not
// seen them yet.  Setting an attribute twice is harmless, so the unguarded
// read-modify-write of the word needs no lock.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

inline bool first_on_device(uint64_t &mask)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return true;
    const uint64_t bit = (uint64_t)1 << dev;
    if (mask & bit) return false;
    mask |= bit;
    return true;
}

// The same for launches that several threads make at once: the device's flag is
// set only when `set` has succeeded, so that a failure is tried again by the
// next launch and no launch goes ahead of the attribute.
template <class F>
inline cudaError_t set_once(std::atomic<uint64_t> &mask, int dev, F set)
{
    const uint64_t bit = dev >= 0 && dev < 64 ? (uint64_t)1 << dev : 0;
    if (mask.load(std::memory_order_acquire) & bit) return cudaSuccess;
    const cudaError_t e = set();
    if (e == cudaSuccess) mask.fetch_or(bit, std::memory_order_release);
    return e;
}

template <class K>
inline cudaError_t set_dynamic_smem(std::atomic<uint64_t> &mask, K kernel, size_t bytes)
{
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess)
        e = set_once(mask, dev, [&] {
            return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        });
    if (e != cudaSuccess) (void)cudaGetLastError();  // reported here, not by the next launch as well
    return e;
}
