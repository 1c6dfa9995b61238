// Owned memory: device buffers, and pinned host memory that kernels write.
#pragma once

#include "../../include/gpe_b200.h"
#include "plan.hpp"

#include <cuda_runtime.h>

#include <string>

namespace gpe {

#define GPE_CUDA(call)                                                                             \
    do {                                                                                           \
        cudaError_t e_ = (call);                                                                   \
        if (e_ != cudaSuccess)                                                                     \
            throw Error(e_ == cudaErrorMemoryAllocation ? GPE_ERR_NOMEM : GPE_ERR_CUDA,            \
                        std::string(#call) + ": " + cudaGetErrorString(e_));                      \
    } while (0)

template <class T> struct DevBuf {
    T *p     = nullptr;
    size_t n = 0;
    void alloc(size_t count) {
        n = count;
        GPE_CUDA(cudaMalloc(&p, sizeof(T) * (count ? count : 1)));
        GPE_CUDA(cudaMemset(p, 0, sizeof(T) * (count ? count : 1)));
    }
    ~DevBuf() {
        if (p)
            cudaFree(p);
    }
};

// Pinned host memory that kernels write (h and p are the same memory, host and device
// address): results the host reads after a stream synchronisation, without a copy of
// their own.
template <class T> struct MappedBuf {
    T *h     = nullptr;
    T *p     = nullptr;
    size_t n = 0;
    void alloc(size_t count) {
        if (h)
            cudaFreeHost(h);
        h = p = nullptr;
        n = 0; // until there is memory again: the allocation may fail
        GPE_CUDA(cudaHostAlloc(&h, sizeof(T) * count, cudaHostAllocMapped | cudaHostAllocPortable));
        GPE_CUDA(cudaHostGetDevicePointer(&p, h, 0));
        n = count;
        clear();
    }
    void clear() {
        for (size_t i = 0; i < n; ++i)
            ((volatile T *)h)[i] = T(0);
    }
    T operator[](size_t i) const { return ((const volatile T *)h)[i]; }
    ~MappedBuf() {
        if (h)
            cudaFreeHost(h);
    }
};

} // namespace gpe
