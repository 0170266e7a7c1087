// dev_buf.h -- the owning device buffer every handle is made of (host code).
#pragma once

#include <cuda_runtime_api.h>

#include <cstddef>
#include <utility>

namespace crt {

// Owning device buffer.  After a failed allocation it is empty (and no error
// stays pending for a later call to find), so the caller may free memory and ask
// again.
struct DevBuf {
    void* p = nullptr;
    size_t bytes = 0;
    ~DevBuf() { if (p) cudaFree(p); }
    cudaError_t alloc(size_t n) {
        if (p) cudaFree(p);
        p = nullptr;
        bytes = 0;
        if (!n) return cudaSuccess;
        const cudaError_t e = cudaMalloc(&p, n);
        if (e == cudaSuccess) {
            bytes = n;
        } else {
            p = nullptr;
            if (e == cudaErrorMemoryAllocation) cudaGetLastError();
        }
        return e;
    }
    // Room for at least n bytes; the contents do not survive growing.
    cudaError_t reserve(size_t n) { return bytes < n ? alloc(n) : cudaSuccess; }
    template <typename T> T* as() const { return static_cast<T*>(p); }
    void swap(DevBuf& o) {
        std::swap(p, o.p);
        std::swap(bytes, o.bytes);
    }
};

}  // namespace crt
