// The owning device buffer on a fake allocator that runs out when told to: a
// failed allocation leaves an empty buffer, so that the next request for the
// same room asks again instead of handing out a null pointer.
#include <cstdio>
#include <cstdlib>

#include "../../cudart_gb300/csrc/dev_buf.h"

static int asked = 0, freed = 0, live = 0;
static cudaError_t pending = cudaSuccess;
static bool full = false;

extern "C" cudaError_t cudaMalloc(void** p, size_t n) {
    ++asked;
    if (full) return pending = cudaErrorMemoryAllocation;   // *p stays as it was
    *p = std::malloc(n);
    ++live;
    return cudaSuccess;
}
extern "C" cudaError_t cudaGetLastError() {
    const cudaError_t e = pending;
    pending = cudaSuccess;
    return e;
}
extern "C" cudaError_t cudaFree(void* p) {
    ++freed;
    --live;
    std::free(p);
    return cudaSuccess;
}

#define CHECK(c) \
    do { \
        if (!(c)) return std::printf("line %d: %s\n", __LINE__, #c), 1; \
    } while (0)

int main() {
    {
        crt::DevBuf b;
        full = true;
        CHECK(b.reserve(100) == cudaErrorMemoryAllocation && b.p == nullptr && b.bytes == 0 && pending == cudaSuccess);
        CHECK(b.reserve(100) == cudaErrorMemoryAllocation && asked == 2);   // asks again
        full = false;
        CHECK(b.reserve(100) == cudaSuccess && b.p != nullptr && b.bytes == 100);
        CHECK(b.reserve(60) == cudaSuccess && asked == 3 && freed == 0);    // room enough
        full = true;                                                        // growing fails: the old room is given back
        CHECK(b.reserve(200) == cudaErrorMemoryAllocation && b.p == nullptr && b.bytes == 0 && freed == 1);
        CHECK(b.reserve(60) == cudaErrorMemoryAllocation && asked == 5);
        full = false;
        CHECK(b.reserve(60) == cudaSuccess && b.bytes == 60);
        CHECK(b.alloc(0) == cudaSuccess && b.p == nullptr && b.bytes == 0 && live == 0);
        CHECK(b.alloc(8) == cudaSuccess && b.bytes == 8);
        crt::DevBuf o;
        b.swap(o);
        CHECK(b.p == nullptr && b.bytes == 0 && o.bytes == 8);
    }
    CHECK(live == 0);
    std::printf("ok\n");
    return 0;
}
