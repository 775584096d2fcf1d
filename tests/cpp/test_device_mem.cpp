// Memory helpers when an allocation fails, with a CUDA runtime of this file's own (host memory): a buffer
// whose growth failed is empty, and asking it for less afterwards allocates again.
#include "../../indexsdk_b200/csrc/device_mem.h"

#include <cstdio>
#include <cstdlib>

static bool fail_next = false;
static cudaError_t take(void** p, size_t n) {
    if (fail_next) {
        fail_next = false;
        return cudaErrorMemoryAllocation;
    }
    *p = std::malloc(n);
    return cudaSuccess;
}
extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) { return take(p, n); }
cudaError_t cudaMallocHost(void** p, size_t n) { return take(p, n); }
cudaError_t cudaFree(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "no memory"; }
}

static int failed = 0;
static void check(bool ok, const char* what) {
    if (!ok) {
        std::printf("FAILED: %s\n", what);
        ++failed;
    }
}

template <typename Buffer>
static void growth_fails(const char* name) {
    Buffer b;
    std::memset(b.ensure(1000), 1, 1000);
    fail_next = true;
    bool thrown = false;
    try {
        b.ensure(100000);
    } catch (const std::exception&) {
        thrown = true;
    }
    check(thrown, name);
    void* p = b.ensure(1000);
    check(p != nullptr, name);
    if (p) std::memset(p, 2, 1000);
}

int main() {
    growth_fails<b200::DeviceBuffer>("DeviceBuffer");
    growth_fails<b200::PinnedBuffer>("PinnedBuffer");
    b200::DeviceBuffer kept;
    std::memset(kept.grow_keep(1000, 0, nullptr), 3, 1000);
    fail_next = true;
    bool thrown = false;
    try {
        kept.grow_keep(100000, 1000, nullptr);
    } catch (const std::exception&) {
        thrown = true;
    }
    check(thrown && kept.get() && kept.as<char>()[999] == 3, "grow_keep leaves what was there");
    std::printf("%d failed\n", failed);
    return failed != 0;
}
