// Dynamic shared memory of kernels that need more than 48 KB.
#pragma once
#include <cuda_runtime.h>

#include <map>
#include <mutex>
#include <utility>

namespace b200 {

// Lets `kern` be launched with as much dynamic shared memory as the current device offers beside its static
// share; done once per kernel and device.  The limit is a property of the function on the device, not of a
// launch: were it set to each call's own size, a thread searching another index could lower it between this
// thread's setting and its launch, which then fails.  It is a permission only: what a launch takes, and how
// many blocks share an SM, follows from the launch's own size.
inline cudaError_t allow_max_smem(const void* kern) {
    static std::mutex mu;
    static std::map<std::pair<const void*, int>, bool> done;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> l(mu);
    bool& ready = done[{kern, dev}];
    if (ready) return cudaSuccess;
    int most = 0;
    e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e != cudaSuccess) return e;
    cudaFuncAttributes fa;
    e = cudaFuncGetAttributes(&fa, kern);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, most - static_cast<int>(fa.sharedSizeBytes));
    ready = e == cudaSuccess;
    return e;
}
template <typename... Args>
cudaError_t allow_max_smem(void (*kern)(Args...)) {
    return allow_max_smem(reinterpret_cast<const void*>(kern));
}

}  // namespace b200
