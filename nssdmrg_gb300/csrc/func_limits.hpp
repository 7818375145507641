// Launch limits of kernels, raised per device.
#pragma once

#include <cuda_runtime_api.h>

#include <cstddef>
#include <map>
#include <mutex>
#include <tuple>

namespace nss {

// Raise `attr` of a kernel on the current device to at least `value`.  The
// attribute belongs to the kernel on one device, shared by every context of the
// process there, so it only ever grows (a context sized for a smaller basis must
// not take the room a larger one was set up with) and is kept per device (a
// context on another one has to raise it again).
inline cudaError_t raise_attribute(const void *fn, cudaFuncAttribute attr, int value) {
    static std::mutex mu;
    static std::map<std::tuple<int, const void *, int>, int> done;
    int dev = 0;
    if (const cudaError_t e = cudaGetDevice(&dev)) return e;
    std::lock_guard<std::mutex> lk(mu);
    int &cur = done[std::make_tuple(dev, fn, (int)attr)];
    if (value <= cur) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(fn, attr, value);
    if (e == cudaSuccess) cur = value;
    return e;
}

// dynamic shared memory beyond the 48 KB that need no opt-in
inline cudaError_t allow_smem(const void *fn, std::size_t bytes) {
    if (bytes <= 48 * 1024) return cudaSuccess;
    return raise_attribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

}  // namespace nss
