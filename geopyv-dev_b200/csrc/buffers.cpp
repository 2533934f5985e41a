// buffers.cpp -- the growing device and pinned host buffers of a context.
#include <cuda_runtime.h>

#include <string>

#include "internal.h"

namespace gpv {

int DevBuf::ensure(size_t want) {
    if (want <= bytes && ptr) return GPV_SUCCESS;
    if (ptr) cudaFree(ptr);
    ptr = nullptr;
    bytes = 0;
    const size_t sz = want < 256 ? 256 : want;
    cudaError_t e = cudaMalloc(&ptr, sz);
    if (e != cudaSuccess) {
        ptr = nullptr;
        set_error(std::string("cudaMalloc(") + std::to_string(sz) + "): " + cudaGetErrorString(e));
        return GPV_ERR_NOMEM;
    }
    bytes = sz;
    return GPV_SUCCESS;
}

void DevBuf::release() {
    if (ptr) cudaFree(ptr);
    ptr = nullptr;
    bytes = 0;
}

int HostBuf::ensure(size_t want) {
    if (want <= bytes && ptr) return GPV_SUCCESS;
    if (ptr) cudaFreeHost(ptr);
    ptr = nullptr;
    bytes = 0;
    const size_t sz = want < 4096 ? 4096 : want;
    cudaError_t e = cudaHostAlloc(&ptr, sz, cudaHostAllocDefault);
    if (e != cudaSuccess) {
        ptr = nullptr;
        set_error(std::string("cudaHostAlloc(") + std::to_string(sz) + "): " + cudaGetErrorString(e));
        return GPV_ERR_NOMEM;
    }
    bytes = sz;
    return GPV_SUCCESS;
}

void HostBuf::release() {
    if (ptr) cudaFreeHost(ptr);
    ptr = nullptr;
    bytes = 0;
}

}  // namespace gpv
