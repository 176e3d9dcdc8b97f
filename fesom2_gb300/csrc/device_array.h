// device_array.h -- whether a caller's array lies in one allocation of this device's memory.
#pragma once
#include <cstddef>
#include <cstdint>

#include <cuda.h>
#include <cuda_runtime.h>

namespace fesom {

// whether [base, base + size) holds the `bytes` bytes from p on
inline bool range_holds(uintptr_t base, size_t size, uintptr_t p, size_t bytes) {
    return p >= base && bytes <= size && p - base <= size - bytes;
}

// base and size of the device allocation p lies in; false where the driver knows none
inline bool allocation_of(const void *p, uintptr_t *base, size_t *size) {
    using Fn = CUresult (*)(CUdeviceptr *, size_t *, CUdeviceptr);
    static const Fn fn = [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuMemGetAddressRange", &f, 12000, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            f = nullptr;
        }
        return (Fn)f;
    }();
    CUdeviceptr b = 0;
    if (!fn || fn(&b, size, (CUdeviceptr)(uintptr_t)p) != CUDA_SUCCESS) return false;
    *base = (uintptr_t)b;
    return true;
}

// whether the n elements from p on are this device's memory, all in one allocation, and aligned: a
// kernel then reads or writes the caller's array as it is, and copies to and from it need no staging.
// Anything else (host memory, another device's, an array that ends before its n elements do, wherever
// its computed end then lies) takes the copies, with their errors.
template <typename S>
bool on_device(const S *p, size_t n) {
    int dev = -1;
    if (!p || !n || (uintptr_t)p % sizeof(S) || cudaGetDevice(&dev) != cudaSuccess) return false;
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();  // no memory of CUDA's: not an error here
        return false;
    }
    if (a.type != cudaMemoryTypeDevice || a.device != dev) return false;
    uintptr_t base = 0;
    size_t size = 0;
    return allocation_of(p, &base, &size) && range_holds(base, size, (uintptr_t)p, n * sizeof(S));
}

}  // namespace fesom
