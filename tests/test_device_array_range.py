"""Which of a caller's arrays a kernel may read or write as they are (device_array.h), on stand-ins for
the driver's answers: two device allocations with a gap, host memory, another device's allocation.  An
array that ends before its n elements do is left to the copies, which refuse it, also where its computed
end lies in the next allocation."""
from tests import host_cpp

SOURCE = r"""
#include <cstdio>
#include <cstring>
#include "device_array.h"

struct Block { uintptr_t base; size_t size; int type, device; };
static const Block blocks[] = {{0x1000, 0x1000, cudaMemoryTypeDevice, 0}, {0x2800, 0x4000, cudaMemoryTypeDevice, 0},
                               {0x6800, 0x1000, cudaMemoryTypeDevice, 0}, {0x9000, 0x1000, cudaMemoryTypeHost, 0},
                               {0xb000, 0x1000, cudaMemoryTypeDevice, 1}, {0xd000, 0x1000, cudaMemoryTypeManaged, 0}};
static const Block *at(uintptr_t p) {
    for (const Block &b : blocks)
        if (p >= b.base && p - b.base < b.size) return &b;
    return nullptr;
}
static CUresult range(CUdeviceptr *base, size_t *size, CUdeviceptr p) {
    const Block *b = at((uintptr_t)p);
    if (!b) return CUDA_ERROR_NOT_FOUND;
    *base = b->base;
    *size = b->size;
    return CUDA_SUCCESS;
}
extern "C" {
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p) {
    const Block *b = at((uintptr_t)p);
    std::memset(a, 0, sizeof *a);
    a->type = b ? (cudaMemoryType)b->type : cudaMemoryTypeUnregistered;
    a->device = b ? b->device : -1;
    return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPointByVersion(const char *, void **f, unsigned int, unsigned long long,
                                             cudaDriverEntryPointQueryResult *q) {
    *f = (void *)range;
    if (q) *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
}
static int bad = 0;
static void check(const char *what, bool got, bool want) {
    if (got != want) { std::printf("%s: %d\n", what, (int)got); bad++; }
}
int main() {
    using fesom::on_device;
    auto f = [](uintptr_t p) { return (const float *)p; };
    auto d = [](uintptr_t p) { return (const double *)p; };
    check("a whole allocation", on_device(f(0x1000), 0x400), true);
    check("its tail", on_device(d(0x1ff8), 1), true);
    check("a part, off 16 bytes", on_device(f(0x1004), 0x3ff), true);
    check("one element too many", on_device(f(0x1000), 0x401), false);
    check("ends in the next allocation, over a gap", on_device(f(0x1000), 0x700), false);
    check("ends in an allocation right behind", on_device(d(0x2800), 0x840), false);
    check("far past its end", on_device(d(0x2800), (size_t)1 << 60), false);
    check("misaligned", on_device(d(0x1004), 4), false);
    check("host memory", on_device(d(0x9000), 4), false);
    check("another device", on_device(d(0xb000), 4), false);
    check("managed memory", on_device(d(0xd000), 4), false);
    check("no allocation", on_device(d(0x100), 4), false);
    check("null", on_device((const double *)nullptr, 4), false);
    check("empty", on_device(d(0x1000), 0), false);
    return bad;
}
"""


def test_arrays_taken_as_they_are(tmp_path):
    host_cpp.run(tmp_path, SOURCE)
