// Whether a caller's memory may be copied by a kernel of the calling thread.
#pragma once

#include <cuda_runtime_api.h>

#include <cstddef>
#include <cstdint>

namespace flamegpu {
namespace detail {

// Whether [p, p + bytes) is memory of `device`, the calling thread's current
// one, inside one allocation, on a 16-byte boundary: what a kernel may copy in
// place of the driver, which looks at the range itself and takes a stream of
// any device (a kernel is only launched on the current device's).
inline bool device_range(const void* p, size_t bytes, int device) {
    using RangeOf = int (*)(unsigned long long* base, size_t* size, unsigned long long p);  // cuMemGetAddressRange
    static const RangeOf range_of = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult r;
        if (cudaGetDriverEntryPointByVersion("cuMemGetAddressRange", &f, 12000, cudaEnableDefault, &r) != cudaSuccess) {
            cudaGetLastError();
            f = nullptr;
        }
        return reinterpret_cast<RangeOf>(f);
    }();
    if (!p || !range_of || (reinterpret_cast<uintptr_t>(p) & 15)) return false;
    int current = -1;
    if (cudaGetDevice(&current) != cudaSuccess || current != device) return false;
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    if (a.type != cudaMemoryTypeDevice || a.device != device) return false;
    unsigned long long base = 0;
    size_t size = 0;
    const unsigned long long at = reinterpret_cast<uintptr_t>(p);
    if (range_of(&base, &size, at) != 0) return false;
    return at >= base && at - base <= size && bytes <= size - (at - base);
}

}  // namespace detail
}  // namespace flamegpu
