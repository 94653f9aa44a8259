// How a caller's host array is read or written: by a kernel, where the GPU
// reaches pageable host memory through the host's page tables, or by copies.
#pragma once

#include <cstdint>

namespace hbt {

enum class HostRoute { kCopies = 1, kKernel = 2 };

// Route of an array of doubles.  The kernels load and store 8 bytes at a time,
// which faults at other addresses than multiples of 8; copies take any.
inline HostRoute host_route(const void *p) {
    return reinterpret_cast<uintptr_t>(p) % 8 == 0 ? HostRoute::kKernel : HostRoute::kCopies;
}

}  // namespace hbt
