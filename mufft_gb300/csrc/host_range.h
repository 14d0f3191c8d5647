// Extents of page-locked host ranges.
#pragma once

#include <stddef.h>
#include <stdint.h>

namespace mgb {

// Whether the range of `size` bytes at `start` holds the `bytes` bytes from p on.
inline bool range_holds(uintptr_t start, size_t size, uintptr_t p, size_t bytes)
{
    return p >= start && p - start <= size && bytes <= size - (p - start);
}

}  // namespace mgb
