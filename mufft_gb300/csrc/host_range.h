// Extents of page-locked host ranges, and the buffers that kernels take in place.
#pragma once

#include <stddef.h>
#include <stdint.h>

namespace mgb {

// Whether the range of `size` bytes at `start` holds the `bytes` bytes from p on.
inline bool range_holds(uintptr_t start, size_t size, uintptr_t p, size_t bytes)
{
    return p >= start && p - start <= size && bytes <= size - (p - start);
}

// Largest buffer of transforms of M complex points that a one-pass execute lets
// the kernel take over the link (real: an r2c or c2r transform).  Staged ->
// direct, us per execute at 1 MiB each way: c2c 1024 34.3 -> 19.3, 64 34.3 ->
// 22.8, 4 34.0 -> 18.7.  Threads that hold a whole row of 8 or 16 points, or half
// a row of 32, read the link in pieces too small for it: c2c of 16 points 26.8 ->
// 22.3 at 256 KiB but 29.1 -> 33.4 at 512 KiB, of 32 28.9 -> 23.1 at 512 KiB but
// 34.2 -> 35.4 at 1 MiB; r2c of 16 reals (8 points) 26.7 -> 24.5 at 256 KiB but 28.8
// -> 32.4 at 512 KiB, of 64 29.3 -> 26.4 at 512 KiB but 34.6 -> 43.1 at 1 MiB.
inline size_t direct_host_bytes(unsigned M, bool real)
{
    if (M == 32)
        return (size_t)512 << 10;
    if (M == 16 || (real && M == 8))
        return (size_t)256 << 10;
    return (size_t)1 << 20;
}

}  // namespace mgb
