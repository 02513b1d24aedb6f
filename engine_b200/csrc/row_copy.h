// What a row-wise fetch of encoded weights copies: plain arithmetic, so that a host program can check it too.
#pragma once

#include <stdint.h>

#if defined(__CUDACC__)
#define RIBN_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define RIBN_HOST_DEVICE inline
#endif

namespace ribn {

// Bulk copies move whole granules of 16 bytes from 16-byte boundaries, and rows of some formats start and end anywhere.  Bytes
// [from, to) of a tensor of `total` bytes come as one copy of `bytes` from `first`, the boundary below, to the boundary above; where
// that boundary lies behind the tensor's end, the last `tail` bytes (at first + bytes) are to be read one by one.
struct RowCopy {
    unsigned long long first;
    uint32_t bytes, tail;
};

RIBN_HOST_DEVICE RowCopy row_copy(unsigned long long from, unsigned long long to, unsigned long long total) {
    const unsigned long long whole = total & ~15ull, end = (to + 15ull) & ~15ull;
    RowCopy copy;
    copy.first = from & ~15ull;
    const unsigned long long copied = end <= whole ? end : whole > copy.first ? whole : copy.first;
    copy.bytes = static_cast<uint32_t>(copied - copy.first);
    copy.tail = to > copied ? static_cast<uint32_t>(to - copied) : 0u;
    return copy;
}

}  // namespace ribn
