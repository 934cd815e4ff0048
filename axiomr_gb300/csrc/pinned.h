// Whether the GPU may read a host array in place: decided by address ranges alone, so that the rule
// can be checked without a GPU (the queries are the caller's).
#pragma once
#include <stddef.h>
#include <stdint.h>

namespace axr {

// What is known of a host pointer: `device` is its address on the device (0: not pinned, or not
// mapped), [start, start + size) the device addresses of the one allocation or registration it lies in
// (size 0: unknown).
struct PinnedRange {
    uint64_t device;
    uint64_t start, size;
};

// The device address of `bytes` bytes at host address `host`, if a kernel may read all of them with
// 16-byte loads: both addresses 16-byte aligned, and every byte inside the range that holds the first. A
// program may have registered only the front of its array; past the registration there is nothing on the
// device to read. 0 otherwise (the array is copied).
inline uint64_t readable_in_place(uint64_t host, uint64_t bytes, const PinnedRange& r) {
    if (!r.device || ((host | r.device) & 15u)) return 0;
    if (r.device < r.start || r.device - r.start > r.size || bytes > r.size - (r.device - r.start)) return 0;
    return r.device;
}

}  // namespace axr
