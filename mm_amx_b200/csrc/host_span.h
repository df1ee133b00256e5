// Whether kernels may read or write a piece of host memory where it is.  Plain C++: the driver's answers come in as a function.
#pragma once
#include <cstddef>
#include <cstdint>

namespace b200fc {

// What the driver knows of a host address: pinned (page-locked, not managed), the device's address of it, and the range of device addresses
// of the one allocation or registration that it lies in, with the device's rights there.
struct HostRange {
    bool pinned, readable, writable;
    uintptr_t device, start;
    size_t size;
};

// The device's address of [p, p + bytes), or 0 where the copy engines must take it: memory that is not pinned, whose pages belong to more
// than one registration (what lies between two may be anything) or that may not be written, and rows that are not 16-byte aligned.
template <class Query>
uintptr_t span_on_device(const void* p, int64_t ld, size_t bytes, bool write, const Query& query) {
    if ((((uintptr_t)p | (uintptr_t)ld) & 15) != 0 || bytes == 0) return 0;
    HostRange r = {};
    if (!query(p, &r) || !r.pinned || !r.readable || (write && !r.writable)) return 0;
    if (r.device == 0 || (r.device & 15) != 0 || r.device < r.start) return 0;
    const size_t offset = r.device - r.start;
    return offset <= r.size && bytes <= r.size - offset ? r.device : 0;
}

}  // namespace b200fc
