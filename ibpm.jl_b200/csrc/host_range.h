// Whether a host array may be read or written by a kernel.
#pragma once

#include <cstddef>
#include <cstdint>

namespace ibpm {

// What is known of a host address: page-locked, the page-locked range it lies in
// (one allocation or one registration) and its device address.
struct HostRange {
    bool locked;
    uintptr_t start;
    size_t size;
    void* dev;
};

// The device address of n values at `host` if all of them lie in one page-locked
// range, else null.  Both ends page-locked is not enough: an array may begin in
// one registration and end in another with pages between that no kernel may
// touch.  `query` gives the HostRange of an address.
template <class Query>
double* locked_whole(const double* host, long long n, Query query) {
    const uintptr_t p = reinterpret_cast<uintptr_t>(host);
    if (n < 1 || p % sizeof(double)) return nullptr;
    const HostRange r = query(host);
    if (!r.locked || !r.dev || p < r.start || p - r.start > r.size) return nullptr;
    return (size_t)n <= (r.size - (p - r.start)) / sizeof(double) ? static_cast<double*>(r.dev) : nullptr;
}

}  // namespace ibpm
