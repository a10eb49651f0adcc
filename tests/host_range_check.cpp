// Prints 1 or 0 for each array of a fake host address space: whether
// locked_whole (ibpm.jl_b200/csrc/host_range.h) hands it to a kernel.  Host code
// only; no address is read.  tests/test_host_ranges.py compiles and runs it.
#include <cstdio>
#include <cstdlib>

#include "host_range.h"

using namespace ibpm;

// argv: ranges as start:size, then "--", then arrays as start:values
int main(int argc, char** argv) {
    HostRange ranges[8];
    int nr = 0, i = 1;
    auto pair = [](const char* s, unsigned long long& a, unsigned long long& b) {
        char* end;
        a = std::strtoull(s, &end, 10);
        b = std::strtoull(end + 1, nullptr, 10);
    };
    unsigned long long a, b;
    for (; i < argc && argv[i][0] != '-' && nr < 8; ++i) {
        pair(argv[i], a, b);
        ranges[nr++] = HostRange{true, (uintptr_t)a, (size_t)b, nullptr};
    }
    auto query = [&](const void* p) -> HostRange {
        const uintptr_t at = reinterpret_cast<uintptr_t>(p);
        for (int r = 0; r < nr; ++r)
            if (at >= ranges[r].start && at - ranges[r].start < ranges[r].size) {
                HostRange h = ranges[r];
                h.dev = const_cast<void*>(p);
                return h;
            }
        return {};
    };
    for (++i; i < argc; ++i) {
        pair(argv[i], a, b);
        std::printf("%d", locked_whole(reinterpret_cast<const double*>((uintptr_t)a), (long long)b, query) != nullptr);
    }
    std::printf("\n");
}
