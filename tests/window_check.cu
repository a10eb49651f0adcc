// Prints 1 or 0 for each pair of floored body coordinates given: whether
// window_inside (ibpm.jl_b200/csrc/ibpm_internal.cuh) takes the window as inside
// a grid of nx × ny cells.  Host code only: it launches nothing and runs without
// a GPU.  tests/test_body_window.py compiles and runs it.
#include <cstdio>
#include <cstdlib>

#include "ibpm_internal.cuh"

int main(int argc, char** argv) {
    const ibpm::Geom g = ibpm::make_geom(std::atoi(argv[1]), std::atoi(argv[2]), 1);
    for (int i = 3; i + 1 < argc; i += 2)
        std::printf("%d", ibpm::window_inside(g, std::strtod(argv[i], nullptr), std::strtod(argv[i + 1], nullptr)));
    std::printf("\n");
}
