"""Which host arrays a state transfer hands to a kernel (locked_whole,
ibpm.jl_b200/csrc/host_range.h), on the CPU with a fake address space: only an
array that lies whole in one page-locked range.  One that begins in a range and
ends in another with a gap between, or beside it, is copied instead; so is one
that ends past its range, begins outside, or is not aligned to its values."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CXX = shutil.which("g++")


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    if CXX is None:
        pytest.skip("no g++")
    exe = str(tmp_path_factory.mktemp("ranges") / "host_range_check")
    subprocess.run([CXX, "-std=c++17", "-I", os.path.join(ROOT, "ibpm.jl_b200", "csrc"),
                    os.path.join(ROOT, "tests", "host_range_check.cpp"), "-o", exe], check=True)

    def run(ranges, arrays):
        out = subprocess.run([exe, *("%d:%d" % r for r in ranges), "--", *("%d:%d" % a for a in arrays)],
                             check=True, capture_output=True, text=True).stdout.strip()
        return [c == "1" for c in out]
    return run


PAGE = 4096


@pytest.mark.parametrize("ranges,array,whole", [
    ([(PAGE, 4 * PAGE)], (PAGE, 4 * PAGE // 8), True),                      # exactly the range
    ([(PAGE, 4 * PAGE)], (2 * PAGE, PAGE // 8), True),                      # inside
    ([(PAGE, 4 * PAGE)], (5 * PAGE - 8, 1), True),                          # its last value
    ([(PAGE, 4 * PAGE)], (PAGE, 4 * PAGE // 8 + 1), False),                 # one value past the end
    ([(PAGE, 4 * PAGE)], (PAGE - 8, 8), False),                             # one value before it
    ([(PAGE, PAGE), (3 * PAGE, PAGE)], (PAGE, 3 * PAGE // 8), False),       # both ends locked, a gap between
    ([(PAGE, PAGE), (2 * PAGE, PAGE)], (PAGE, 2 * PAGE // 8), False),       # two ranges side by side
    ([(PAGE, 4 * PAGE)], (PAGE + 4, 8), False),                             # not aligned
    ([(PAGE, PAGE - 4)], (PAGE, PAGE // 8), False),                         # the range ends inside the last value
    ([], (PAGE, 8), False),                                                 # pageable
    ([(PAGE, PAGE)], (PAGE, 0), False),                                     # no values
])
def test_only_whole_arrays_of_one_range(check, ranges, array, whole):
    assert check(ranges, [array]) == [whole]


@pytest.mark.gpu
def test_arrays_inside_registered_memory():
    """A state read into one registration of ordinary memory (page-locked after
    it was allocated), and into the two registrations beside each other."""
    import numpy as np
    import torch

    import ibpm_gpu as G
    g = G.make_grid(1.0 / 16, (-2.0, 2.0, -2.0, 2.0), 2)
    p = G.IBProblem(g, [G.make_cylinder(0.5, g.h, 0.01, 0.02, n=12)], 0.01, 50.0, freestream=(1.0, 0.3, 0.0))
    src = G.IBState(p)
    rng = np.random.default_rng(8)
    src.Gamma[...] = rng.standard_normal(src.Gamma.shape)
    src.q[...] = rng.standard_normal(src.q.shape)
    G.push_state(src, p, fields=("Gamma", "q"))
    nG, nq = src.Gamma.size, src.q.size
    block = np.zeros((8 * (nG + nq) + 4 * PAGE) // 8)
    first = -block.ctypes.data % PAGE                        # bytes to the first whole page
    gb = -(-8 * nG // PAGE) * PAGE                           # whole pages for Γ, then for q
    qb = -(-8 * nq // PAGE) * PAGE
    rt = torch.cuda.cudart()
    at = block.ctypes.data + first
    assert int(rt.cudaHostRegister(at, gb, 0)) == 0 and int(rt.cudaHostRegister(at + gb, qb, 0)) == 0
    try:
        gam = block[first // 8:][:nG]
        q = block[(first + gb) // 8:][:nq]
        p._check(p.lib.ibpm_get_state(p.handle, G._ptr(gam), G._ptr(q), *[None] * 5))
        assert np.array_equal(gam, src.Gamma.reshape(-1, order="F"))
        assert np.array_equal(q, src.q.reshape(-1, order="F"))
    finally:
        rt.cudaHostUnregister(at)
        rt.cudaHostUnregister(at + gb)
        p.close()
