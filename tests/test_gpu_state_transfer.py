"""State transfers (ibpm_set_state, ibpm_get_state): page-locked host arrays of
a small state go through a kernel (hostio.cu), everything else through copies.
Either way every value comes back as it was sent, for page-locked and pageable
arrays, arrays inside a larger page-locked block, states below and above the
size limit, and any subset of the fields."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(n, mg):
    import ibpm_gpu as G
    g = G.make_grid(4.0 / n, (-2.0, 2.0, -2.0, 2.0), mg)
    return G.IBProblem(g, [G.make_cylinder(0.5, g.h, 0.01, 0.02, n=12)], 0.01, 50.0, freestream=(1.0, 0.3, 0.0))


def _fill(st, seed):
    rng = np.random.default_rng(seed)
    for a in (st.Gamma, st.q, st.psi, st.nonlin[0], st.nonlin[1], st.Fb):
        a[...] = rng.standard_normal(a.shape)


def _same(a, b):
    return all(np.array_equal(x, y) for x, y in [(a.Gamma, b.Gamma), (a.q, b.q), (a.q0, b.q0), (a.psi, b.psi),
                                                 (a.nonlin[0], b.nonlin[0]), (a.nonlin[1], b.nonlin[1]), (a.Fb, b.Fb)])


@pytest.mark.parametrize("n,mg", [(32, 1), (64, 3), (200, 3), (256, 5)])
@pytest.mark.parametrize("pinned_in,pinned_out", [(True, True), (True, False), (False, True)])
def test_round_trip(n, mg, pinned_in, pinned_out):
    import ibpm_gpu as G
    p = _problem(n, mg)
    src = G.pinned_state(p) if pinned_in else G.IBState(p)
    dst = G.pinned_state(p) if pinned_out else G.IBState(p)
    _fill(src, n + mg)
    G.push_state(src, p)
    G.pull_state(dst, p)
    assert _same(src, dst)
    p.close()


def test_pieces_inside_a_page_locked_block_and_subsets():
    import ibpm_gpu as G
    p = _problem(64, 2)
    src = G.IBState(p)
    _fill(src, 3)
    G.push_state(src, p)
    nG, nq = src.Gamma.size, src.q.size
    block = G.PinnedArray((nG + nq + 5,))
    block.array[...] = -7.0
    buf = block.array
    gam, q = buf[1:1 + nG], buf[3 + nG:3 + nG + nq]
    p._check(p.lib.ibpm_get_state(p.handle, G._ptr(gam), G._ptr(q), *[None] * 5))
    assert np.array_equal(gam, src.Gamma.reshape(-1, order="F")) and np.array_equal(q, src.q.reshape(-1, order="F"))
    assert buf[0] == -7.0 and np.all(buf[1 + nG:3 + nG] == -7.0) and np.all(buf[3 + nG + nq:] == -7.0)
    fb = G.PinnedArray(src.Fb.shape)
    p._check(p.lib.ibpm_get_state(p.handle, *[None] * 6, G._ptr(fb.array)))
    assert np.array_equal(fb.array, src.Fb)
    p.close()
