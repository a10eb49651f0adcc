"""The tridiagonal y-solve (ibpm.jl_b200/csrc/ysolve.cu) at the edges of its
layout: every number of chunks per scan lane, chunk counts that do not fill a
warp (25, 50), the smallest and largest ny, and grids far from square, where
the boundary source's correction is largest.  On a single level vort2flux! is
one Δ⁻¹ solve, so ψ is compared with the DST-I definition of that solve
evaluated in extended precision.

The tolerance is n·ε, n = max(nx, ny): a rounding of relative size ε/2 in
either recursion is carried by r^m, in all at most 1/(1 − r) ≤ nx/π times, and
the x-transforms add ε log₂ nx."""
import numpy as np
import pytest
import scipy.fft as sfft

pytestmark = pytest.mark.gpu
SIZES = [(32, 32), (64, 32), (32, 64), (128, 128), (200, 400), (400, 200), (256, 192), (192, 256), (384, 384),
         (512, 512), (2048, 32), (32, 2048), (64, 768), (256, 1024)]


def delta_inv_extended(f):
    """Δ⁻¹ f of the 5-point Laplacian, f (nx−1, ny−1), in extended precision."""
    L = np.longdouble
    nx, ny = f.shape[0] + 1, f.shape[1] + 1
    pi = L("3.14159265358979323846264338327950288")
    lx = 4 * np.sin(pi * np.arange(1, nx, dtype=L) / (2 * nx)) ** 2
    ly = 4 * np.sin(pi * np.arange(1, ny, dtype=L) / (2 * ny)) ** 2
    w = sfft.dst(sfft.dst(f.astype(L), type=1, axis=0), type=1, axis=1) / (lx[:, None] + ly[None, :])
    return sfft.dst(sfft.dst(w, type=1, axis=0), type=1, axis=1) / (4 * nx * ny)


@pytest.mark.parametrize("nx,ny", SIZES)
def test_single_level_solve(nx, ny):
    import ibpm_gpu as G
    h = 1.0 / 64
    g = G.make_grid(h, (-nx * h / 2, nx * h / 2, -ny * h / 2, ny * h / 2), 1)
    assert (g.nx, g.ny) == (nx, ny)
    p = G.IBProblem(g, [G.make_cylinder(4 * h, h, 0.3 * h, 0.4 * h, n=8)], 0.01, 100.0)
    rng = np.random.default_rng(nx + 7 * ny)
    x, y = np.arange(1, nx)[:, None] / nx, np.arange(1, ny)[None, :] / ny
    corner = np.zeros((nx - 1, ny - 1))
    corner[-1, 0] = 1.0
    for f in (rng.standard_normal((nx - 1, ny - 1)), np.exp(-30 * ((x - 0.4) ** 2 + (y - 0.6) ** 2)), corner):
        st = G.IBState(p)
        st.Gamma[:, 0] = f.flatten(order="F")
        G.push_state(st, p, fields=("Gamma",))
        G.vort2flux(st, p)
        want = delta_inv_extended(f)
        got = st.psi[:, 0].reshape(want.shape, order="F")
        err = float(np.linalg.norm((got - want).astype(float)) / np.linalg.norm(want.astype(float)))
        assert err <= max(nx, ny) * np.finfo(float).eps, (nx, ny, err)
    p.close()
