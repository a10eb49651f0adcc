"""The device inverse of the Schur complement (linalg.cu) at the edges of its
panels: one block for the whole matrix (32, 64, 104 and 128 rows are its sizes),
panels of 64 columns and their row counts, panels of 32 and 16 columns inside a
block of 64, a last panel of a few columns, and column by column beyond 5120
rows.  The library builds B for that many points; B⁻¹ is checked against the
oracle's B (B_times!, laplacian.jl:143-169) by its residual: Gauss–Jordan with
partial pivoting leaves ‖B⁻¹B − I‖ ≲ n ε cond(B), 1-norms, taken with a factor
10."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb", [1, 2, 16, 17, 32, 33, 51, 52, 53, 64, 65, 96, 104, 105, 160, 161, 176, 177, 200, 352, 353,
                                2820])
def test_inverse_of_B(nb):
    import ibpm_gpu as G
    from oracle import ibpm_ref as R
    h, bnd = 1.0 / 32, (-2.0, 2.0, -2.0, 2.0)
    # points 2h apart on rows 2h apart, off the grid lines: B well conditioned
    cols = int(np.ceil(np.sqrt(nb)))
    k = np.arange(nb)
    xb = np.stack([-1.75 + 2 * h * (k % cols) + 0.3 * h, -1.75 + 2 * h * (k // cols) + 0.4 * h], axis=1)
    ds = np.full(nb, 2 * h)
    og = R.make_grid(h, bnd, 1)
    op = R.IBProblem(grid=og, bodies=[R.Body(xb=xb, ds=ds)], dt=0.01, Re=100.0, build_binv=False)
    B = R.build_B(op)
    gp = G.IBProblem(G.make_grid(h, bnd, 1), [G.RigidBody(xb=xb, ds=ds)], 0.01, 100.0)
    binv = gp.binv()
    gp.close()
    n = 2 * nb
    res = np.linalg.norm(binv @ B - np.eye(n), 1)
    cond = np.linalg.norm(B, 1) * np.linalg.norm(binv, 1)
    assert res <= 10 * n * np.finfo(float).eps * cond, (nb, res, cond)
