"""The device inverse of the Schur complement (linalg.cu) beyond 706 rows: panels
of 16, 8 and 4 columns and column by column, at the first and last size of every
width and of every row count that a width is built for.  Each column j of the
oracle's B (B_times!, laplacian.jl:143-169) must be taken to e_j: Gauss–Jordan
with partial pivoting leaves ‖B⁻¹B − I‖ ≲ n ε ‖B‖ ‖B⁻¹‖, 1-norms, taken with a
factor 10 over 48 columns, the first and last and those at the panels' edges
among them (‖B‖ is then that of these columns, which only tightens the bound;
B has no zeros to speak of, so an error in any column of B⁻¹ shows)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb", [416, 417, 640, 641, 704, 705, 832, 833, 1280, 1281, 1408, 1409, 1664, 1665, 2560, 2561])
def test_inverse_takes_columns_of_B_to_unit_vectors(nb):
    import ibpm_gpu as G
    from oracle import ibpm_ref as R
    h, bnd = 1.0 / 32, (-2.0, 2.0, -2.0, 2.0)
    # points 2h apart on rows 2h apart, off the grid lines: B well conditioned
    cols = int(np.ceil(np.sqrt(nb)))
    k = np.arange(nb)
    xb = np.stack([-1.75 + 2 * h * (k % cols) + 0.3 * h, -1.75 + 2 * h * (k // cols) + 0.4 * h], axis=1)
    ds = np.full(nb, 2 * h)
    op = R.IBProblem(grid=R.make_grid(h, bnd, 1), bodies=[R.Body(xb=xb, ds=ds)], dt=0.01, Re=100.0, build_binv=False)
    n = 2 * nb
    edges = [0, 1, 3, 4, 7, 8, 15, 16, 63, 64, nb - 1, nb, n - 65, n - 64, n - 2, n - 1]
    rest = np.setdiff1d(np.arange(n), edges)
    j = np.concatenate([edges, np.random.default_rng(nb).choice(rest, 32, replace=False)])
    E = np.zeros((n, len(j)))
    E[j, np.arange(len(j))] = 1.0
    B = R.B_times(op, E)
    gp = G.IBProblem(G.make_grid(h, bnd, 1), [G.RigidBody(xb=xb, ds=ds)], 0.01, 100.0)
    binv = gp.binv()
    gp.close()
    res = np.linalg.norm(binv @ B - E, 1)
    cond = np.linalg.norm(B, 1) * np.linalg.norm(binv, 1)
    assert res <= 10 * n * np.finfo(float).eps * cond, (nb, res, cond)
