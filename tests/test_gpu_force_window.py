"""E reads q = C ψ around the bodies only (trial_window, capi.cu; E_kernel,
body.cu): bodies whose 13×13 windows just touch the first or last flux of a row
or column (the level's edge values enter) and bodies one cell inside, against
the oracle to 1e-10 on every field and on CD, CL, single and nested grids, one
and several rows of bodies."""
import numpy as np
import pytest

from ibpm_cases import random_state, rel, to_gpu_state

pytestmark = pytest.mark.gpu
TOL = 1e-10
N, H = 64, 1.0 / 16
# body_idx of the first point (1-based): windows reach idx - 6 … idx + 6 + 4
EDGES = {"left": (7, 30), "right": (N - 10, 30), "bottom": (30, 7), "top": (30, N - 10), "corner": (7, 7),
         "inside": (8, 8), "inside_far": (N - 11, N - 11)}


@pytest.mark.parametrize("where", sorted(EDGES))
@pytest.mark.parametrize("mg", [1, 3])
def test_windows_at_the_edge(where, mg):
    import ibpm_gpu as G
    from oracle import ibpm_ref as R
    bx, by = EDGES[where]
    bnd = (-2.0, 2.0, -2.0, 2.0)
    # three points 2h apart along each direction, off the grid lines
    x = bnd[0] + H * (bx + 0.37 + np.array([0.0, 2.0, 4.0]))
    y = bnd[2] + H * (by + 0.61 + np.array([0.0, 2.0, 4.0]))
    xb = np.stack([a.ravel() for a in np.meshgrid(x, y, indexing="ij")], axis=1)
    ds = np.full(len(xb), 2 * H)
    og = R.make_grid(H, bnd, mg)
    op = R.IBProblem(grid=og, bodies=[R.Body(xb=xb, ds=ds)], dt=0.01, Re=50.0, inclination=0.1)
    gp = G.IBProblem(G.make_grid(H, bnd, mg), [G.RigidBody(xb=xb, ds=ds)], 0.01, 50.0, freestream=(1.0, 0.0, 0.1))
    ost = random_state(op, seed=5)
    gst = G.IBState(gp)
    to_gpu_state(ost, gst)
    G.push_state(gst, gp)
    cd, cl = G.advance(gst, gp, 0.0, nsteps=4)
    ocd, ocl = R.run(op, ost, 4)
    gp.close()
    assert rel(cd, ocd) < TOL and rel(cl, ocl) < TOL
    assert rel(gst.Gamma, R.gamma_to_ref(ost.Gamma)) < TOL
    assert rel(gst.psi, R.gamma_to_ref(ost.psi)) < TOL
    assert rel(gst.q, R.flux_to_ref(ost.qx, ost.qy)) < TOL
    assert rel(gst.Fb[:, 0], ost.Fb) < TOL
