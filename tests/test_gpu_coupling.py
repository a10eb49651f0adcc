"""The lists of E' and C'E' are counted, scanned and ranked on the device
(coupling.cu): one point on the smallest grid, blocks of points 2h apart (up to 42
contributors at a flux point, more than a warp takes at once), fluxes of two scan
blocks (2112 of 2048) and of several, two bodies on one grid.  Forces and the projected circulation after two steps against the oracle
to 1e-10, the bound the other step tests use."""
import numpy as np
import pytest

from ibpm_cases import random_state, rel, to_gpu_state

pytestmark = pytest.mark.gpu
TOL = 1e-10
H = 1.0 / 16
# nx, ny, levels, first body_idx and number of points along x and y of each body
CASES = [(32, 32, 1, [(8, 9, 1, 1)]),
         (32, 32, 2, [(8, 8, 3, 2)]),
         (32, 32, 1, [(8, 8, 7, 7)]),
         (64, 32, 3, [(9, 9, 6, 5), (30, 12, 5, 4)]),
         (128, 64, 2, [(20, 20, 7, 9), (100, 40, 1, 6)])]


@pytest.mark.parametrize("nx,ny,mg,blocks", CASES)
def test_lists(nx, ny, mg, blocks):
    import ibpm_gpu as G
    from oracle import ibpm_ref as R
    bnd = (-nx * H / 2, nx * H / 2, -ny * H / 2, ny * H / 2)
    pts = []
    for bx, by, kx, ky in blocks:
        x = bnd[0] + H * (bx + 0.37 + 2.0 * np.arange(kx))
        y = bnd[2] + H * (by + 0.61 + 2.0 * np.arange(ky))
        pts.append(np.stack([a.ravel() for a in np.meshgrid(x, y, indexing="ij")], axis=1))
    op = R.IBProblem(grid=R.make_grid(H, bnd, mg), bodies=[R.Body(xb=p, ds=np.full(len(p), 2 * H)) for p in pts],
                     dt=0.01, Re=50.0, inclination=0.1)
    gp = G.IBProblem(G.make_grid(H, bnd, mg), [G.RigidBody(xb=p, ds=np.full(len(p), 2 * H)) for p in pts], 0.01, 50.0,
                     freestream=(1.0, 0.0, 0.1))
    ost = random_state(op, seed=11)
    gst = G.IBState(gp)
    to_gpu_state(ost, gst)
    G.push_state(gst, gp)
    cd, cl = G.advance(gst, gp, 0.0, nsteps=2)
    ocd, ocl = R.run(op, ost, 2)
    gp.close()
    assert rel(cd, ocd) < TOL and rel(cl, ocl) < TOL
    assert rel(gst.Gamma, R.gamma_to_ref(ost.Gamma)) < TOL
    assert rel(gst.Fb[:, 0], ost.Fb) < TOL
