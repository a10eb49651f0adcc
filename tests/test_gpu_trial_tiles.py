"""The trial right-hand side of large grids takes 2 × 2 points per thread and the rim
in blocks of its own (stencil.cu): square and oblong grids just above the size where
that begins, two steps against the oracle to 1e-10 (the bound of the other step
tests), and a group of two such simulations against single runs bit for bit."""
import numpy as np
import pytest

from ibpm_cases import random_state, rel, to_gpu_state

pytestmark = pytest.mark.gpu
TOL = 1e-10
H = 1.0 / 64


def case(nx, ny):
    bnd = (-nx * H / 2, nx * H / 2, -ny * H / 2, ny * H / 2)
    p = H * (0.37 + 2.0 * np.arange(3))
    xb = np.stack([a.ravel() for a in np.meshgrid(p, p, indexing="ij")], axis=1)
    return bnd, xb, np.full(len(xb), 2 * H)


@pytest.mark.parametrize("nx,ny,mg", [(512, 512, 3), (1024, 512, 2), (512, 1024, 2)])
def test_tiles(nx, ny, mg):
    import ibpm_gpu as G
    from oracle import ibpm_ref as R
    bnd, xb, ds = case(nx, ny)
    op = R.IBProblem(grid=R.make_grid(H, bnd, mg), bodies=[R.Body(xb=xb, ds=ds)], dt=0.002, Re=50.0, inclination=0.1)
    gp = G.IBProblem(G.make_grid(H, bnd, mg), [G.RigidBody(xb=xb, ds=ds)], 0.002, 50.0, freestream=(1.0, 0.0, 0.1))
    ost = random_state(op, seed=3)
    gst = G.IBState(gp)
    to_gpu_state(ost, gst)
    G.push_state(gst, gp)
    cd, cl = G.advance(gst, gp, 0.0, nsteps=2)
    ocd, ocl = R.run(op, ost, 2)
    gp.close()
    assert rel(cd, ocd) < TOL and rel(cl, ocl) < TOL
    assert rel(gst.Gamma, R.gamma_to_ref(ost.Gamma)) < TOL
    assert rel(gst.q, R.flux_to_ref(ost.qx, ost.qy)) < TOL


def test_group_of_tiled_members():
    import ibpm_gpu as G
    bnd, xb, ds = case(512, 512)
    specs = [dict(grid=G.make_grid(H, bnd, 3), bodies=[G.RigidBody(xb=xb, ds=ds)], dt=0.002, Re=re,
                  freestream=(1.0, 0.0, 0.1), precision="fp64") for re in (50.0, 120.0)]
    batch = G.Batch(specs, lanes=1)
    forces = batch.advance(3)
    for i, sp in enumerate(specs):
        solo = G.IBProblem(sp["grid"], sp["bodies"], sp["dt"], sp["Re"], freestream=sp["freestream"], sync_fields=False)
        G.set_transform_plan(solo, *G.transform_plan(batch.members[i]))
        G.set_level_chain(solo, G.level_chain(batch.members[i]))
        st = G.IBState(solo)
        cd, cl = G.advance(st, solo, 0.0, nsteps=3)
        G.pull_state(st, solo)
        bst = G.IBState(batch.members[i])
        assert np.array_equal(forces[i][0], cd) and np.array_equal(forces[i][1], cl)
        assert np.array_equal(bst.Gamma, st.Gamma) and np.array_equal(bst.q, st.q)
        solo.close()
    batch.close()
