"""FP64 groups on the boundary-transfer chain whose members' bodies sit at
different heights (trial_window, capi.cu): a member transforms the rows of the
trial ψ around its own body alone, and in a group those around every member's,
or two whole levels where one window meets the level's edge.  Its forces and
state are the same bits either way: windows of both parities and of different
extents, with and without a member at the edge, on a length whose x-pass takes
one line pair per group of threads and one whose blocks loop over the pairs,
with one transform plan for all launches and with another for launches of
several slabs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
H = 1.0 / 16
# body_idx of the first point and the points along y, 2h apart
INSIDE = [((20, 20), 3), ((24, 27), 2), ((22, 33), 4), ((30, 23), 1)]
EDGE = ((30, 7), 3)


def _spec(n, where, re):
    import ibpm_gpu as G
    (bx, by), rows = where
    bnd = (-n * H / 2, n * H / 2, -n * H / 2, n * H / 2)
    x = bnd[0] + H * (bx + 0.37 + np.array([0.0, 2.0]))
    y = bnd[2] + H * (by + 0.61 + 2.0 * np.arange(rows))
    xb = np.stack([a.ravel() for a in np.meshgrid(x, y, indexing="ij")], axis=1)
    return dict(grid=G.make_grid(H, bnd, 3), bodies=[G.RigidBody(xb=xb, ds=np.full(len(xb), 2 * H))], dt=0.01,
                Re=re, freestream=(1.0, 0.0, 0.1), precision="fp64")


def _start(m, seed):
    import ibpm_gpu as G
    st = G.IBState(m)
    st.Gamma[...] = 1e-3 * np.random.default_rng(seed).standard_normal(st.Gamma.shape)
    G.push_state(st, m)
    G.vort2flux(st, m)


@pytest.mark.parametrize("n", [64, 192])
@pytest.mark.parametrize("plans", [(0, 2), (0, 1), (1, 0)])
@pytest.mark.parametrize("edge", [False, True])
def test_members_of_a_group_with_different_windows(n, plans, edge):
    import ibpm_gpu as G
    specs = [_spec(n, w, 40.0 + 20.0 * i) for i, w in enumerate(INSIDE + ([EDGE] if edge else []))]
    batch = G.Batch(specs, lanes=1)
    batch.set_grouped(True)
    batch.set_chain(G.IBPM_CHAIN_BOUNDARY_TRANSFER)
    for m in batch.members:
        G.set_transform_plan(m, *plans)
    batch.set_plan(plans[0])
    for i, m in enumerate(batch.members):
        _start(m, 40 + i)
    forces = batch.advance(5)
    for i, sp in enumerate(specs):
        assert tuple(G.transform_plan(batch.members[i])) == plans
        solo = G.IBProblem(sp["grid"], sp["bodies"], sp["dt"], sp["Re"], freestream=sp["freestream"], sync_fields=False)
        G.set_transform_plan(solo, *plans)
        G.set_level_chain(solo, G.IBPM_CHAIN_BOUNDARY_TRANSFER)
        _start(solo, 40 + i)
        st = G.IBState(solo)
        cd, cl = G.advance(st, solo, 0.0, nsteps=5)
        G.pull_state(st, solo)
        bst = G.IBState(batch.members[i])
        assert np.array_equal(forces[i][0], cd) and np.array_equal(forces[i][1], cl), i
        assert np.array_equal(bst.Gamma, st.Gamma) and np.array_equal(bst.q, st.q) and np.array_equal(bst.Fb, st.Fb), i
        solo.close()
    batch.close()
