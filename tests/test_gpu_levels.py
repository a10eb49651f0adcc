"""The boundary-transfer vort2flux! (src/fluid-operators/curl.jl:133-165) for
every number of levels the library takes (its chain kernels are instantiated
per level count), against the oracle to 1e-10."""
import numpy as np
import pytest

from ibpm_cases import rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(64, 64), (128, 32)])
@pytest.mark.parametrize("mg", range(2, 9))
def test_vort2flux_levels(nx, ny, mg):
    import ibpm_gpu as G
    from oracle import ibpm_ref as R
    h = 1.0 / 16
    bnd = (-nx * h / 2, nx * h / 2, -ny * h / 2, ny * h / 2)
    gp = G.IBProblem(G.make_grid(h, bnd, mg), [G.make_cylinder(0.25, h, 0.02, 0.01, n=8)], 0.01, 100.0)
    assert G.level_chain(gp) == G.IBPM_CHAIN_BOUNDARY_TRANSFER
    og = R.make_grid(h, bnd, mg)
    Gam = np.random.default_rng(mg).standard_normal((mg, nx - 1, ny - 1))
    st = G.IBState(gp)
    st.Gamma[:] = R.gamma_to_ref(Gam)
    G.push_state(st, gp, fields=("Gamma",))
    G.vort2flux(st, gp)
    gp.close()
    psi, qx, qy = R.vort2flux(Gam, R.lap_eigs(og), og)
    assert rel(st.psi, R.gamma_to_ref(psi)) < 1e-10
    assert rel(st.q, R.flux_to_ref(qx, qy)) < 1e-10
