"""The conservative form's own stage kernel on Gauss-Legendre flux nodes and with overintegration (affine
periodic cells): residual and one RK step against the oracle at every order and number of flux nodes it
is compiled for, the numerical fluxes in turn. Tolerance: the residual contract, 1e-12 relative max-norm."""
import pytest

from oracle.oracle import Oracle
from philip_b200.dg import DGStrong, RungeKuttaODESolver
from philip_b200.prm import Parameters

from helpers import perturbed_tgv, prm_dict, rel_max_err

SIZES = [(p, o) for p in range(1, 7) for o in range(3) if p + 1 + o <= 7]
FLUXES = [("lax_friedrichs", "symm_internal_penalty"), ("roe", "bassi_rebay_2"),
          ("central_flux", "symm_internal_penalty"), ("roe", "central_visc_flux")]


@pytest.mark.gpu
@pytest.mark.parametrize("pde", ["euler", "navier_stokes"])
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("p,over", SIZES)
def test_gl_conservative_residual_and_step(p, over, shift, pde):
    conv, diss = FLUXES[(2 * shift + p + over) % len(FLUXES)]
    d = prm_dict(poly_degree=p, n_cells=2, pde=pde, split=False, conv=conv, diss=diss, fr="cHU")
    d["flux_nodes_type"] = "GL"
    d["overintegration"] = over
    prm = Parameters.from_dict(d)
    orc, dg = Oracle(prm.oracle_cfg(), prm.n_cells, *prm.grid_bounds), DGStrong(prm)
    U = perturbed_tgv(orc, seed=p)
    err = rel_max_err(dg.residual_of(U), orc.residual(U))
    V = U.copy()
    orc.rk_step(V, 1e-4)
    dg.solution = U
    RungeKuttaODESolver(dg).step_in_time(1e-4)
    err2 = rel_max_err(dg.solution, V)
    print(f"p={p} over={over} {pde} {conv} {diss}: residual {err:.2e}, step {err2:.2e}")
    assert err <= 1e-12 and err2 <= 1e-12
    assert dg.status() == 0
