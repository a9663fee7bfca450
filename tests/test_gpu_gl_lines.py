"""The line form of the uncollocated stage kernel (Gauss-Legendre flux nodes and overintegration,
Chandrashekar + EC/Roe + BR2) against the oracle, at every order and number of flux nodes it is
compiled for, with and without gradients that need the logarithms of the means. Tolerance: the
residual contract, 1e-12 relative max-norm."""
import numpy as np
import pytest

from oracle.oracle import Oracle
from philip_b200.dg import DGStrong, RungeKuttaODESolver
from philip_b200.prm import Parameters

from helpers import perturbed_tgv, prm_dict, rel_max_err

SIZES = [(p, o) for p in range(1, 7) for o in range(3) if p + 1 + o <= 7]


def _case(p, over, pde, **kw):
    d = prm_dict(poly_degree=p, n_cells=2, pde=pde, diss="bassi_rebay_2", **kw)
    d["flux_nodes_type"] = "GL"
    d["overintegration"] = over
    prm = Parameters.from_dict(d)
    return Oracle(prm.oracle_cfg(), prm.n_cells, *prm.grid_bounds), DGStrong(prm)


@pytest.mark.gpu
@pytest.mark.parametrize("strong", [False, True], ids=["smooth", "strong"])
@pytest.mark.parametrize("pde", ["euler", "navier_stokes"])
@pytest.mark.parametrize("p,over", SIZES)
def test_gl_line_kernel_residual_and_step(p, over, pde, strong):
    orc, dg = _case(p, over, pde, fr="cHU")
    U = perturbed_tgv(orc, seed=p)
    if strong:
        U = U * (1.0 + 0.4 * np.random.default_rng(p).random(U.shape))
    err = rel_max_err(dg.residual_of(U), orc.residual(U))
    V = U.copy()
    orc.rk_step(V, 1e-4)
    dg.solution = U
    RungeKuttaODESolver(dg).step_in_time(1e-4)
    err2 = rel_max_err(dg.solution, V)
    print(f"p={p} over={over} {pde} strong {strong}: residual {err:.2e}, step {err2:.2e}")
    assert err <= 1e-12 and err2 <= 1e-12
    assert dg.status() == 0
