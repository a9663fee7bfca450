"""Uncollocated kernels (Gauss-Legendre flux nodes and overintegration) on 3^3 cells, where a cell's two
neighbours along an axis are different cells, so that an exchange of them shows: residual against the
oracle at every order and number of flux nodes, blocks wider than their lines (up to four flux nodes)
among them. Tolerance: the residual contract, 1e-12 relative max-norm."""
import numpy as np
import pytest

from oracle.oracle import Oracle
from philip_b200.dg import DGStrong
from philip_b200.prm import Parameters

from helpers import perturbed_tgv, prm_dict, rel_max_err

SIZES = [(p, o) for p in range(1, 7) for o in range(3) if p + 1 + o <= 7]


def _case(p, over, **kw):
    d = prm_dict(poly_degree=p, n_cells=3, **kw)
    d["flux_nodes_type"] = "GL"
    d["overintegration"] = over
    prm = Parameters.from_dict(d)
    return Oracle(prm.oracle_cfg(), prm.n_cells, *prm.grid_bounds), DGStrong(prm)


@pytest.mark.gpu
@pytest.mark.parametrize("strong", [False, True], ids=["smooth", "strong"])
@pytest.mark.parametrize("p,over", SIZES)
def test_split_form(p, over, strong):
    orc, dg = _case(p, over, pde="navier_stokes", diss="bassi_rebay_2")
    U = perturbed_tgv(orc, seed=20 + p)
    if strong:
        U = U * (1.0 + 0.4 * np.random.default_rng(p).random(U.shape))
    err = rel_max_err(dg.residual_of(U), orc.residual(U))
    print(f"p={p} over={over} strong {strong}: {err:.2e}")
    assert err <= 1e-12 and dg.status() == 0
