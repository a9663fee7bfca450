"""The wide form of the line kernel (a warp group per direction, meshes of one wave of CTAs) has the bits of the
narrow form. A block of 2^3 cells repeated over a mesh that is large enough for the narrow form has the
block's solution in every copy; h = 1/2 on both meshes, so that every operation has the same operands."""
import numpy as np
import pytest

from oracle.oracle import Oracle
from philip_b200 import _lib
from philip_b200.dg import DGStrong, RungeKuttaODESolver
from philip_b200.prm import Parameters

from helpers import perturbed_tgv, prm_dict

LARGE = {1: 20, 2: 12, 3: 12, 5: 8}   # cells per direction past one wave of the wide form


def _step(n, U, p, pde, fr, precision):
    prm = Parameters.from_dict(prm_dict(poly_degree=p, n_cells=n, pde=pde, diss="bassi_rebay_2", fr=fr,
                                        left=0.0, right=0.5 * n))
    dg = DGStrong(prm, precision=precision, cell_order=1)   # (lexicographic, as the copies are laid out)
    dg.solution = U
    RungeKuttaODESolver(dg).step_in_time(1e-3)
    assert dg.status() == 0
    return dg.solution.reshape(n, n, n, -1)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [_lib.PH_FP64, _lib.PH_FP32_RESIDUAL], ids=["fp64", "fp32"])
@pytest.mark.parametrize("pde,fr", [("euler", "cDG"), ("navier_stokes", "cDG"), ("euler", "cHU")])
@pytest.mark.parametrize("p", sorted(LARGE))
def test_wide_form_has_the_bits_of_the_narrow_form(p, pde, fr, precision):
    prm = Parameters.from_dict(prm_dict(poly_degree=p, n_cells=2, pde=pde, left=0.0, right=1.0))
    orc = Oracle(prm.oracle_cfg(), prm.n_cells, *prm.grid_bounds)
    U = perturbed_tgv(orc, seed=p)
    small = _step(2, U, p, pde, fr, precision)
    n = LARGE[p]
    V = np.tile(U.reshape(2, 2, 2, -1), (n // 2, n // 2, n // 2, 1)).reshape(U.size * (n // 2) ** 3)
    large = _step(n, V.reshape((-1,) + U.shape[1:]) if U.ndim > 1 else V, p, pde, fr, precision)
    assert np.array_equal(large, np.tile(small, (n // 2, n // 2, n // 2, 1)))
    assert not np.array_equal(small, U.reshape(small.shape))
