"""The line form of the stage kernel (Chandrashekar + EC/Roe, no boundary faces): every order's split of
lines over lanes, tile lists, cell counts that leave the last CTA partly filled, affine and curved cells,
states with and without gradients that need the logarithms of the means. Against the general kernel
bit by bit, and whole steps against the oracle (1e-12 relative max-norm)."""
import numpy as np
import pytest

from oracle.oracle import Oracle
from philip_b200 import _lib
from philip_b200.dg import DGStrong, RungeKuttaODESolver
from philip_b200.prm import Parameters
from philip_b200.serve import Batch

from helpers import perturbed_tgv, prm_dict, rel_max_err


def _pair(kw, warp, precision):
    prm = Parameters.from_dict(prm_dict(**kw))
    orc = Oracle(prm.oracle_cfg(), prm.n_cells, *prm.grid_bounds, warp=warp)
    return orc, DGStrong(prm, precision=precision, warp=warp)


def _state(orc, strong, seed):
    """strong: neighbouring nodes differ by tens of percent, so no tile takes the series alone."""
    U = perturbed_tgv(orc, seed=seed, amp=1e-3)
    return U * (1.0 + 0.6 * np.random.default_rng(seed).random(U.shape)) if strong else U


@pytest.mark.gpu
@pytest.mark.parametrize("strong", [False, True], ids=["smooth", "strong"])
@pytest.mark.parametrize("warp", [0.0, 0.1])
@pytest.mark.parametrize("p", [1, 2, 3, 4, 5, 6])
def test_line_kernel_has_the_bits_of_the_general_kernel(p, warp, strong):
    """Slip walls on the z sides of 4^3 cells: a context runs the line kernel on the tiles of the two
    inner layers (from its tile list) and the boundary-face form of the general kernel on the outer
    ones, a batch runs the general kernel on every tile. Both evaluate every flux in the same order
    of operations: one RK4 step is the same to the last bit."""
    bnd = ["periodic"] * 4 + ["slip_wall"] * 2
    prm = Parameters.from_dict(prm_dict(poly_degree=p, n_cells=4))
    orc = Oracle(prm.oracle_cfg(), prm.n_cells, *prm.grid_bounds)
    U = _state(orc, strong, seed=p)
    mesh = _lib.PhMeshDesc(prm.n_cells, 0, *prm.grid_bounds, warp, p)
    for f, t in enumerate(_lib.boundary_ids(bnd)):
        mesh.boundary_type[f] = t
    b = Batch(1 << 28, _lib.PH_FP64)
    slot = b.admit(mesh, prm.to_ph_params(_lib.PH_FP64), U, 1e-3, 1)
    b.step(1)
    Ub = b.state(slot, U.size)
    b.close()
    dg = DGStrong(prm, warp=warp, boundaries=bnd)
    dg.solution = U
    RungeKuttaODESolver(dg).step_in_time(1e-3)
    assert np.array_equal(dg.solution, Ub) and not np.array_equal(Ub, U)


@pytest.mark.gpu
@pytest.mark.parametrize("p", [2, 3, 5])
@pytest.mark.parametrize("warp", [0.0, 0.1])
@pytest.mark.parametrize("fr,rk", [("cDG", "ssprk3_ex"), ("cHU", "rk4_ex")])
def test_line_kernel_steps(fr, rk, warp, p):
    """Every output of the epilogue: running sum, next stage, carry and the FR mass inverse."""
    orc, dg = _pair(dict(poly_degree=p, n_cells=3, fr=fr, rk=rk), warp, _lib.PH_FP64)
    U = _state(orc, False, seed=11 + p)
    V = U.copy()
    dg.solution = U
    for _ in range(2):
        orc.rk_step(V, 1e-3)
    RungeKuttaODESolver(dg).step_in_time(1e-3, nsteps=2)
    err = rel_max_err(dg.solution, V)
    print(f"p={p} {fr} {rk} warp {warp}: {err:.2e}")
    assert err <= 1e-12
