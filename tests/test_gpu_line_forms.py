"""The narrow form of the line kernel, which meshes past the wide form's range run, at the orders that have
both: meshes that no B200 takes the wide form on (past two waves of its CTAs at p = 1, past one at the other
orders, were the SMs filled to their 2048 threads), with a last CTA that is partly filled.
Tile lists, curved cells and states that need the logarithms of the means against the general kernel bit by
bit; both forms (at p = 1 the wide one also in its second wave) against each other bit by bit, viscous and in
both precisions."""
import numpy as np
import pytest

from oracle.oracle import Oracle
from philip_b200 import _lib
from philip_b200.dg import DGStrong, RungeKuttaODESolver
from philip_b200.prm import Parameters
from philip_b200.serve import Batch

from helpers import perturbed_tgv, prm_dict

SMS = 148
# order: (threads and cells of a wide CTA, waves of them that still run wide)
WIDE = {1: (96, 4, 2), 2: (96, 1, 1), 3: (96, 1, 1), 5: (384, 1, 1)}
BOTH = [(p, prec) for p in sorted(WIDE) for prec in (_lib.PH_FP64, _lib.PH_FP32_RESIDUAL)]
IDS = [f"p{p}-{'fp64' if prec == _lib.PH_FP64 else 'fp32'}" for p, prec in BOTH]


def _narrow(p, cells):
    threads, per_cta, waves = WIDE[p]
    return cells > 2048 // threads * SMS * per_cta * waves


def _strong(U, seed):
    return U * (1.0 + 0.6 * np.random.default_rng(seed).random(U.shape))


@pytest.mark.gpu
@pytest.mark.parametrize("strong", [False, True], ids=["smooth", "strong"])
@pytest.mark.parametrize("warp", [0.0, 0.1])
@pytest.mark.parametrize("p,n", [(1, 31), (2, 17), (3, 17), (5, 11)])
def test_narrow_form_has_the_bits_of_the_general_kernel(p, n, warp, strong):
    """Slip walls on the z sides: a context runs the line kernel on the inner layers' tiles (a tile list), a
    batch runs the general kernel on every tile."""
    assert _narrow(p, n * n * (n - 2) - 2 * 16)   # (a tile that reaches into a layer at the wall is not inner)
    bnd = ["periodic"] * 4 + ["slip_wall"] * 2
    prm = Parameters.from_dict(prm_dict(poly_degree=p, n_cells=n))
    orc = Oracle(prm.oracle_cfg(), prm.n_cells, *prm.grid_bounds)
    U = perturbed_tgv(orc, seed=p, amp=1e-3)
    if strong:
        U = _strong(U, p)
    mesh = _lib.PhMeshDesc(prm.n_cells, 0, *prm.grid_bounds, warp, p)
    for f, t in enumerate(_lib.boundary_ids(bnd)):
        mesh.boundary_type[f] = t
    b = Batch(1 << 30, _lib.PH_FP64)
    slot = b.admit(mesh, prm.to_ph_params(_lib.PH_FP64), U, 1e-4, 1)
    b.step(1)
    Ub = b.state(slot, U.size)
    b.close()
    dg = DGStrong(prm, warp=warp, boundaries=bnd)
    dg.solution = U
    RungeKuttaODESolver(dg).step_in_time(1e-4)
    assert np.array_equal(dg.solution, Ub) and not np.array_equal(Ub, U)


def _step(n, U, p, pde, precision):
    prm = Parameters.from_dict(prm_dict(poly_degree=p, n_cells=n, pde=pde, diss="bassi_rebay_2", left=0.0,
                                        right=0.5 * n))
    dg = DGStrong(prm, precision=precision, cell_order=1)   # (lexicographic, as the copies are laid out)
    dg.solution = np.ascontiguousarray(U).reshape(-1)
    RungeKuttaODESolver(dg).step_in_time(1e-4)
    assert dg.status() == 0
    return dg.solution.reshape(n, n, n, -1)


@pytest.mark.gpu
@pytest.mark.parametrize("strong", [False, True], ids=["smooth", "strong"])
@pytest.mark.parametrize("pde", ["euler", "navier_stokes"])
@pytest.mark.parametrize("p,precision", BOTH, ids=IDS)
def test_both_forms_have_the_same_bits(p, precision, pde, strong):
    """A block of 3^3 cells, and its copies over a larger mesh of the same cell size."""
    copies = {1: 10, 2: 5, 3: 5, 5: 4}[p]
    assert _narrow(p, (3 * copies) ** 3) and 27 <= SMS
    prm = Parameters.from_dict(prm_dict(poly_degree=p, n_cells=3, pde=pde, left=0.0, right=1.5))
    U = perturbed_tgv(Oracle(prm.oracle_cfg(), prm.n_cells, *prm.grid_bounds), seed=p)
    if strong:
        U = _strong(U, p)
    U = U.reshape(3, 3, 3, -1)
    small = _step(3, U, p, pde, precision)
    assert not np.array_equal(small, U)
    for k in (6, copies) if p == 1 else (copies,):   # (18^3 cells at p = 1: more than one wave of the wide form)
        large = _step(3 * k, np.tile(U, (k, k, k, 1)), p, pde, precision)
        assert np.array_equal(large, np.tile(small, (k, k, k, 1)))
