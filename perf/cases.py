"""The work that programs have this framework do, as cases that can be timed and checked.

A case is one pass through a public entry point (the C-ABI, DGStrong, RungeKuttaODESolver, Batch):

  residual ... ph_residual on device arrays (DGBase::assemble_residual)
  steps ...... set the state, RK steps of one dt, read the state back (ODESolverBase::step_in_time)
  adaptive ... RK step + the Taylor-Green integrals that give the next time step (FlowSolver::run
               with adaptive_time_step)
  batch ...... RK steps of several solves resident in one arena, and their states on the host

The state is the Taylor-Green vortex with random smooth modes added (seeded). `exact` is the same
discretisation written with plain torch in 64 bits: the dense tensor-product operators, every node
pair and every face, no kernel of this repository.
"""
import math

import numpy as np
import torch

from philip_b200 import _lib
from philip_b200.dg import DGStrong, RungeKuttaODESolver
from philip_b200.prm import Parameters
from philip_b200.serve import Batch

TWO_PI = 6.28318530717958623200
GAMMA, MACH, REYNOLDS, PRANDTL, TEMPERATURE = 1.4, 0.1, 1600.0, 0.71, 273.15
MAX_DOFS = 14_929_920   # 24^3 cells, p = 5

CONV = {"lf": "lax_friedrichs", "roe": "roe", "ec": "two_point_flux",
        "ec_lf": "two_point_flux_with_lax_friedrichs_dissipation", "ec_roe": "two_point_flux_with_roe_dissipation"}
DISS = {"sipg": "symm_internal_penalty", "br2": "bassi_rebay_2", "central": "central_visc_flux"}


def _case(kind, n, p, *, pde="navier_stokes", nodes="GLL", two_point="CH", conv="ec_roe", diss="br2",
          precision="fp64", warp=0.0, steps=1, rk="rk4_ex", mach=MACH, name=None):
    """two_point "" is the conservative strong form (use_split_form = false)."""
    c = {"kind": kind, "n": n, "p": p, "pde": pde, "nodes": nodes, "two_point": two_point, "conv": conv, "diss": diss,
         "precision": precision, "warp": warp, "steps": steps, "rk": rk, "mach": mach}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: one residual of a test-sized mesh, launch latency
        _case("residual", 4, 3, pde="euler", name="residual_euler_4_p3"),
        # the inviscid Taylor-Green benchmark (8^3, p = 3): state resident in L2, several steps per call
        _case("steps", 8, 3, pde="euler", steps=4, name="steps_euler_8_p3"),
        # the headline benchmark: viscous Taylor-Green, 24^3, p = 5, GLL, CH split + Roe, BR2, RK4
        _case("steps", 24, 5, steps=2, name="steps_ns_24_p5"),
        # the same in the precision form (FP32 residual, FP64 state)
        _case("steps", 24, 5, steps=2, precision="fp32", name="steps_ns_24_p5_f32"),
        # the low-order benchmark: viscous Taylor-Green, 32^3, p = 3
        _case("steps", 32, 3, steps=2, name="steps_ns_32_p3"),
        # an odd size at an odd number of nodes, precision form
        _case("steps", 17, 4, steps=2, precision="fp32", name="steps_ns_17_p4_f32"),
        # the benchmark on Gauss-Legendre flux nodes (the reference's default flux_nodes_type)
        _case("steps", 24, 5, nodes="GL", steps=1, name="steps_ns_gl_24_p5"),
        # the reference's strong-form energy check: conservative form, Roe + SIPG on GL nodes, one SSPRK3 step
        _case("steps", 12, 3, nodes="GL", two_point="", conv="roe", diss="sipg", rk="ssprk3_ex",
              name="steps_ns_gl_strong_12_p3"),
        # adaptive time step: every step is followed by the integrals that set the next one
        _case("adaptive", 16, 5, name="adaptive_ns_16_p5"),
        # other fluxes of the .prm surface on an odd mesh: Ismail-Roe, Lax-Friedrichs dissipation, SIPG
        _case("residual", 13, 2, two_point="IR", conv="ec_lf", diss="sipg", name="residual_ns_ir_13_p2"),
        # a curved (sine-warped) cube, Euler, as served solves use
        _case("steps", 12, 4, pde="euler", warp=0.1, steps=2, mach=0.3, name="steps_euler_curved_12_p4"),
        # a small batch of served solves (orders 2..5 on warped meshes, precision form), eight steps at a time
        _case("batch", 8, 2, pde="euler", precision="fp32", warp=0.1, steps=8, mach=0.2, name="batch_served_f32"),
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, p, top, lo=3):
    most = int((top / (5.0 * (p + 1) ** 3)) ** (1.0 / 3.0) + 1e-9)
    return max(lo, min(most, _spread(rng, lo, max(lo, most))))


def draw(rng):
    kind = rng.choice(["residual", "steps", "steps", "steps_f32", "steps_f32", "gl", "gl", "adaptive", "curved", "batch"])
    p = rng.choice([2, 3, 3, 4, 5, 5, 6])
    if kind == "residual":
        tp = rng.choice(["CH", "IR", "Ra", "KG", ""])
        return _case("residual", _size(rng, p, 4e6), p, pde=rng.choice(["euler", "navier_stokes"]), two_point=tp,
                     conv=rng.choice(["lf", "roe"] if not tp else ["lf", "roe", "ec", "ec_lf", "ec_roe"]),
                     diss=rng.choice(["sipg", "br2", "central"]))
    if kind in ("steps", "steps_f32"):
        return _case("steps", _size(rng, p, MAX_DOFS), p, pde=rng.choice(["euler", "navier_stokes", "navier_stokes"]),
                     steps=2, precision="fp32" if kind == "steps_f32" else "fp64")
    if kind == "gl":
        split = rng.random() < 0.6
        return _case("steps", _size(rng, p, MAX_DOFS), p, nodes="GL", pde=rng.choice(["euler", "navier_stokes", "navier_stokes"]),
                     two_point="CH" if split else "", conv="ec_roe" if split else "roe", diss=rng.choice(["br2", "sipg"]))
    if kind == "adaptive":
        return _case("adaptive", _size(rng, p, 6e6), p)
    if kind == "curved":
        return _case("steps", _size(rng, p, 3e6), p, pde="euler", warp=0.1, steps=2, mach=0.3)
    return _case("batch", rng.randint(4, 10), 2, pde="euler", precision="fp32", warp=rng.choice([0.0, 0.1]), steps=8,
                 mach=rng.choice([0.15, 0.2, 0.25]))


# ------------------------------------------------------------------------------------------------
# what a program has in hand
# ------------------------------------------------------------------------------------------------
def _parameters(case, n, p):
    return Parameters.from_dict({
        "dimension": 3, "pde_type": case["pde"], "use_weak_form": False, "flux_nodes_type": case["nodes"],
        "use_split_form": bool(case["two_point"]), "two_point_num_flux_type": case["two_point"] or "KG",
        "conv_num_flux": CONV[case["conv"]], "diss_num_flux": DISS[case["diss"]], "flux_reconstruction": "cDG",
        "use_inverse_mass_on_the_fly": True, "all_boundaries_are_periodic": True, "do_renumber_dofs": False,
        "ODE solver/ode_solver_type": "runge_kutta", "ODE solver/runge_kutta_method": case["rk"],
        "euler/mach_infinity": case["mach"], "euler/gamma_gas": GAMMA, "navier_stokes/reynolds_number_inf": REYNOLDS,
        "navier_stokes/prandtl_number": PRANDTL, "navier_stokes/temperature_inf": TEMPERATURE,
        "flow_solver/flow_case_type": "taylor_green_vortex", "flow_solver/poly_degree": p,
        "flow_solver/courant_friedrichs_lewy_number": 0.1, "flow_solver/adaptive_time_step": True,
        "flow_solver/grid/grid_left_bound": 0.0, "flow_solver/grid/grid_right_bound": TWO_PI,
        "flow_solver/grid/number_of_grid_elements_per_dimension": n})


def _solves(case):
    """(cells per direction, order) of every solve of a case."""
    if case["kind"] != "batch":
        return [(case["n"], case["p"])]
    n = case["n"]
    return [(n, 2), (n + 1, 3), (n, 4), (n + 3, 2), (n + 2, 5), (n + 5, 3)]


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _legendre(n, x):
    p0, p1 = torch.ones_like(x), x
    for k in range(2, n + 1):
        p0, p1 = p1, ((2 * k - 1) * x * p1 - (k - 1) * p0) / k
    return (p0, p1) if n > 0 else (torch.zeros_like(x), p0)


def _gauss(n):
    x, w = np.polynomial.legendre.leggauss(n)
    x = torch.from_numpy(x)
    for _ in range(3):
        p0, p1 = _legendre(n, x)
        x = x - p1 * (x * x - 1) / (n * (x * p1 - p0))
    p0, p1 = _legendre(n, x)
    dp = n * (x * p1 - p0) / (x * x - 1)
    return 0.5 * (x + 1), 1.0 / ((1 - x * x) * dp * dp)


def _lobatto(n):
    m = n - 1
    x = -torch.cos(math.pi * torch.arange(n, dtype=torch.float64) / m)
    for _ in range(60):
        p0, p1 = _legendre(m, x)
        dx = (x * p1 - p0) / (n * p1)
        dx[0] = dx[-1] = 0.0
        x = x - dx
    _, p1 = _legendre(m, x)
    return 0.5 * (x + 1), 1.0 / (m * n * p1 * p1)


def _coordinates(n, p, warp):
    """Solution nodes [cz, cy, cx, 3, z, y, x] of the (warped) cube, cells lexicographic."""
    d = _device()
    x = (torch.arange(n, dtype=torch.float64, device=d)[:, None] + _lobatto(p + 1)[0].to(d)) * (TWO_PI / n)
    X = x[None, None, :, None, None, :].expand(n, n, n, p + 1, p + 1, p + 1)
    Y = x[None, :, None, None, :, None].expand_as(X)
    Z = x[:, None, None, :, None, None].expand_as(X)
    s = warp * torch.sin(X) * torch.sin(Y) * torch.sin(Z)
    return torch.stack([X + s, Y + s, Z + s], dim=3)


def _initial_state(n, p, warp, mach, seed):
    """Taylor-Green vortex + random smooth modes, [cz, cy, cx, 5, z, y, x]."""
    C = _coordinates(n, p, warp)
    X, Y, Z = C[:, :, :, 0], C[:, :, :, 1], C[:, :, :, 2]
    rng = np.random.default_rng(seed)
    f = []
    for amplitude in (0.02, 0.05, 0.05, 0.05, 0.1):
        v = 0.0
        for _ in range(3):
            k, ph = rng.integers(-2, 3, 3), rng.uniform(0, TWO_PI)
            v = v + amplitude / 3 * rng.uniform(0.5, 1.0) * torch.cos(float(k[0]) * X + float(k[1]) * Y + float(k[2]) * Z + ph)
        f.append(v)
    rho = 1 + f[0]
    u = torch.sin(X) * torch.cos(Y) * torch.cos(Z) + f[1]
    v = -torch.cos(X) * torch.sin(Y) * torch.cos(Z) + f[2]
    w = f[3] * torch.ones_like(X)
    pr = 1 / (GAMMA * mach * mach) + (torch.cos(2 * X) + torch.cos(2 * Y)) * (torch.cos(2 * Z) + 2) / 16 + f[4]
    E = pr / (GAMMA - 1) + 0.5 * rho * (u * u + v * v + w * w)
    U = torch.stack([rho, rho * u, rho * v, rho * w, E], dim=3)
    wave = (torch.sqrt(u * u + v * v + w * w) + torch.sqrt(GAMMA * pr / rho)).max().item()
    dt = 0.1 * (TWO_PI / (n * (p + 1))) / wave
    return U.contiguous(), dt


def prepare(case, seed):
    prec = _lib.PH_FP32_RESIDUAL if case["precision"] == "fp32" else _lib.PH_FP64
    if case["kind"] == "batch":
        batch = Batch(1 << 30, prec)
        slots = []
        for i, (n, p) in enumerate(_solves(case)):
            prm = _parameters(case, n, p)
            mesh = _lib.PhMeshDesc(n, 1, 0.0, TWO_PI, case["warp"], p)
            U, dt = _initial_state(n, p, case["warp"], case["mach"], seed + 1000 * i)
            slots.append((batch.admit(mesh, prm.to_ph_params(prec), U.reshape(-1).cpu().numpy(), dt, 1 << 30), U.numel()))
        return {"case": case, "batch": batch, "slots": slots}
    n, p = case["n"], case["p"]
    # the program's own stream: its solver and its buffers stay on it
    stream = torch.cuda.Stream()
    dg = DGStrong(_parameters(case, n, p), precision=prec, cell_order=1, warp=case["warp"], stream=stream.cuda_stream)
    U, dt = _initial_state(n, p, case["warp"], case["mach"], seed)
    out = torch.empty_like(U)
    torch.cuda.synchronize()
    return {"case": case, "stream": stream, "dg": dg, "ode": RungeKuttaODESolver(dg), "U": U, "dt": dt, "out": out}


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        state["batch"].step(case["steps"])
        return [state["batch"].state(slot, ndofs) for slot, ndofs in state["slots"]]
    dg, L, out = state["dg"], state["dg"].L, state["out"]
    if case["kind"] == "residual":
        _lib.check(L.ph_residual(dg.handle, state["U"].data_ptr(), out.data_ptr(), _lib.PH_DEVICE))
        return out
    _lib.check(L.ph_set_state(dg.handle, state["U"].data_ptr(), _lib.PH_DEVICE))
    state["ode"].step_in_time(state["dt"], nsteps=case["steps"])
    rows = dg.integrals() if case["kind"] == "adaptive" else None
    _lib.check(L.ph_get_state(dg.handle, out.data_ptr(), _lib.PH_DEVICE))
    return out if rows is None else [out, rows]


# ------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------------
def _stages(case):
    return 3 if case["rk"] == "ssprk3_ex" else 4


def work(case):
    """Bytes: a residual reads the state and writes as much; an RK step's stages read and write the
    state and the running sum (32 B per DOF and stage on average); setting and reading the state
    copies it. Operations per node and stage, add / mul / fma 1, 1, 2 and division, root and
    logarithm 1: each node pair once (76), each face node once (226, or 206 inviscid), 67 per node;
    Navier-Stokes: gradient, viscous flux and divergence; GL nodes: the dense interpolations."""
    B = F = 0.0
    for n, p in _solves(case):
        n1 = p + 1
        nodes = float(n ** 3 * n1 ** 3)
        dofs = 5 * nodes
        visc = case["pde"] == "navier_stokes"
        flops = (1.5 * (n1 - 1) * 76 if case["two_point"] else 30 * n1) + 3.0 / n1 * (226 if visc else 206) + 67
        if visc:
            flops += 54 * n1 + 100
        if case["nodes"] == "GL":
            flops += 3 * 2 * n1 * 5 * 4 + (3 * 2 * n1 * 15 if visc else 0)
        if case["warp"]:
            flops += 1.5 * (n1 - 1) * 15 if case["two_point"] else 45
        if case["kind"] == "residual":
            B += 16 * dofs
            F += flops * nodes
            continue
        B += case["steps"] * _stages(case) * 32 * dofs + (8 if case["kind"] == "batch" else 32) * dofs
        F += case["steps"] * _stages(case) * flops * nodes
        if case["kind"] == "adaptive":
            ne = n1 + 10
            B += 8 * dofs
            F += n ** 3 * (ne ** 3 * (2 * n1 * 14 + 70.0) + ne * ne * n1 * 2 * n1 * 14)
    return {"bytes": B, "flops": F}


# ------------------------------------------------------------------------------------------------
# the same results in 64 bits, with plain torch
# ------------------------------------------------------------------------------------------------
def _lagrange(nodes, x):
    """Values and derivatives of the Lagrange basis on `nodes` at the points x: [point, basis]."""
    n = len(nodes)
    V, D = torch.zeros(len(x), n, dtype=torch.float64), torch.zeros(len(x), n, dtype=torch.float64)
    for j in range(n):
        others = [m for m in range(n) if m != j]
        c = 1.0
        for m in others:
            c = c / (nodes[j] - nodes[m])
        V[:, j] = c
        for m in others:
            V[:, j] = V[:, j] * (x - nodes[m])
        for k in others:
            t = torch.full_like(x, 1.0) * c
            for m in others:
                if m != k:
                    t = t * (x - nodes[m])
            D[:, j] += t
    return V, D


def _apply(A, f, d):
    """The 1-D operator A [rows, cols] along direction d (0: x, the last axis)."""
    return torch.movedim(torch.tensordot(f, A, dims=([f.dim() - 1 - d], [1])), -1, f.dim() - 1 - d)


def _apply3(A, f):
    for d in range(3):
        f = _apply(A[d] if isinstance(A, (list, tuple)) else A, f, d)
    return f


def _surface(chi, row, d, f):
    """Face values of f on the side that `row` [1, nodes] stands for, tangential axes through chi;
    the axis of direction d keeps its place with one entry."""
    return _apply3([row if e == d else chi for e in range(3)], f)


def _pick(f, s):
    return f.select(3, s)


def _primitive(u):
    rho = _pick(u, 0)
    v = [_pick(u, 1 + k) / rho for k in range(3)]
    p = (GAMMA - 1) * (_pick(u, 4) - 0.5 * rho * (v[0] ** 2 + v[1] ** 2 + v[2] ** 2))
    return rho, v, p


def _log_mean(a, b):
    f = (a - b) / (a + b)
    u = f * f
    series = (a + b) / (2 * (1 + u / 3 + u * u / 5 + u * u * u / 7))
    plain = (a - b) / torch.where(u < 1e-2, torch.ones_like(a), torch.log(a) - torch.log(b))
    return torch.where(u < 1e-2, series, plain)


def _two_point(kind, i, j, n):
    """Two-point flux dotted with n (three fields or numbers); i, j from _primitive + E."""
    (ri, vi, pi, Ei), (rj, vj, pj, Ej) = i, j
    va = [0.5 * (a + b) for a, b in zip(vi, vj)]
    vv = lambda v: v[0] ** 2 + v[1] ** 2 + v[2] ** 2  # noqa: E731
    extra = 0.0
    if kind == "CH":
        r = _log_mean(ri, rj)
        bi, bj = ri / (2 * pi), rj / (2 * pj)
        p = 0.5 * (ri + rj) / (bi + bj)
        H = 1 / (2 * _log_mean(bi, bj) * (GAMMA - 1)) + p / r + vv(va) - 0.25 * (vv(vi) + vv(vj))
        v = va
    elif kind == "Ra":
        r, b = _log_mean(ri, rj), _log_mean(ri / pi, rj / pj)
        p, v = 0.5 * (pi + pj), va
        H = (r + 2 * b * (GAMMA - 1) * p) / (b * (GAMMA - 1) * r) + vv(va) - 0.25 * (vv(vi) + vv(vj))
        extra = -0.5 * sum((pi * a + pj * b) * c for a, b, c in zip(vi, vj, n))
    elif kind == "IR":
        zi, zj, yi, yj = torch.sqrt(ri / pi), torch.sqrt(rj / pj), torch.sqrt(ri * pi), torch.sqrt(rj * pj)
        za = 0.5 * (zi + zj)
        l0, l4 = _log_mean(zi, zj), _log_mean(yi, yj)
        r, p = za * l4, 0.5 * (yi + yj) / za
        v = [0.5 * (zi * a + zj * b) / za for a, b in zip(vi, vj)]
        H = ((GAMMA + 1) * l4 / l0 + (GAMMA - 1) * p) / (2 * GAMMA) * GAMMA / (r * (GAMMA - 1)) + 0.5 * vv(v)
    else:
        r, p, v = 0.5 * (ri + rj), 0.5 * (pi + pj), va
        H = 0.5 * (Ei / ri + Ej / rj) + p / r
    m = r * sum(a * b for a, b in zip(v, n))
    return torch.stack([m] + [m * v[k] + p * n[k] for k in range(3)] + [m * H + extra], dim=3)


def _quantities(u):
    return (*_primitive(u), _pick(u, 4))


def _euler_flux(u, n):
    rho, v, p = _primitive(u)
    vn = sum(a * b for a, b in zip(v, n))
    m = rho * vn
    return torch.stack([m] + [m * v[k] + p * n[k] for k in range(3)] + [vn * (_pick(u, 4) + p)], dim=3)


def _numerical_flux(case, uL, uR, n):
    """Convective numerical flux along the unit normal n (left to right)."""
    conv = case["conv"]
    if conv in ("ec", "ec_lf", "ec_roe"):
        F = _two_point(case["two_point"], _quantities(uL), _quantities(uR), n)
    else:
        F = 0.5 * (_euler_flux(uL, n) + _euler_flux(uR, n))
    (rL, vL, pL), (rR, vR, pR) = _primitive(uL), _primitive(uR)
    cL, cR = torch.sqrt(GAMMA * pL / rL), torch.sqrt(GAMMA * pR / rR)
    nL, nR = sum(a * b for a, b in zip(vL, n)), sum(a * b for a, b in zip(vR, n))
    if conv in ("lf", "ec_lf"):
        lam = torch.maximum(nL.abs() + cL, nR.abs() + cR)
        return F - 0.5 * lam.unsqueeze(3) * (uR - uL)
    if conv not in ("roe", "ec_roe"):
        return F
    hL, hR = (_pick(uL, 4) + pL) / rL, (_pick(uR, 4) + pR) / rR
    r = torch.sqrt(rR / rL)
    ra = r * rL
    va = [(r * b + a) / (r + 1) for a, b in zip(vL, vR)]
    ha = (r * hR + hL) / (r + 1)
    v2, vn = sum(a * a for a in va), sum(a * b for a, b in zip(va, n))
    c2 = (GAMMA - 1) * (ha - 0.5 * v2)
    ca = torch.sqrt(c2)
    eig = []
    for e, eL, eR in ((vn - ca, nL - cL, nR - cR), (vn, nL, nR), (vn + ca, nL + cL, nR + cR)):
        e, eL, eR = e.abs(), eL.abs(), eR.abs()
        eps = torch.maximum((e - eL).abs(), (eR - e).abs())
        eig.append(torch.where(e < eps, 0.5 * (e * e / torch.where(eps > 0, eps, torch.ones_like(eps)) + eps), e))
    dp, dr, dn = pR - pL, rR - rL, nR - nL
    dt = [(b - a) - dn * k for a, b, k in zip(vL, vR, n)]
    a0 = eig[0] * (dp - ra * ca * dn) / (2 * c2)
    a1 = eig[1] * (dr - dp / c2)
    a2 = eig[1] * ra
    a3 = eig[2] * (dp + ra * ca * dn) / (2 * c2)
    A = [a0 + a1 + a3] + [a0 * (va[k] - ca * n[k]) + a1 * va[k] + a2 * dt[k] + a3 * (va[k] + ca * n[k]) for k in range(3)]
    A.append(a0 * (ha - ca * vn) + a1 * v2 * 0.5 + a2 * sum(a * b for a, b in zip(va, dt)) + a3 * (ha + ca * vn))
    return F - 0.5 * torch.stack(A, dim=3)


def _viscous_flux(case, u, g, d):
    """Component d of the viscous flux from the state and the gradients g[0..2] of the conservative variables."""
    rho, v, p = _primitive(u)
    gv = [[(_pick(g[e], 1 + a) - v[a] * _pick(g[e], 0)) / rho for e in range(3)] for a in range(3)]
    m2 = case["mach"] ** 2
    T = GAMMA * m2 * p / rho
    tr = 110.4 / TEMPERATURE
    mu = (1 + tr) / (T + tr) * T ** 1.5 / REYNOLDS
    gp = (GAMMA - 1) * (_pick(g[d], 4) - 0.5 * sum(v[m] * _pick(g[d], 1 + m) + _pick(u, 1 + m) * gv[m][d] for m in range(3)))
    gT = (GAMMA * m2 * gp - T * _pick(g[d], 0)) / rho
    tau = [mu * (gv[k][d] + gv[d][k]) for k in range(3)]
    tau[d] = tau[d] - 2.0 / 3.0 * mu * (gv[0][0] + gv[1][1] + gv[2][2])
    q = -mu / ((GAMMA - 1) * m2 * PRANDTL) * gT
    return torch.stack([torch.zeros_like(rho)] + [-t for t in tau] + [q - sum(a * b for a, b in zip(v, tau))], dim=3)


def _entropy_variables(u):
    rho, v, p = _primitive(u)
    s = torch.log(p * rho ** (-GAMMA))
    rt = p / (GAMMA - 1)
    return torch.stack([(rt * (GAMMA + 1 - s) - _pick(u, 4)) / rt] + [_pick(u, 1 + k) / rt for k in range(3)] + [-rho / rt], dim=3)


def _from_entropy_variables(w):
    w5 = _pick(w, 4)
    k = 0.5 * sum(_pick(w, 1 + m) ** 2 for m in range(3)) / w5
    s = GAMMA - _pick(w, 0) + k
    rt = ((GAMMA - 1) / (-w5) ** GAMMA) ** (1 / (GAMMA - 1)) * torch.exp(-s / (GAMMA - 1))
    return torch.stack([-rt * w5] + [rt * _pick(w, 1 + m) for m in range(3)] + [rt * (1 - k)], dim=3)


class _Exact:
    """The discretisation of one solve: operators on the device and the residual of a state."""

    def __init__(self, case, n, p):
        dev = _device()
        self.case, self.n, self.p, self.h = case, n, p, TWO_PI / n
        nodes = _lobatto(p + 1)[0]
        xq, w = _gauss(p + 1) if case["nodes"] == "GL" else _lobatto(p + 1)
        self.collocated = case["nodes"] != "GL"
        chi = _lagrange(nodes, xq)[0] if not self.collocated else torch.eye(p + 1, dtype=torch.float64)
        ends = torch.tensor([0.0, 1.0], dtype=torch.float64)
        chis, (_, D), phis = _lagrange(nodes, ends)[0], _lagrange(xq, xq), _lagrange(xq, ends)[0]
        Q = w[:, None] * D
        M = chi.T @ (w[:, None] * chi)
        self.chi, self.D, self.w, self.skew = chi.to(dev), D.to(dev), w.to(dev), (Q - Q.T).to(dev)
        self.chis = [chis[s:s + 1].to(dev) for s in range(2)]
        self.phis = [phis[s:s + 1].to(dev) for s in range(2)]
        self.Minv = torch.linalg.inv(M).to(dev)
        self.proj = self.Minv @ (self.chi.T * self.w)
        self.W = self.w[:, None, None] * self.w[None, :, None] * self.w[None, None, :]
        self.C = self.detj = None
        if case["warp"]:
            self._metric()

    def _metric(self):
        """Cofactors C[k][d] = J (d xi_d / d x_k) at the nodes by the conservative curl form, and det J (GLL nodes)."""
        X = _coordinates(self.n, self.p, self.case["warp"])
        X = [X[:, :, :, k] for k in range(3)]
        G = [[_apply(self.D, X[m], j) for j in range(3)] for m in range(3)]
        self.C = []
        for k in range(3):
            m, l = (k + 1) % 3, (k + 2) % 3
            f = [X[l] * G[m][j] for j in range(3)]
            self.C.append([_apply(self.D, f[(d + 1) % 3], (d + 2) % 3) - _apply(self.D, f[(d + 2) % 3], (d + 1) % 3)
                           for d in range(3)])
        J = G
        self.detj = (J[0][0] * (J[1][1] * J[2][2] - J[1][2] * J[2][1]) - J[0][1] * (J[1][0] * J[2][2] - J[1][2] * J[2][0])
                     + J[0][2] * (J[1][0] * J[2][1] - J[1][1] * J[2][0]))

    def _normal(self, d):
        """C[:, d] at the volume nodes (numbers h^2 e_d on the straight cube)."""
        return [c[d] for c in self.C] if self.C else [self.h ** 2 if k == d else 0.0 for k in range(3)]

    def _face_weights(self, d):
        w = [self.w if e != d else torch.ones(1, dtype=torch.float64, device=self.w.device) for e in range(3)]
        return w[2][:, None, None] * w[1][None, :, None] * w[0][None, None, :]

    def _lift(self, side, d, f):
        return _apply3([(self.chis[side] if e == d else self.chi).T.contiguous() for e in range(3)], f * self._face_weights(d))

    def _test(self, f):
        return f if self.collocated else _apply3(self.chi.T.contiguous(), f)

    @staticmethod
    def _next(f, d):
        """The value that the cell at +1 along d holds, for every cell (cells are [cz, cy, cx])."""
        return torch.roll(f, -1, dims=2 - d)

    @staticmethod
    def _previous(f, d):
        return torch.roll(f, 1, dims=2 - d)

    def residual(self, U):
        case, h = self.case, self.h
        chi3 = (lambda f: f) if self.collocated else (lambda f: _apply3(self.chi, f))
        face = lambda f, s, d: _surface(self.chi, self.chis[s], d, f)  # noqa: E731
        visc, split = case["pde"] == "navier_stokes", bool(case["two_point"])
        uq = chi3(U)
        area = h * h
        grad = None
        if visc:   # the lifted gradient (straight cells): its coefficients per direction
            grad = []
            for d in range(3):
                r = self._test(self.W * _apply(self.D, uq, d)) * area
                lo, hi = face(U, 0, d), face(U, 1, d)
                r = r + area * self._lift(1, d, 0.5 * (hi + self._next(lo, d)) - hi)
                r = r - area * self._lift(0, d, 0.5 * (lo + self._previous(hi, d)) - lo)
                grad.append(_apply3(self.Minv, r) / h ** 3)
        ut, coef = uq, U
        if split and not self.collocated:
            coef = _apply3(self.proj, _entropy_variables(uq))
            ut = _from_entropy_variables(chi3(coef))
        q = _quantities(ut)
        div = torch.zeros_like(uq)
        for d in range(3):
            nd = self._normal(d)
            if not split:
                div = div + self.W * _apply(self.D, _euler_flux(ut, nd), d)
                continue
            ax = uq.dim() - 1 - d
            perp = [self.w if e != d else torch.ones_like(self.w) for e in range(3)]
            perp = perp[2][:, None, None] * perp[1][None, :, None] * perp[0][None, None, :]
            at = lambda f, k: f.narrow(f.dim() - 1 - d, k, 1) if torch.is_tensor(f) else f  # noqa: E731
            acc = torch.zeros_like(uq)
            sub = [(at(q[0], k), [at(v, k) for v in q[1]], at(q[2], k), at(q[3], k)) for k in range(self.p + 1)]
            for i in range(self.p + 1):
                for j in range(i + 1, self.p + 1):
                    nij = [0.5 * (at(m, i) + at(m, j)) for m in nd]
                    F = _two_point(case["two_point"], sub[i], sub[j], nij)
                    acc.narrow(ax, i, 1).add_(F, alpha=self.skew[i, j].item())
                    acc.narrow(ax, j, 1).add_(F, alpha=self.skew[j, i].item())
            div = div + acc * perp
        if visc:
            gq = [chi3(g) for g in grad]
            for d in range(3):
                div = div + self.W * _apply(self.D, area * _viscous_flux(case, ut, gq, d), d)
        R = -self._test(div)
        # faces: every face once, seen from the cell on its left (side 1) and the one on its right (side 0)
        pen = self.p * (self.p + 1) / h if case["diss"] == "sipg" else 0.0
        for d in range(3):
            nd = self._normal(d)
            if self.C:
                nf = [face(m.unsqueeze(3), 1, d).select(3, 0) for m in nd]
                J = torch.sqrt(nf[0] ** 2 + nf[1] ** 2 + nf[2] ** 2)
                unit = [m / J for m in nf]
                J = J.unsqueeze(3)
            else:
                J, unit = area, [1.0 if k == d else 0.0 for k in range(3)]
            tr = [face(coef, s, d) for s in range(2)]
            if split and not self.collocated:
                tr = [_from_entropy_variables(t) for t in tr]
            flux = J * _numerical_flux(case, tr[1], self._next(tr[0], d), unit)
            if visc:
                raw = [face(U, s, d) for s in range(2)]
                gr = [[face(g, s, d) for g in grad] for s in range(2)]
                own = [_viscous_flux(case, raw[s], gr[s], d) for s in range(2)]
                fv = 0.5 * (own[1] + self._next(own[0], d))
                if pen:
                    zero = torch.zeros_like(raw[0])
                    uR = self._next(raw[0], d)
                    jump = [raw[1] - uR if e == d else zero for e in range(3)]
                    fv = fv - pen * 0.5 * (_viscous_flux(case, raw[1], jump, d) + _viscous_flux(case, uR, jump, d))
                flux = flux + J * fv
                vol = [_viscous_flux(case, uq, gq, d)]
                for s in range(2):
                    inside = area * _apply(self.phis[s], vol[0], d)
                    R = R + (1 if s else -1) * self._lift(s, d, inside)
            R = R - self._lift(1, d, flux) + self._lift(0, d, self._previous(flux, d))
            for s in range(2):
                sign = 1 if s else -1
                if not split:
                    R = R + sign * self._lift(s, d, _apply(self.phis[s], _euler_flux(ut, nd), d))
                elif not self.collocated:   # the hybrid terms between a face node and its normal line
                    uf = _quantities(tr[s])
                    F = _two_point(case["two_point"], q, (uf[0], uf[1], uf[2], uf[3]), nd)
                    phi = self.phis[s][0].reshape([-1 if e == d else 1 for e in (2, 1, 0)])
                    F = F * phi * self._face_weights(d)
                    ones = torch.ones(1, self.p + 1, dtype=torch.float64, device=F.device)
                    R = R - sign * self._test(F)
                    R = R + sign * _apply3([(self.chis[s] if e == d else self.chi).T.contiguous() for e in range(3)],
                                           _apply(ones, F, d))
        return R

    def rate(self, U):
        R = self.residual(U)
        if self.C:
            return R / (self.W * self.detj.unsqueeze(3))
        return _apply3(self.Minv, R) / self.h ** 3

    def step(self, U, dt):
        if self.case["rk"] == "ssprk3_ex":
            k1 = self.rate(U)
            k2 = self.rate(U + dt * k1)
            k3 = self.rate(U + dt * (0.25 * k1 + 0.25 * k2))
            return U + dt * (k1 / 6 + k2 / 6 + k3 * (2.0 / 3.0))
        k1 = self.rate(U)
        k2 = self.rate(U + 0.5 * dt * k1)
        k3 = self.rate(U + 0.5 * dt * k2)
        k4 = self.rate(U + dt * k3)
        return U + dt * (k1 + 2 * k2 + 2 * k3 + k4) / 6

    def integrals(self, U):
        """Kinetic energy, enstrophy, vorticity-based dissipation, maximum wave speed (QGauss(p+11))."""
        x, w = _gauss(self.p + 11)
        V, D = (m.to(U.device) for m in _lagrange(_lobatto(self.p + 1)[0], x))
        w = w.to(U.device)
        W = w[:, None, None] * w[None, :, None] * w[None, None, :] * self.h ** 3 / TWO_PI ** 3
        ke = en = wave = 0.0
        for layer in U.split(1):
            u = _apply3(V, layer)
            g = [_apply3([D if e == d else V for e in range(3)], layer) / self.h for d in range(3)]
            rho, v, p = _primitive(u)
            gv = [[(_pick(g[d], 1 + a) - v[a] * _pick(g[d], 0)) / rho for d in range(3)] for a in range(3)]
            om2 = (gv[2][1] - gv[1][2]) ** 2 + (gv[0][2] - gv[2][0]) ** 2 + (gv[1][0] - gv[0][1]) ** 2
            v2 = v[0] ** 2 + v[1] ** 2 + v[2] ** 2
            ke += (0.5 * rho * v2 * W).sum().item()
            en += (0.5 * rho * om2 * W).sum().item()
            wave = max(wave, (torch.sqrt(v2) + torch.sqrt(GAMMA * p / rho)).max().item())
        return np.array([ke, en, 2 * en / REYNOLDS, wave])


def exact(case, seed):
    got = []
    for i, (n, p) in enumerate(_solves(case)):
        s = seed + (1000 * i if case["kind"] == "batch" else 0)
        U, dt = _initial_state(n, p, case["warp"], case["mach"], s)
        E = _Exact(case, n, p)
        if case["kind"] == "residual":
            return E.residual(U)
        for _ in range(case["steps"]):
            U = E.step(U, dt)
        if case["kind"] == "adaptive":
            return [U, E.integrals(U)]
        got.append(U)
    return [u.reshape(-1).cpu().numpy() for u in got] if case["kind"] == "batch" else got[0]
