"""Performance cases: the calls a user of jaxrans_b200 makes, from one residual on a small
O-grid to a Newton step of the 3.9-million-cell wing.

``listed()`` names the cases, ``draw(rng)`` makes others of the same ranges; ``prepare``
builds a case's device plan and inputs from a seed, ``run`` is one pass through the public
entry points, ``work`` the bytes and operations a pass cannot do without, ``exact`` the
same outputs in plain torch FP64 (the operator calls), ``tolerance`` how far another
correct implementation of the same precision may be.

The paths:

* ``residual`` / ``jvp`` -- the residual operator: R2(U), and the exact tangent of the
  first-order residual along v (a linearisation and its application);
* ``line`` -- the line-implicit preconditioner: the factor at (U, CFL) and one solve;
* ``newton`` -- pseudo-transient Newton-Krylov steps from a device-resident state and the
  force coefficients after them, as the march runs them: one case, or a batch.
"""

from __future__ import annotations

import functools
import math
import sys
import tempfile
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parents[1]
if str(ROOT / "jax-rans_b200") not in sys.path:   # the package's folder in this repository
    sys.path.insert(0, str(ROOT / "jax-rans_b200"))

# --- the cases ---------------------------------------------------------------------------

_COMMON = {"kappa": 0.0, "subspace": 10, "restarts": 2, "precision": "fp64", "preconditioner": "line_j",
           "cfl": 10.0, "cfl_max": 1e3, "limit_update": 0.0, "steps": 1, "angles": 0, "uneven": False,
           "sutherland": 0.0, "wake": 0, "span": 0, "tip": 0, "cap": 0}


def _case(**kw) -> dict:
    return {**_COMMON, **kw}


def _euler_o(**kw):
    """The 2D Euler O-grid workload (NACA 0012, M 0.8, HLLC, van Albada)."""
    base = {"grid": "o", "airfoil": "naca0012", "around": 256, "normal": 64, "spacing": 1e-3, "model": "euler",
            "mach": 0.8, "alpha": 1.25, "reynolds": 0.0, "flux": "hllc", "limiter": "van_albada"}
    return _case(**{**base, **kw})


def _sa_c(**kw):
    """The SA-RANS C-grid workload (NACA 4412, M 0.2, Re 6e6, Roe, minmod, GMRES(30))."""
    base = {"grid": "c", "airfoil": "naca4412", "around": 256, "wake": 64, "normal": 96, "spacing": 1e-6,
            "model": "sa", "mach": 0.2, "alpha": 8.0, "reynolds": 6e6, "flux": "roe", "limiter": "minmod",
            "subspace": 30, "limit_update": 0.2, "cfl_max": 1e5}
    return _case(**{**base, **kw})


def _wing(**kw):
    """The swept wing on its 4-block C-H grid (SA, M 0.8, Re 1e7, HLLC, smooth van Albada)."""
    base = {"grid": "wing", "airfoil": "naca0012", "around": 256, "wake": 64, "normal": 64, "span": 80, "tip": 80,
            "cap": 4, "spacing": 2e-6, "model": "sa", "mach": 0.8, "alpha": 2.5, "reynolds": 1e7, "flux": "hllc",
            "limiter": "van_albada_smooth", "subspace": 30, "limit_update": 0.2, "cfl_max": 1e3}
    return _case(**{**base, **kw})


_WING_SMALL = {"around": 64, "wake": 16, "normal": 16, "span": 16, "tip": 16, "cap": 3, "spacing": 1e-4}
_WING_MID = {"around": 128, "wake": 32, "normal": 32, "span": 40, "tip": 40, "cap": 4, "spacing": 2e-5}


def listed() -> list[dict]:
    return [
        # the smallest call: one residual of a coarse Euler grid, where the call itself counts
        {"name": "residual_euler_65x17", "path": "residual", **_euler_o(around=64, normal=16, spacing=1e-2)},
        # the residual operator on the SA workload's grid, as a monitor or another solver calls it
        {"name": "residual_sa_385x97", "path": "residual", **_sa_c()},
        # one exact matrix-vector product on the batched polar's middle grid
        {"name": "jvp_sa_513x129", "path": "jvp",
         **_sa_c(airfoil="naca2412", around=344, wake=84, normal=128)},
        # the preconditioner alone in the mixed form on the largest 2D grid
        {"name": "line_sa_769x193_mixed", "path": "line",
         **_sa_c(airfoil="naca4415", around=512, wake=128, normal=192, mach=0.3, reynolds=9e6, precision="mixed",
                 cfl=25.0)},
        # the Euler workload's march: short GMRES(10) cycles
        {"name": "newton_euler_257x65", "path": "newton", **_euler_o(steps=4)},
        # laminar flow on a grid of odd sizes, Sutherland's law, kappa-scheme reconstruction
        {"name": "newton_laminar_c_odd", "path": "newton",
         **_sa_c(airfoil="naca0012", around=94, wake=21, normal=37, spacing=1e-3, model="laminar", mach=0.5,
                 alpha=3.0, reynolds=5e3, sutherland=0.38, flux="roe", limiter="none", kappa=1.0 / 3.0, subspace=15,
                 cfl_max=1e3, steps=3)},
        # the benchmark's own march: SA-RANS, FP64, GMRES(30)
        {"name": "newton_sa_385x97", "path": "newton", **_sa_c(steps=2)},
        # a batched polar on uneven grids in the mixed form (eight angles and the 769 x 193 grid)
        {"name": "newton_polar8_mixed", "path": "newton",
         **_sa_c(angles=8, uneven=True, precision="mixed", steps=1)},
        # the 3D residual on a wing of ordinary size
        {"name": "residual_wing_490k", "path": "residual", **_wing(**_WING_MID)},
        # the 3D matrix-vector product on a wing of ordinary size
        {"name": "jvp_wing_490k", "path": "jvp", **_wing(**_WING_MID)},
        # a coarse wing in FP64, the split line preconditioner: launches and waits count
        {"name": "newton_wing_49k", "path": "newton", **_wing(**_WING_SMALL, steps=2)},
        # the 3.9-million-cell wing in the mixed form, the coupled line preconditioner
        {"name": "newton_wing_3900k_mixed", "path": "newton",
         **_wing(precision="mixed", preconditioner="line_j_coupled")},
    ]


def draw(rng) -> dict:
    """A case of the same ranges: sizes spread over their logarithm, odd ones among them."""
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    path = rng.choice(["residual", "jvp", "line", "newton", "newton", "newton"])
    kind = rng.choice(["euler", "laminar", "sa", "sa", "wing"])
    flow = {"flux": rng.choice(["hllc", "roe"]), "limiter": rng.choice(["minmod", "van_albada", "van_albada_smooth"]),
            "alpha": rng.uniform(-4.0, 10.0)}
    if kind == "laminar" and rng.random() < 0.5:
        flow.update(limiter="none", kappa=rng.choice([1.0 / 3.0, -1.0]))
    solver = {"subspace": rng.choice([10, 15, 20, 30]), "restarts": rng.choice([1, 2]), "steps": rng.choice([1, 2]),
              "cfl": rng.uniform(5.0, 50.0), "precision": rng.choice(["fp64", "mixed"])}
    if kind == "euler":
        case = _euler_o(around=2 * size(20, 256), normal=size(11, 97), mach=rng.uniform(0.3, 0.8), **flow, **solver)
    elif kind == "wing":
        if path == "line":
            path = "newton"
        around = 4 * size(16, 34)
        case = _wing(around=around, wake=int(around * rng.uniform(0.25, 0.35)), normal=size(16, 34),
                     span=size(12, 41), tip=size(12, 41), spacing=rng.choice([1e-4, 2e-5]),
                     **{**flow, **solver, "alpha": rng.uniform(0.0, 4.0)},
                     preconditioner=rng.choice(["line_j", "line_j_coupled"]))
    else:
        around = 2 * size(32, 256)
        grid = {"around": around, "wake": int(around * rng.uniform(0.25, 0.35)), "normal": size(24, 192),
                "airfoil": rng.choice(["naca0012", "naca2412", "naca4412"])}
        if kind == "laminar":
            case = _sa_c(**grid, spacing=1e-3, model="laminar", mach=rng.uniform(0.2, 0.6), cfl_max=1e3,
                         reynolds=rng.uniform(2e3, 2e4), sutherland=rng.choice([0.0, 0.38]), **flow, **solver)
        else:
            case = _sa_c(**grid, spacing=rng.choice([1e-6, 1e-5]), mach=rng.uniform(0.15, 0.4),
                         reynolds=rng.uniform(3e6, 9e6), **flow, **solver,
                         preconditioner=rng.choice(["line_j", "line_j", "line_j_coupled"]))
            if path == "newton" and grid["around"] * grid["normal"] < 30000 and rng.random() < 0.5:
                case["angles"] = rng.randint(2, 6)
                case["uneven"] = rng.random() < 0.5
    return {"path": path, **case}


# --- the framework's objects of a case ------------------------------------------------------


def _far_field(normal: int) -> float:
    """Chords to the far field: nearer on the coarsest grids, which would fold otherwise."""
    return 50.0 if normal >= 24 else 20.0


def _documents(c: dict, alpha: float, scale: int = 1):
    domain = {"grid": f"{c['grid']}_grid", "airfoil": c["airfoil"], "cells_airfoil": scale * c["around"],
              "cells_normal": scale * c["normal"], "wall_spacing": c["spacing"],
              "far_field": _far_field(scale * c["normal"])}
    if c["grid"] == "c":
        domain["cells_wake"] = scale * c["wake"]
        domain["normal_stretching"] = 1.1
    flow = {"mach": c["mach"], "alpha_deg": alpha}
    case = {"general": {"case_name": "perf"}, "freestream": flow,
            "boundary_conditions": {"wall": {"type": "slip_wall" if c["model"] == "euler" else "no_slip_wall"},
                                    "farfield": {"type": "far_field"}}}
    if c["model"] != "euler":
        flow["reynolds"] = c["reynolds"]
    if c["model"] == "sa":
        case["turbulence"] = {"model": "sa_noft2"}
    if c["sutherland"] > 0.0:
        flow["temperature"] = 288.15
        case["material_properties"] = {"dynamic_viscosity": "sutherland",
                                       "sutherland_temperature": c["sutherland"] * 288.15}
    fluxes = {"riemann_solver": c["flux"], "limiter": c["limiter"]}
    if c["kappa"] != 0.0:
        fluxes["muscl_kappa"] = c["kappa"]
    implicit = {"krylov_subspace": c["subspace"], "krylov_restarts": c["restarts"], "precision": c["precision"],
                "preconditioner": c["preconditioner"], "cfl": c["cfl"], "cfl_max": c["cfl_max"]}
    if c["limit_update"] > 0.0:
        implicit["max_relative_update"] = c["limit_update"]
    numerics = {"convective_fluxes": fluxes, "time_integration": {"solver": "implicit"}, "implicit": implicit,
                "convergence": {"max_iters": 1000, "tol": 1e-12, "block_iters": 20}}
    case["domain"] = domain
    return case, numerics


def _parse(c: dict, alpha: float, scale: int = 1):
    from jaxrans_b200.case import parse_case
    case_doc, num_doc = _documents(c, alpha, scale)
    if c["grid"] == "wing":   # the grid is a file's (below); any grid kind parses the flow and the solver
        case_doc["domain"] = {"grid": "c_grid", "airfoil": "naca0012", "cells_airfoil": 32, "cells_wake": 8,
                              "cells_normal": 16, "wall_spacing": 1e-4, "far_field": 20.0}
    return parse_case(case_doc, num_doc)


@functools.lru_cache(maxsize=6)
def _grid2d(key):
    """A generated 2D grid's plan (host tables), made once per grid."""
    domain, model = dict(key[0]), key[1]
    c = {**_COMMON, **domain, "model": model, "mach": 0.2, "reynolds": 1e6, "flux": "hllc", "limiter": "minmod"}
    return _parse(c, 0.0).grid()


def _plan2d(c: dict, scale: int = 1):
    domain = {k: c[k] for k in ("grid", "airfoil", "spacing")}
    domain.update({k: scale * c[k] for k in ("around", "wake", "normal")})
    return _grid2d((tuple(sorted(domain.items())), c["model"]))


@functools.lru_cache(maxsize=3)
def _grid3d(around, wake, normal, span, tip, cap, spacing):
    """The wing's grid file written and loaded: ``(Plan3, reference area, length, moment centre)``."""
    import json
    from jaxrans_b200.case import load_case
    from jaxrans_b200.geometry import section_source
    from jaxrans_b200.grid3d import wing_ch_blocks, write_plot3d
    g = wing_ch_blocks(section_source("naca0012"), cells_airfoil=around, cells_wake=wake, cells_normal=normal,
                       cells_span=span, cells_tip=tip, wall_spacing=spacing, far_field=_far_field(normal),
                       cap_cells=cap,
                       semispan=1.6, taper=0.6, sweep_deg=25.0)
    with tempfile.TemporaryDirectory() as d:
        write_plot3d(Path(d) / "grid.x", g.blocks)
        case_doc = {"general": {"case_name": "perf"},
                    "domain": {"grid": "file", "file": "grid.x", "patches": g.patches,
                               "reference_area": g.reference_area, "reference_length": g.reference_length,
                               "moment_centre": list(g.moment_centre)},
                    "boundary_conditions": {"wall": {"type": "no_slip_wall"}, "farfield": {"type": "far_field"},
                                            "symmetry": {"type": "symmetry"}},
                    "freestream": {"mach": 0.8, "alpha_deg": 2.5, "reynolds": 1e7},
                    "turbulence": {"model": "sa_noft2"}}
        num_doc = {"convective_fluxes": {"riemann_solver": "hllc", "limiter": "van_albada_smooth"},
                   "time_integration": {"solver": "implicit"}}
        (Path(d) / "case.json").write_text(json.dumps(case_doc))
        (Path(d) / "numerical.json").write_text(json.dumps(num_doc))
        plan = load_case(Path(d)).grid()
    return plan, g.reference_area, g.reference_length, tuple(g.moment_centre)


def _plan3d(c: dict):
    return _grid3d(*(c[k] for k in ("around", "wake", "normal", "span", "tip", "cap")), c["spacing"])


# --- inputs ------------------------------------------------------------------------------------


def _freestream(flow, dim: int) -> np.ndarray:
    a = math.radians(flow.alpha_deg)
    velocity = [flow.mach * math.cos(a), flow.mach * math.sin(a)]
    if dim == 3:
        velocity.insert(1, 0.0)
    q = [1.0] + velocity + [1.0 / flow.gamma]
    if flow.turbulence is not None:
        q.append(flow.nu_tilde_ratio)
    return np.array(q)


def _conservative(q, dim: int, gamma: float):
    rho, vel, p = q[0], q[1:1 + dim], q[1 + dim]
    rows = [rho] + [rho * v for v in vel] + [p / (gamma - 1.0) + 0.5 * rho * (vel * vel).sum(0)]
    if q.shape[0] > 2 + dim:
        rows.append(rho * q[2 + dim])
    return torch.stack(rows)


def _state(plan, case, dim: int, rng) -> torch.Tensor:
    """A state a march passes through: the freestream slowed to rest at a viscous wall over
    a layer of a few hundredths of a chord, an eddy viscosity bump in the layer, and a
    smooth disturbance of a few percent round the body that dies out slowly (so that no
    cell is exactly uniform, where |vorticity| has its kink); ghosts and gaps the
    freestream, as the march starts them (the residual there is U - U_inf, exactly 0)."""
    from jaxrans_b200.solver import freestream_state
    from jaxrans_b200.solver3d import freestream_state3
    flow = case.flow
    cuda = functools.partial(torch.as_tensor, dtype=torch.float64, device="cuda")
    x = cuda(np.ascontiguousarray(plan.centres[(slice(None),) + (slice(1, -1),) * dim]))
    inside = torch.as_tensor(np.ascontiguousarray(plan.interior), device="cuda")
    q_inf = _freestream(flow, dim)
    shape = (len(q_inf),) + tuple(plan.shape)
    q = cuda(q_inf).reshape((-1,) + (1,) * dim).expand(shape).clone()
    near = 1.0 / (1.0 + ((x - 0.5) ** 2).sum(0) / 9.0)
    layer = None
    if plan.distance is not None:
        layer = cuda(np.ascontiguousarray(plan.distance)) / rng.uniform(0.02, 0.04)
    elif not flow.inviscid:   # no wall distance: the normal index of the one block
        j = torch.arange(plan.shape[1], device="cuda", dtype=torch.float64)
        layer = (6.0 * (j - 1.5) / (plan.shape[1] - 4)).clamp(min=0.0).expand(tuple(plan.shape))
    if layer is not None:
        q[1:1 + dim] *= torch.tanh(layer)
        if flow.turbulence is not None:
            q[-1] = q[-1] * torch.tanh(layer * 50.0) + 100.0 * layer * torch.exp(1.0 - layer)
    speed = flow.mach
    for v in range(len(q_inf)):
        wave = torch.zeros_like(near)
        for _ in range(3):
            k = cuda(rng.uniform(-4.0, 4.0, dim)).reshape((-1,) + (1,) * dim)
            wave = wave + torch.sin((k * x).sum(0) + rng.uniform(0.0, 2.0 * math.pi)) / 3.0
        wave = 0.05 * near * wave
        if 1 <= v <= dim:
            q[v] = q[v] + speed * wave * (1.0 if layer is None else torch.tanh(layer))
        else:
            q[v] = q[v] * (1.0 + wave)
    free = freestream_state3(case, plan) if dim == 3 else freestream_state(case, plan)
    return torch.where(inside, _conservative(q, dim, flow.gamma), cuda(free)).contiguous()


def _noise(plan, nvar: int, dim: int, rng) -> torch.Tensor:
    """A rough vector on the block cells, as the Krylov vectors are."""
    gen = torch.Generator(device="cuda").manual_seed(int(rng.integers(1 << 31)))
    v = torch.randn((nvar,) + tuple(plan.shape), dtype=torch.float64, device="cuda", generator=gen)
    return torch.where(torch.as_tensor(np.ascontiguousarray(plan.interior), device="cuda"), v, 0.0).contiguous()


class _View:
    """A plan's own device state as an array another library can take without a copy."""

    def __init__(self, pointer: int, n: int):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f8", "data": (pointer, False), "version": 3,
                                         "strides": None}


def prepare(c: dict, seed: int):
    rng = np.random.default_rng([seed, 20261204])
    if c["grid"] == "wing":
        return _prepare3d(c, rng)
    from jaxrans_b200.batch import batch_device
    from jaxrans_b200.residual import make_residual
    from jaxrans_b200.solver import device_for
    alphas = [c["alpha"] + rng.uniform(-0.5, 0.5)]
    scales = [1]
    if c["angles"]:
        alphas = list(np.linspace(-4.0, 16.0, c["angles"]) + rng.uniform(-0.5, 0.5))
        scales = [1] * c["angles"]
        if c["uneven"]:
            alphas.append(c["alpha"])
            scales.append(2)
    cases = [_parse(c, float(a), s) for a, s in zip(alphas, scales)]
    plans = [_plan2d(c, s) for s in scales]
    state = {"case": c, "plans": plans, "cases": cases}
    U = [_state(p, k, 2, rng) for p, k in zip(plans, cases)]
    nvar = U[0].shape[0]
    if c["path"] in ("residual", "jvp"):
        op = make_residual(plans[0], cases[0].flow, cases[0].numerics, first_order=c["path"] == "jvp")
        state.update(operator=op, U=U[0])
    elif c["angles"]:
        state.update(device=batch_device(cases, plans), U=torch.cat([u.reshape(-1) for u in U]))
    else:
        state.update(device=device_for(cases[0], plans[0]), U=U[0])
    if c["path"] in ("jvp", "line"):
        state["v"] = _noise(plans[0], nvar, 2, rng)
    torch.cuda.synchronize()
    return state


def _prepare3d(c: dict, rng):
    from jaxrans_b200.solver3d import device3_for
    plan, area, length, centre = _plan3d(c)
    case = _parse(c, c["alpha"] + rng.uniform(-0.5, 0.5))
    state = {"case": c, "plans": [plan], "cases": [case], "device": device3_for(case, plan),
             "U": _state(plan, case, 3, rng), "forces": (area, length, np.array(centre, dtype=np.float64))}
    if c["path"] == "jvp":
        state["v"] = _noise(plan, 6, 3, rng)
    torch.cuda.synchronize()
    return state


# --- one pass -----------------------------------------------------------------------------------


def run(state):
    c = state["case"]
    if c["grid"] == "wing":
        return _run3d(state)
    U = state["U"]
    if c["path"] == "residual":
        return list(state["operator"].residual(U))
    if c["path"] == "jvp":
        return list(state["operator"].jvp(U, state["v"]))
    dev = state["device"]
    if c["path"] == "line":
        return list(dev.precondition(U, c["cfl"], state["v"]))
    dev.set_state_device(U, c["cfl"])
    history = dev.newton_steps(c["steps"])
    forces = dev.forces()
    with torch.cuda.stream(torch.cuda.ExternalStream(dev.stream_handle())):   # in the plan's own order
        flat = torch.as_tensor(_View(dev.state_device_ptr(), dev.n_vec), device="cuda").clone()
    rows = [r for k, shape in enumerate(dev.shapes)
            for r in flat[int(dev.offsets[k]):int(dev.offsets[k + 1])].reshape(shape)]
    return {"history": history, "forces": forces[..., :4], "state": rows}


def _run3d(state):
    """Through the C ABI: the 3D entry points take device pointers there."""
    from jaxrans_b200.native import NativeError
    import ctypes as C
    c, dev, U = state["case"], state["device"], state["U"]

    def call(name, *args):
        if getattr(dev.lib, name)(dev.handle, *args) != 0:
            raise NativeError(f"{name}: {dev.lib.jr_last_error().decode()}")

    if c["path"] == "residual":
        out = torch.empty_like(U)
        call("jr_residual3d", U.data_ptr(), out.data_ptr(), 0)
        return list(out)
    if c["path"] == "jvp":
        out = torch.empty_like(U)
        call("jr_jvp3d", U.data_ptr(), state["v"].data_ptr(), out.data_ptr())
        return list(out)
    u = U.clone()
    torch.cuda.current_stream().synchronize()   # the plan runs on a stream of its own
    cfl, norm, history = C.c_double(c["cfl"]), C.c_double(math.inf), np.zeros(c["steps"])
    call("jr_newton_steps3d", u.data_ptr(), c["steps"], C.byref(cfl), C.byref(norm), history.ctypes.data)
    area, length, centre = state["forces"]
    forces = np.zeros(4)
    call("jr_forces3d", u.data_ptr(), float(area), float(length), centre.ctypes.data, forces.ctypes.data)
    return {"history": history, "forces": forces, "state": list(u)}


# --- what a pass cannot do without ---------------------------------------------------------------


def _cells(c: dict) -> int:
    if c["grid"] == "wing":
        return 2 * (c["around"] // 2 + c["wake"]) * c["normal"] * (c["span"] + c["tip"])
    one = (c["around"] + 2 * c["wake"]) * c["normal"]
    return one * (max(1, c["angles"]) + (4 if c["uneven"] and c["angles"] else 0))


def work(c: dict) -> dict:
    """Compulsory bytes (inputs and grid tables read once, outputs written once, FP64) and
    operations.  A Newton step reads its linearised operator, its preconditioner's factor
    and its Krylov basis once per Arnoldi step; their smallest forms are counted: one cycle
    of GMRES, the basis and the vector read once per orthogonalisation, the operator's
    states and geometry, the chains' blocks."""
    dim = 3 if c["grid"] == "wing" else 2
    nvar = dim + 2 + (c["model"] == "sa")
    n = _cells(c)
    geometry = dim * dim + dim + 1 + (c["model"] == "sa")   # face vectors, centre, volume, wall distance
    flux = {"euler": 150, "laminar": 300, "sa": 450}[c["model"]] * dim * (2 if dim == 3 else 1)
    operator = 8.0 * n * (3 * nvar + geometry)
    if c["path"] == "residual":
        return {"bytes": 8.0 * n * (2 * nvar + geometry), "flops": float(n * flux)}
    if c["path"] == "jvp":
        return {"bytes": operator, "flops": 3.0 * n * flux}
    m = dim + 2
    block = 3 * m * m + (3 if c["model"] == "sa" else 0)
    b = 4.0 if c["precision"] == "mixed" else 8.0
    factor_bytes, apply_bytes = n * block * b, n * (block * b + 16.0 * nvar)
    line_flops = n * (2.0 * block + 4 * m)
    if c["path"] == "line":
        return {"bytes": 8.0 * n * (nvar + geometry) + factor_bytes + apply_bytes,
                "flops": n * 12.0 * m ** 3 + line_flops}
    k = c["subspace"]
    basis = 8.0 if dim == 3 else b   # the 3D basis is FP64 in both forms
    orth = sum((j + 2) * nvar * n * basis for j in range(k))
    step = (8.0 * n * (4 * nvar + geometry) + factor_bytes + k * (operator + apply_bytes) + orth)
    flops = n * flux * (1 + 3) + n * 12.0 * m ** 3 + k * (n * 10.0 * nvar * nvar * dim + line_flops) + \
        sum(8.0 * (j + 1) * nvar * n for j in range(k))
    return {"bytes": c["steps"] * step, "flops": c["steps"] * flops}


def tolerance(c: dict) -> dict:
    """About four times the largest change seen over the ranges when the last bit of half
    the state's entries is flipped (FP64), or between the mixed form and FP64 (mixed)."""
    mixed, sa = c["precision"] == "mixed", c["model"] == "sa"
    if c["path"] == "residual":   # net fluxes: differences of far larger face fluxes
        return {"rel": 1e-11, "max": 4e-10}
    if c["path"] == "jvp":        # the SA row's tangent: a small difference of large source terms
        return {"rel": 4e-9, "max": 6e-7} if sa else {"rel": 1e-12, "max": 1e-11}
    if c["path"] == "line":
        return {"rel": 1e-6, "max": 1e-5} if mixed else {"rel": 1e-12, "max": 1e-11}
    # a step's GMRES amplifies round-off by a few decades at the largest CFL numbers
    return {"rel": 1e-7, "max": 2e-6} if mixed else {"rel": 1e-10, "max": 1e-9}


# --- the operators in plain torch, FP64 -------------------------------------------------------------
# A restatement for checking: the residual (MUSCL, HLLC or Roe, the diamond gradients, the
# Newtonian stress, the SA row), its tangent by forward-mode differentiation and the line
# solve by block elimination, on the canvas tables of a plan.

_CB1, _SIGMA, _CB2, _KARMAN, _CW2, _CW3, _CV1 = 0.1355, 2.0 / 3.0, 0.622, 0.41, 0.3, 2.0, 7.1
_CW1 = _CB1 / _KARMAN ** 2 + (1.0 + _CB2) / _SIGMA
_PR, _PRT = 0.72, 0.9


def _pad(a, g: int, dim: int):
    for axis in range(a.dim() - dim, a.dim()):
        n = a.shape[axis]
        a = a.index_select(axis, torch.arange(-g, n + g, device=a.device).clamp(0, n - 1))
    return a


def _cut(a, axis: int, lo: int, n: int):
    return a.narrow(axis, lo, n)


def _dot(a, b):
    return (a * b).sum(0)


class _Model:
    """The tables of a plan and the physics of a case as torch tensors."""

    def __init__(self, plan, case):
        t = functools.partial(torch.as_tensor, device="cuda")

        def f(a):
            return t(np.ascontiguousarray(a), dtype=torch.float64)

        flow, num = case.flow, case.numerics
        self.dim = dim = 3 if getattr(plan, "dim", 2) == 3 else 2
        self.shape, self.gamma = tuple(plan.shape), flow.gamma
        self.flux, self.limiter, self.kappa = num.flux, num.limiter, num.kappa
        self.mu_inf = None if flow.inviscid else flow.mu_inf
        self.sutherland, self.sa = flow.sutherland_ratio, flow.turbulence is not None
        self.faces = [f(a) for a in (plan.faces if dim == 3 else (plan.faces_i, plan.faces_j))]
        self.centres, self.volume = f(plan.centres), f(plan.volume)
        self.interior = t(np.ascontiguousarray(plan.interior))
        self.distance = f(plan.distance) if plan.distance is not None else None
        self.neighbours = t(np.ascontiguousarray(plan.neighbours), dtype=torch.int64).reshape(-1)
        self.q_inf = f(_freestream(flow, dim))
        self.U_inf = _conservative(self.q_inf, dim, self.gamma)
        lines = plan.lines if dim == 3 else plan.chains
        self.lines = {k: t(np.ascontiguousarray(getattr(lines, k)), dtype=torch.int64)
                      for k in ("cells", "up_face", "up_sign", "down_face", "down_sign")}
        names = ("copy", "slip_wall", "no_slip_wall", "symmetry", "far_field")
        self.stages = []   # (gather index, [(kind, source, normal)])
        for st in plan.stages:
            if dim == 3:
                self.stages.append((t(st.index, dtype=torch.int64),
                                    [(k, t(s, dtype=torch.int64), f(n)) for k, s, n, _ in st.conditions]))
                continue
            index = np.arange(plan.n_canvas)
            index[st.ghost[st.kind == 0]] = st.source[st.kind == 0]
            rows, offset = [], plan.n_canvas
            for kind in np.unique(st.kind[st.kind != 0]):
                m = st.kind == kind
                index[st.ghost[m]] = offset + np.arange(int(m.sum()))
                offset += int(m.sum())
                rows.append((names[int(kind)], t(st.source[m], dtype=torch.int64), f(st.normal[:, m])))
            self.stages.append((t(index, dtype=torch.int64), rows))

    def primitive(self, U):
        d = self.dim
        v = U[1:1 + d] / U[0]
        p = (self.gamma - 1.0) * (U[1 + d] - 0.5 * U[0] * (v * v).sum(0))
        rows = [U[0:1], v, p[None]]
        return torch.cat(rows + [U[2 + d:] / U[0]]) if self.sa else torch.cat(rows)

    def temperature(self, q):
        return self.gamma * q[1 + self.dim] / q[0]

    def viscosity(self, T):
        s = self.sutherland
        return self.mu_inf * torch.ones_like(T) if s is None else self.mu_inf * T * T.sqrt() * (1.0 + s) / (T + s)

    # the ghosts
    def condition(self, kind, q, n):
        d, g = self.dim, self.gamma
        v, scalars = q[1:1 + d], q[2 + d:]
        if kind in ("slip_wall", "symmetry"):
            mirrored = v - 2.0 * _dot(v, n) * n
            return torch.cat([q[:1], mirrored, q[1 + d:2 + d], -scalars if kind == "slip_wall" else scalars])
        if kind == "no_slip_wall":
            return torch.cat([q[:1], -v, q[1 + d:2 + d], -scalars])
        f = self.q_inf[:, None].expand(q.shape)
        vf, pf, rf = f[1:1 + d], f[1 + d], f[0]
        p, r = q[1 + d], q[0]
        vn, vnf = _dot(v, n), _dot(vf, n)
        plus = vn + 2.0 / (g - 1.0) * (g * p / r).sqrt()
        minus = vnf - 2.0 / (g - 1.0) * (g * pf / rf).sqrt()
        vb, ab = 0.5 * (plus + minus), 0.25 * (g - 1.0) * (plus - minus)
        out = vb > 0.0
        s = torch.where(out, p / r ** g, pf / rf ** g)
        rb = (ab * ab / (g * s)) ** (1.0 / (g - 1.0))
        vel = vb * n + torch.where(out, v - vn * n, vf - vnf * n)
        return torch.cat([rb[None], vel, (rb * ab * ab / g)[None], torch.where(out, scalars, f[2 + d:])])

    def filled(self, q):
        flat = q.reshape(q.shape[0], -1)
        for index, rows in self.stages:
            parts = [flat] + [self.condition(k, flat[:, s], n) for k, s, n in rows]
            flat = torch.cat(parts, 1)[:, index]
        return flat.reshape(q.shape)

    # the inviscid flux
    def limited(self, a, b):
        if self.limiter == "none":
            return 0.5 * (a + b)
        if self.limiter == "van_albada_smooth":
            e = 1e-12
            return ((b * b + e) * a + (a * a + e) * b) / (a * a + b * b + 2.0 * e)
        same = a * b > 0.0
        if self.limiter == "minmod":
            return torch.where(same, torch.where(a.abs() < b.abs(), a, b), 0.0)
        return torch.where(same, a * b * (a + b) / torch.where(same, a * a + b * b, 1.0), 0.0)

    def normal_flux(self, q, n):
        d = self.dim
        v, p = q[1:1 + d], q[1 + d]
        vn = _dot(v, n)
        E = p / (self.gamma - 1.0) + 0.5 * q[0] * (v * v).sum(0)
        return torch.cat([(q[0] * vn)[None], q[0] * v * vn + p * n, ((E + p) * vn)[None]])

    def riemann(self, qL, qR, S):
        d, g = self.dim, self.gamma
        length = (S * S).sum(0).sqrt()
        n = S / length.clamp(min=1e-300)
        rl, rr, vl, vr, pl, pr = qL[0], qR[0], qL[1:1 + d], qR[1:1 + d], qL[1 + d], qR[1 + d]
        hl = g / (g - 1.0) * pl / rl + 0.5 * (vl * vl).sum(0)
        hr = g / (g - 1.0) * pr / rr + 0.5 * (vr * vr).sum(0)
        w = (rr / rl).sqrt()
        v, H = (vl + w * vr) / (1.0 + w), (hl + w * hr) / (1.0 + w)
        a = ((g - 1.0) * (H - 0.5 * (v * v).sum(0))).sqrt()
        vn, vnl, vnr = _dot(v, n), _dot(vl, n), _dot(vr, n)
        fl, fr = self.normal_flux(qL, n), self.normal_flux(qR, n)
        if self.flux == "roe":
            rho = (rl * rr).sqrt()
            dr, dp, dv = rr - rl, pr - pl, vr - vl
            dvn = _dot(dv, n)
            dvt = dv - dvn * n
            one, zero = torch.ones_like(rho)[None], torch.zeros_like(rho)[None]
            wave = ((vn - a).abs() * (dp - rho * a * dvn) / (2.0 * a * a) * torch.cat([one, v - a * n, (H - a * vn)[None]])
                    + vn.abs() * (dr - dp / (a * a)) * torch.cat([one, v, 0.5 * (v * v).sum(0)[None]])
                    + vn.abs() * rho * torch.cat([zero, dvt, _dot(v, dvt)[None]])
                    + (vn + a).abs() * (dp + rho * a * dvn) / (2.0 * a * a)
                    * torch.cat([one, v + a * n, (H + a * vn)[None]]))
            return length * (0.5 * (fl + fr) - 0.5 * wave)
        sl = torch.minimum(vnl - (g * pl / rl).sqrt(), vn - a)
        sr = torch.maximum(vnr + (g * pr / rr).sqrt(), vn + a)
        ml, mr = rl * (sl - vnl), rr * (sr - vnr)
        sm = (pr - pl + ml * vnl - mr * vnr) / (ml - mr)

        def star(q, vk, f, s, wide):
            r, vel, p = q[0], q[1:1 + d], q[1 + d]
            E = p / (g - 1.0) + 0.5 * r * (vel * vel).sum(0)
            ps, rs = p + r * (vk - s) * (vk - sm), r * (s - vk) / wide
            es = ((s - vk) * E - p * vk + ps * sm) / wide
            return f + s * (torch.cat([rs[None], rs * (vel + (sm - vk) * n), es[None]])
                            - torch.cat([r[None], r * vel, E[None]]))

        F = torch.where(sr >= 0.0, star(qR, vnr, fr, sr, sr - sm), fr)
        F = torch.where(sm >= 0.0, star(qL, vnl, fl, sl, sl - sm), F)
        return length * torch.where(sl >= 0.0, fl, F)

    # gradients
    def sides(self, p1, a):
        """Cells before and after every face of family a, of a field with one ghost ring."""
        lead = p1.dim() - self.dim
        for b in range(self.dim):
            if b != a:
                p1 = _cut(p1, lead + b, 1, self.shape[b])
        n = self.shape[a] + 1
        return _cut(p1, lead + a, 0, n), _cut(p1, lead + a, 1, n)

    def nodes(self, a):
        for axis in range(a.dim() - self.dim, a.dim()):
            n = a.shape[axis] - 1
            a = 0.5 * (_cut(a, axis, 0, n) + _cut(a, axis, 1, n))
        return a

    def gradients(self, phi, a):
        """(dim, nphi, face): the linear field through the two cells' difference and the
        face's node differences (its edge in 2D, its two diagonals in 3D)."""
        others = [b for b in range(self.dim) if b != a]

        def corner(field, shifts):
            for b, s in zip(others, shifts):
                field = _cut(field, field.dim() - self.dim + b, s, self.shape[b])
            return field

        xn, pn = self.nodes(self.centres), self.nodes(phi)
        (xl, xh), (fl, fh) = self.sides(self.centres, a), self.sides(phi, a)
        d1, p1 = xh - xl, fh - fl
        if self.dim == 2:
            d2, p2 = corner(xn, (1,)) - corner(xn, (0,)), corner(pn, (1,)) - corner(pn, (0,))
            det = d1[0] * d2[1] - d2[0] * d1[1]
            return torch.stack([(p1 * d2[1] - p2 * d1[1]) / det, (d1[0] * p2 - d2[0] * p1) / det])
        d2, p2 = (corner(f, (1, 1)) - corner(f, (0, 0)) for f in (xn, pn))
        d3, p3 = (corner(f, (0, 1)) - corner(f, (1, 0)) for f in (xn, pn))
        c23, c31, c12 = (torch.linalg.cross(x, y, dim=0) for x, y in ((d2, d3), (d3, d1), (d1, d2)))
        return (p1 * c23[:, None] + p2 * c31[:, None] + p3 * c12[:, None]) / _dot(d1, c23)

    def green_gauss(self, values):
        """(dim, ...) gradients of a field from its values on the faces, one per family."""
        return torch.stack([self.divergence([v * S[c] for v, S in zip(values, self.faces)]) / self.volume
                            for c in range(self.dim)])

    def divergence(self, fluxes):
        total = 0.0
        for a, F in enumerate(fluxes):
            axis = F.dim() - self.dim + a
            n = F.shape[axis] - 1
            total = total + _cut(F, axis, 1, n) - _cut(F, axis, 0, n)
        return total

    # the SA model
    def eddy(self, q, mu):
        nut = q[-1] * self.mu_inf
        chi3 = (torch.where(nut > 0.0, nut, 0.0) * q[0] / mu) ** 3
        return torch.where(nut > 0.0, q[0] * nut * chi3 / (chi3 + _CV1 ** 3), 0.0)

    def sa_diffusivity(self, q, mu):
        nut = q[-1] * self.mu_inf
        chi3 = torch.where(nut >= 0.0, 0.0, (nut * q[0] / mu) ** 3)
        return (mu + q[0] * nut * torch.where(nut >= 0.0, 1.0, (16.0 + chi3) / (16.0 - chi3))) / _SIGMA

    def s_tilde(self, omega, nut, nu):
        chi = nut / nu
        fv1 = chi ** 3 / (chi ** 3 + _CV1 ** 3)
        bar = nut * (1.0 - chi / (1.0 + chi * fv1)) / (_KARMAN * self.distance) ** 2
        usual = bar >= -0.7 * omega
        den = torch.where(usual, 1.0, (0.9 - 1.4) * omega - bar)
        return torch.where(usual, omega + bar, omega + omega * (0.49 * omega + 0.9 * bar) / den)

    def f_w(self, nut, st):
        den = st * (_KARMAN * self.distance) ** 2
        ok = den > 0.0
        r = torch.where(ok, nut / torch.where(ok, den, 1.0), 10.0).clamp(max=10.0)
        gg = r + _CW2 * (r ** 6 - r)
        return gg * ((1.0 + _CW3 ** 6) / (gg ** 6 + _CW3 ** 6)) ** (1.0 / 6.0)

    def vorticity(self, gx):
        if self.dim == 2:
            return (gx[0, 1] - gx[1, 0]).abs()
        curl = torch.stack([gx[1, 2] - gx[2, 1], gx[2, 0] - gx[0, 2], gx[0, 1] - gx[1, 0]])
        square = (curl * curl).sum(0)
        return torch.where(square > 0.0, torch.where(square > 0.0, square, 1.0).sqrt(), 0.0)

    def sa_source(self, p1):
        d = self.dim
        mean = [0.5 * (lo + hi) for lo, hi in (self.sides(p1, a) for a in range(d))]
        cell = p1
        for b in range(d):
            cell = _cut(cell, 1 + b, 1, self.shape[b])
        omega = self.vorticity(self.green_gauss([m[1:1 + d] for m in mean]))
        grad = self.green_gauss([m[-1] for m in mean])
        nut = cell[-1] * self.mu_inf
        nu = self.viscosity(self.temperature(cell)) / cell[0]
        pos = nut >= 0.0
        st = self.s_tilde(omega, torch.where(pos, nut, 0.0), nu)
        production = torch.where(pos, _CB1 * st, _CB1 * omega) * nut
        destruction = torch.where(pos, _CW1 * self.f_w(nut, st), -_CW1) * (nut / self.distance) ** 2
        return self.volume * cell[0] * ((production - destruction) / self.mu_inf
                                        + _CB2 / _SIGMA * self.mu_inf * (grad * grad).sum(0))

    def residual(self, U, first_order: bool):
        d, g = self.dim, self.gamma
        padded = _pad(self.filled(self.primitive(U)), 2, d)
        p1 = padded
        for b in range(d):
            p1 = _cut(p1, 1 + b, 1, self.shape[b] + 2)
        fluxes = []
        for a in range(d):
            cells = padded[:2 + d]
            for b in range(d):
                if b != a:
                    cells = _cut(cells, 1 + b, 2, self.shape[b])
            mm, m, p, pp = (_cut(cells, 1 + a, o, self.shape[a] + 1) for o in range(4))
            if first_order:
                qL, qR = m, p
            elif self.kappa != 0.0:
                lo, hi = 0.25 * (1.0 - self.kappa), 0.25 * (1.0 + self.kappa)
                qL, qR = m + lo * (m - mm) + hi * (p - m), p - lo * (pp - p) - hi * (p - m)
            else:
                qL, qR = m + 0.5 * self.limited(m - mm, p - m), p - 0.5 * self.limited(p - m, pp - p)
            S = self.faces[a]
            F = self.riemann(qL, qR, S)
            if self.mu_inf is not None:
                lo, hi = self.sides(p1, a)
                mean = 0.5 * (lo + hi)
                T = 0.5 * (self.temperature(lo) + self.temperature(hi))
                mu = self.viscosity(T)
                k = mu / (_PR * (g - 1.0))
                phi = [p1[1:1 + d], self.temperature(p1)[None]] + ([p1[-1:]] if self.sa else [])
                G = self.gradients(torch.cat(phi), a)
                if self.sa:
                    mu_f = self.viscosity(self.temperature(mean))
                    mut = self.eddy(mean, mu_f)
                    up = torch.where(F[0] > 0.0, lo[-1], hi[-1])
                    row = F[0] * up - self.sa_diffusivity(mean, mu_f) * _dot(G[:, -1], S)
                    mu, k = mu + mut, k + mut / (_PRT * (g - 1.0))
                div = sum(G[b, b] for b in range(d))
                force = torch.stack([mu * (sum((G[b, c] + G[c, b]) * S[b] for b in range(d)) - 2.0 / 3.0 * div * S[c])
                                     for c in range(d)])
                energy = _dot(mean[1:1 + d], force) + k * _dot(G[:, d], S)
                F = F - torch.cat([torch.zeros_like(energy)[None], force, energy[None]])
                if self.sa:
                    F = torch.cat([F, row[None]])
            fluxes.append(F)
        R = self.divergence(fluxes)
        if self.sa:
            R = torch.cat([R[:-1], (R[-1] - self.sa_source(p1))[None]])
        outside = U - self.U_inf.reshape((-1,) + (1,) * d)
        return torch.where(self.interior, R, outside)

    # the line preconditioner
    def face_means(self, f):
        lead = f.dim() - self.dim
        f = f.reshape(f.shape[:lead] + (-1,))[..., self.neighbours].reshape(f.shape)
        padded, out = _pad(f, 1, self.dim), []
        for a in range(self.dim):
            lo, hi = self.sides(padded, a)
            out.append(0.5 * (lo + hi))
        return out

    def cell_sum(self, values):
        total = 0.0
        for a, v in enumerate(values):
            total = total + _cut(v, a, 0, self.shape[a]) + _cut(v, a, 1, self.shape[a])
        return total

    def line_solve(self, U, cfl: float, r, coupled: bool):
        d, g, m = self.dim, self.gamma, self.dim + 2
        q = self.primitive(U)
        means, vols = self.face_means(q), self.face_means(self.volume)
        lam, mass, diff = [], [], []
        for f, S, vol in zip(means, self.faces, vols):
            ss, vn = (S * S).sum(0), _dot(f[1:1 + d], S)
            speed = vn.abs() + (g * f[1 + d] / f[0]).sqrt() * ss.sqrt()
            if self.mu_inf is not None:
                mu = self.viscosity(self.temperature(f))
                total = mu + self.eddy(f, mu) if self.sa else mu
                speed = speed + 2.0 * g / _PR * total * ss / (f[0] * vol)
                if self.sa:
                    mass.append(f[0] * vn)
                    diff.append(self.sa_diffusivity(f, mu) * ss / vol)
            lam.append(speed)
        ln = self.lines
        valid = ln["cells"] >= 0
        cells = ln["cells"].clamp(min=0)
        L = cells.shape[1]

        def on_lines(field):
            return field.reshape(field.shape[:field.dim() - d] + (-1,))[..., cells]

        def on_faces(fields, side):
            flat = torch.cat([x.reshape(x.shape[:x.dim() - d] + (-1,)) for x in fields], -1)
            return flat[..., ln[side + "_face"]]

        def jacobian(nb, S):
            cons = _conservative(nb[:m], d, g)
            cols = []
            for k in range(m):
                e = torch.zeros_like(cons)
                e[k] = 1.0

                def flux(u):
                    v = u[1:1 + d] / u[0]
                    p = (g - 1.0) * (u[1 + d] - 0.5 * u[0] * (v * v).sum(0))
                    return self.normal_flux(torch.cat([u[:1], v, p[None]]), S)
                cols.append(torch.func.jvp(flux, (cons,), (e,))[1])
            return torch.stack(cols, 1).permute(3, 2, 0, 1)   # (L, lines, row, variable)

        eye = torch.eye(m, dtype=torch.float64, device=U.device)
        on = on_lines(q)
        above = torch.cat([on[:, :, 1:], on[:, :, -1:]], 2)

        def side(which, nb):
            sign = ln[which + "_sign"].double()
            S, l = on_faces(self.faces, which), on_faces(lam, which)
            block = 0.5 * jacobian(nb, sign * S) - 0.5 * l.t()[..., None, None] * eye
            return torch.where((sign != 0).t()[..., None, None], block, 0.0)

        def shifted(x):
            return torch.cat([torch.zeros_like(x[:1]), x[:-1]])

        diag = torch.where(valid, on_lines(self.cell_sum(lam) * (1.0 / cfl + 0.5)), 1.0).t()[..., None, None] * eye
        upper, lower = side("up", above), shifted(side("down", on))

        def eliminate(lo, di, up, rhs):
            C, D = [], []
            for k in range(L):
                P = di[k] if k == 0 else di[k] - lo[k] @ C[-1]
                b = rhs[k] if k == 0 else rhs[k] - (lo[k] @ D[-1][..., None])[..., 0]
                both = torch.linalg.solve(P, torch.cat([up[k], b[..., None]], -1))
                C.append(both[..., :-1])
                D.append(both[..., -1])
            for k in range(L - 2, -1, -1):
                D[k] = D[k] - (C[k] @ D[k + 1][..., None])[..., 0]
            return torch.stack(D)

        z = r.clone().reshape(r.shape[0], -1)
        rhs = torch.where(valid, on_lines(r), 0.0)
        x = eliminate(lower, diag, upper, rhs[:m].permute(2, 1, 0))
        z[:m, cells[valid]] = x.permute(2, 1, 0)[:, valid]
        if self.sa:
            rho = on_lines(q[0])
            dg = 0.0
            for a, (mf, df) in enumerate(zip(mass, diff)):
                n = self.shape[a]
                dg = dg + _cut(mf.clamp(min=0.0) + df, a, 1, n) + _cut((-mf).clamp(min=0.0) + df, a, 0, n)
            omega = self.vorticity(self.green_gauss([f[1:1 + d] for f in means]))
            nut = q[-1] * self.mu_inf
            nu = self.viscosity(self.temperature(q)) / q[0]
            fw = self.f_w(nut, self.s_tilde(omega, nut, nu))
            dest = torch.where(nut > 0.0, 2.0 * _CW1 * fw * nut / self.distance ** 2, 0.0)
            dg = dg / q[0] + dest * self.volume + self.cell_sum(lam) / cfl
            dg = torch.where(valid, on_lines(dg), 1.0).t()[..., None, None]

            def scalar(which, rho_nb):
                sign = ln[which + "_sign"].double()
                b = -((-sign * on_faces(mass, which)).clamp(min=0.0) + on_faces(diff, which)) / rho_nb
                return torch.where(sign != 0, b, 0.0).t()[..., None, None]

            def flow_coupling(which, nb):   # half the Jacobian of rho nu V.S in the neighbour's mean flow
                S = ln[which + "_sign"].double() * on_faces(self.faces, which)
                row = torch.cat([-_dot(nb[1:1 + d], S)[None], S, torch.zeros_like(S[:1])])
                return (0.5 * nb[-1] * row).permute(2, 1, 0)

            us = scalar("up", torch.cat([rho[:, 1:], rho[:, -1:]], 1))
            ls = shifted(scalar("down", rho))
            b = rhs[-1].t()
            if coupled:
                up, low = flow_coupling("up", above), shifted(flow_coupling("down", on))
                nxt = torch.cat([x[1:], torch.zeros_like(x[:1])])
                b = b - (up * nxt).sum(-1) - (low * shifted(x)).sum(-1)
            y = eliminate(ls, dg, us, b[..., None])[..., 0]
            z[-1, cells[valid]] = y.t()[valid]
        return z.reshape(r.shape)


def exact(c: dict, seed: int):
    """What ``run`` returns, in plain torch FP64; None for the marches (a Newton step's
    inexact solve is defined by its iterations, and takes too long here)."""
    if c["path"] == "newton":
        return None
    # the inputs are prepare's own
    state = prepare(c, seed)
    model, U = _Model(state["plans"][0], state["cases"][0]), state["U"]
    if c["path"] == "residual":
        return list(model.residual(U, False))
    if c["path"] == "jvp":
        return list(torch.func.jvp(lambda u: model.residual(u, True), (U,), (state["v"],))[1])
    return list(model.line_solve(U, c["cfl"], state["v"], c["preconditioner"] == "line_j_coupled"))
