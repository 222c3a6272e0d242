"""The FP64 kernels that take one of two forms by how many cases a launch holds: the J.v tile
(coefficients loaded ahead while every tile is resident, or where they are used) and the
orthogonalisation (a thread's vectors in registers, or a warp a vector), and the linearisation's
two instances (QCR2000's stress in the launch or not).  A case's history and
state are bitwise the same whichever form its launch took, for each model's instances, on grids
whose edges cut the tiles and the blocks' parts, and for every number of vectors a form has its
own kernel for."""

from __future__ import annotations

from dataclasses import replace

import numpy as np
import pytest

from jaxrans_b200.case import parse_case
from jaxrans_b200.solver import freestream_state

pytestmark = pytest.mark.gpu

CASES = 6   # 6 x 76 tiles of the J.v and 6 x 53 blocks of the basis: more than are resident at once


@pytest.mark.parametrize("model,subspace", [("euler", 8), ("euler", 10), ("euler", 33), ("laminar", 10), ("sa", 20)])
def test_a_batch_past_the_rule_is_bitwise_the_cases_alone(cuda, model, subspace):
    from jaxrans_b200.native import DevicePlan
    case = o_grid(model, subspace)
    plan = case.grid()
    flows = [replace(case.flow, alpha_deg=float(a)) for a in np.linspace(-2.0, 4.0, CASES)]
    compare(DevicePlan, case, plan, flows)


def test_a_batch_with_a_qcr_case_is_bitwise_the_cases_alone(cuda):
    from jaxrans_b200.native import DevicePlan
    case = o_grid("sa", 12)
    flows = [case.flow, replace(case.flow, turbulence="sa_noft2_qcr"), replace(case.flow, alpha_deg=4.0)]
    compare(DevicePlan, case, case.grid(), flows)


def o_grid(model, subspace):
    euler = model == "euler"
    return parse_case({"general": {"case_name": "forms"},
                       "domain": {"grid": "o_grid", "airfoil": "naca0012", "cells_airfoil": 126, "cells_normal": 46,
                                  "wall_spacing": 1e-3, "far_field": 20.0},
                       "boundary_conditions": {"wall": {"type": "slip_wall" if euler else "no_slip_wall"},
                                               "farfield": {"type": "far_field"}},
                       "freestream": {"mach": 0.5, "alpha_deg": 2.0, **({} if euler else {"reynolds": 1e5})},
                       **({"turbulence": {"model": "sa_noft2"}} if model == "sa" else {})},
                      {"convective_fluxes": {"riemann_solver": "hllc", "limiter": "van_albada"},
                       "time_integration": {"solver": "implicit"},
                       "implicit": {"krylov_subspace": subspace, "krylov_restarts": 1, "max_relative_update": 0.2}})


def compare(DevicePlan, case, plan, flows):
    states = [freestream_state(replace(case, flow=f), plan) for f in flows]
    batch = DevicePlan.batch(plan, flows, case.numerics, case.implicit)
    batch.set_state(np.concatenate([u.ravel() for u in states]), 5.0)
    hist = batch.newton_steps(4)
    for k in (0, 1, len(flows) - 1):
        one = DevicePlan(plan, flows[k], case.numerics, case.implicit)
        one.set_state(states[k], 5.0)
        assert np.array_equal(hist[:, k], one.newton_steps(4))
        assert np.array_equal(batch.case_state(k)[0], one.get_state()[0])
        one.close()
    assert not np.array_equal(hist[:, 0], hist[:, 1])   # (the cases differ)
    batch.close()


@pytest.mark.parametrize("cases,far", [(2, "freestream"), (9, "freestream"), (9, "point_vortex")])
def test_a_batch_residual_is_bitwise_the_cases_alone(cuda, cases, far):
    """The residual entry point's two ghost fills: by the tiles (few ghosts: 704 a case) or by a
    launch (many, or a point-vortex far field; here in one case of the batch)."""
    from jaxrans_b200.native import DevicePlan
    case = o_grid("euler", 10)
    plan = case.grid()
    flows = [replace(case.flow, alpha_deg=float(a)) for a in np.linspace(-2.0, 4.0, cases)]
    nums = [case.numerics] * cases
    if far == "point_vortex":
        nums[1] = replace(case.numerics, far_field="characteristic_point_vortex")
    rng = np.random.default_rng(5)
    states = [freestream_state(replace(case, flow=f), plan) for f in flows]
    states = [np.where(plan.interior, u * (1.0 + 0.02 * rng.uniform(-1.0, 1.0, u.shape)), u) for u in states]
    batch = DevicePlan.batch([plan] * cases, flows, nums, [case.implicit] * cases)
    for first in (False, True):
        got = batch.residual(np.concatenate([u.ravel() for u in states]), first_order=first)
        for k in (0, 1, cases - 1):
            one = DevicePlan(plan, flows[k], nums[k], case.implicit)
            ref = one.residual(states[k], first_order=first)
            one.close()
            assert np.array_equal(got[k * ref.size:(k + 1) * ref.size], ref.ravel())
    batch.close()
