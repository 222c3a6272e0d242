"""The FP64 orthogonalisation passes through Newton steps against the oracle's: subspaces either
side of every register form (8, 16, 32 vectors a thread, then slices) and cases whose size
leaves blocks and threads short of elements."""

from __future__ import annotations

import numpy as np
import pytest

from jaxrans_b200.case import parse_case
from jaxrans_b200.config import freestream_primitive

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("around,normal", [(24, 11), (64, 24)])   # 1,680 and 7,616 unknowns
@pytest.mark.parametrize("subspace", [1, 8, 9, 17, 33, 64])
def test_newton_step_matches_the_oracle(cuda, around, normal, subspace):
    from jaxrans_b200.native import DevicePlan
    from oracle import implicit as im
    from oracle import numerics as nm
    case = parse_case({"general": {"case_name": "orth"},
                       "domain": {"grid": "o_grid", "airfoil": "naca0012", "cells_airfoil": around,
                                  "cells_normal": normal, "wall_spacing": 2e-2, "far_field": 20.0},
                       "boundary_conditions": {"wall": {"type": "slip_wall"}, "farfield": {"type": "far_field"}},
                       "freestream": {"mach": 0.5, "alpha_deg": 2.0}},
                      {"convective_fluxes": {"riemann_solver": "hllc", "limiter": "van_albada"},
                       "time_integration": {"solver": "implicit"},
                       "implicit": {"krylov_subspace": subspace, "krylov_restarts": 1}})
    plan, flow = case.grid(), case.flow
    model = nm.Model(plan, np.array(freestream_primitive(flow)), flow.gamma, "hllc", "van_albada", 0.0, None, None,
                     False, 0.0, "characteristic", None)
    rng = np.random.default_rng(5)
    U = nm.initial_state(model)
    U = np.where(plan.interior, U * (1.0 + 0.02 * rng.uniform(-1.0, 1.0, U.shape)), U)
    step, norm = im.newton_step(im.NewtonState(U, 20.0, np.inf), model, case.implicit)
    dev = DevicePlan(plan, flow, case.numerics, case.implicit)
    try:
        dev.set_state(U, 20.0)
        hist = dev.newton_steps(1)
        got = dev.get_state()[0]
    finally:
        dev.close()
    assert np.isclose(hist[0], norm, rtol=1e-12, atol=0.0)
    for v in range(4):   # products within 1e-12 of their largest entry, amplified over the cycle
        d, ref = got[v] - U[v], step.U[v] - U[v]
        assert np.abs(d - ref).max() <= 1e-8 * np.abs(ref).max(), v
