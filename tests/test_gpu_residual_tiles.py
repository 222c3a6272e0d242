"""The residual entry point against the oracle on grids whose edges cut the 7 x 16 tiles at
different places: the tiles evaluate the ghosts of their halos (two layers, the corners of
both stages, the wake cut of a C-grid), and a point-vortex far field has them filled."""

from __future__ import annotations

import numpy as np
import pytest

from jaxrans_b200.case import parse_case
from jaxrans_b200.config import freestream_primitive

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first_order", [False, True])
@pytest.mark.parametrize("model", ["freestream", "point_vortex"])
@pytest.mark.parametrize("grid,around,normal", [("o_grid", 24, 12), ("o_grid", 30, 14), ("o_grid", 66, 17),
                                                ("c_grid", 24, 12), ("c_grid", 40, 29)])
def test_residual_matches_the_oracle(cuda, grid, around, normal, model, first_order):
    from jaxrans_b200.native import DevicePlan
    from oracle import numerics as nm
    domain = {"grid": grid, "airfoil": "naca0012", "cells_airfoil": around, "cells_normal": normal,
              "wall_spacing": 2e-2, "far_field": 20.0}
    if grid == "c_grid":
        domain["cells_wake"] = around // 2
    case = parse_case({"general": {"case_name": "tiles"}, "domain": domain,
                       "boundary_conditions": {"wall": {"type": "slip_wall"},
                                               "farfield": {"type": "far_field", "model": model}},
                       "freestream": {"mach": 0.5, "alpha_deg": 2.0}},
                      {"convective_fluxes": {"riemann_solver": "hllc", "limiter": "van_albada"},
                       "time_integration": {"solver": "implicit"}})
    plan, flow = case.grid(), case.flow
    far = "characteristic" if model == "freestream" else "characteristic_point_vortex"
    oracle = nm.Model(plan, np.array(freestream_primitive(flow)), flow.gamma, "hllc", "van_albada", far_field=far)
    rng = np.random.default_rng(5)
    U = nm.initial_state(oracle)
    U = np.where(plan.interior, U * (1.0 + 0.02 * rng.uniform(-1.0, 1.0, U.shape)), U)
    ref = nm.residual(U, oracle, first_order)
    dev = DevicePlan(plan, flow, case.numerics, case.implicit)
    try:
        got = [dev.residual(U, first_order=first_order) for _ in range(2)]
    finally:
        dev.close()
    assert np.array_equal(got[0], got[1])
    for v in range(4):   # a few hundred roundings a cell, against the sums' largest entry
        assert np.abs(got[0][v] - ref[v]).max() <= 1e-12 * np.abs(ref[v]).max(), v
