"""The 3D line solve's kernels (four chains a warp, eight lanes a chain) against the oracle's,
on grids whose chain counts leave every remainder of a warp's four, chains of odd lengths, in
each form: mean flow only, split and coupled SA, FP64 and FP32."""

from __future__ import annotations

import numpy as np
import pytest

from jaxrans_b200.config import FlowConditions, ImplicitConfig, freestream_primitive3
from jaxrans_b200.geometry import section_source
from jaxrans_b200.grid3d import wing_block
from jaxrans_b200.plan3d import build_plan3d

pytestmark = pytest.mark.gpu

# cells round the airfoil, in each wake half, normal, along the span (the wake's chains run
# through the cut: twice the normal cells)
SIZES = [(24, 6, 10, 4), (26, 8, 11, 5), (28, 8, 12, 3), (26, 8, 13, 9)]


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("model,preconditioner", [("euler", "line_j"), ("sa", "line_j"), ("sa", "line_j_coupled")])
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-10), ("mixed", 1e-4)])   # the solves' bounds on the fixtures
def test_line_solve_matches_the_oracle(cuda, size, model, preconditioner, precision, tol):
    from jaxrans_b200.native3d import DevicePlan3
    from oracle import implicit3d as i3
    from oracle import numerics3d as n3
    block = wing_block(section_source("naca0012"), *size, wall_spacing=1e-3, far_field=20.0, semispan=2.0, taper=0.6,
                       sweep_deg=25.0)
    plan = build_plan3d([block.with_kinds({"wall": "slip_wall" if model == "euler" else "no_slip_wall",
                                           "farfield": "far_field", "root": "symmetry", "tip": "symmetry"})])
    flow = FlowConditions(mach=0.6, alpha_deg=2.5, reynolds=None if model == "euler" else 1e5,
                          turbulence="sa_noft2" if model == "sa" else None)
    q_inf = np.array(freestream_primitive3(flow))
    mu = None if model == "euler" else flow.mu_inf
    oracle = n3.Model3(plan, q_inf, flow.gamma, "hllc", "minmod", 0.0, mu, None, model == "sa", plan.distance)
    rng = np.random.default_rng(11)
    U = n3.initial_state(oracle)
    U = U * (1.0 + 0.02 * rng.uniform(-1.0, 1.0, U.shape))
    r = rng.standard_normal(U.shape)
    solve = i3.precondition if preconditioner == "line_j" else i3.precondition_coupled
    ref = solve(U, n3.wave_speeds(U, oracle), 40.0, oracle)(r)
    dev = DevicePlan3(plan, q_inf, flow.gamma, "hllc", "minmod", 0.0, mu, None,
                      ImplicitConfig(preconditioner=preconditioner, precision=precision))
    try:
        z = dev.precondition(U, 40.0, r)
    finally:
        dev.close()
    for v in range(U.shape[0]):
        assert np.abs(z[v] - ref[v]).max() <= tol * np.abs(ref[v]).max(), v
