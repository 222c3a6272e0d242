"""The linearised 3D J.v (linearize3d.cu) and the one-launch ghost fill, through Newton steps
on canvases whose sizes leave every remainder of its 4 x 8 x 8 tiles and 8-face rows, for
each model it has factors for, against the oracle's step (complex-step J.v)."""

from __future__ import annotations

import numpy as np
import pytest

from jaxrans_b200.config import FlowConditions, ImplicitConfig, freestream_primitive3
from jaxrans_b200.geometry import section_source
from jaxrans_b200.grid3d import wing_block
from jaxrans_b200.plan3d import build_plan3d

pytestmark = pytest.mark.gpu

# cells round the airfoil, in each wake half, normal, along the span: canvas sizes (NI, NJ,
# NK) modulo the tile are (0, 6, 0), (2, 7, 1), (0, 0, 7), (2, 5, 5)
SIZES = [(24, 6, 10, 4), (26, 8, 11, 5), (28, 8, 12, 3), (26, 8, 13, 9)]
# model, QCR2000's constant, flux
MODELS = [("euler", 0.0, "hllc"), ("laminar", 0.0, "roe"), ("sa", 0.0, "hllc"), ("sa", 0.3, "roe")]


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("model,c_cr1,flux", MODELS)
def test_newton_step_matches_the_oracle(cuda, size, model, c_cr1, flux):
    from jaxrans_b200.native3d import DevicePlan3
    from oracle import implicit as im
    from oracle import implicit3d as i3
    from oracle import numerics3d as n3
    wall = "slip_wall" if model == "euler" else "no_slip_wall"
    block = wing_block(section_source("naca0012"), *size, wall_spacing=1e-3, far_field=20.0, semispan=2.0, taper=0.6,
                       sweep_deg=25.0)
    plan = build_plan3d([block.with_kinds({"wall": wall, "farfield": "far_field", "root": "symmetry",
                                           "tip": "symmetry"})])
    flow = FlowConditions(mach=0.6, alpha_deg=2.5, reynolds=None if model == "euler" else 1e5,
                          turbulence="sa_noft2" if model == "sa" else None)
    q_inf = np.array(freestream_primitive3(flow))
    mu = None if model == "euler" else flow.mu_inf
    imp = ImplicitConfig(krylov_subspace=5, krylov_restarts=1, max_relative_update=0.2)
    oracle = n3.Model3(plan, q_inf, flow.gamma, flux, "van_albada_smooth", 0.0, mu, None, model == "sa", plan.distance,
                       c_cr1)
    rng = np.random.default_rng(7)
    U = n3.initial_state(oracle)
    U = np.where(plan.interior, U * (1.0 + 0.02 * rng.uniform(-1.0, 1.0, U.shape)), U)
    U[2] = np.where(plan.interior, 0.05 * rng.uniform(-1.0, 1.0, plan.shape), U[2])   # off V.n = 0, a kink
    step, norm = i3.newton_step(im.NewtonState(U, 10.0, np.inf), oracle, imp)
    dev = DevicePlan3(plan, q_inf, flow.gamma, flux, "van_albada_smooth", 0.0, mu, None, imp, c_cr1=c_cr1)
    try:
        got, cfl, _, hist = dev.newton_steps(U, 1, 10.0)
    finally:
        dev.close()
    assert np.isclose(hist[0], norm, rtol=1e-12, atol=0.0) and cfl == step.cfl
    # the products agree to 1e-10 of their largest entry (the SA row's, a difference of far
    # larger sources); five Arnoldi steps amplify that by at most a few tens
    for v in range(U.shape[0]):
        d, ref = got[v] - U[v], step.U[v] - U[v]
        assert np.abs(d - ref).max() <= 1e-8 * np.abs(ref).max(), v
