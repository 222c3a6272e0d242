"""The 3D Newton step's two matrix-vector products -- the stored linearisation and, without the
memory for its factors, the dual-number kernels: each against the oracle's step, the caller's
limit, what a plan reports, and the factors given back where another plan needs the memory."""

from __future__ import annotations

import numpy as np
import pytest

from jaxrans_b200.config import FlowConditions, ImplicitConfig, freestream_primitive3
from jaxrans_b200.geometry import section_source
from jaxrans_b200.grid3d import wing_block
from jaxrans_b200.plan3d import build_plan3d

pytestmark = pytest.mark.gpu


def wing(model, sutherland, size):
    block = wing_block(section_source("naca0012"), *size, wall_spacing=1e-3, far_field=20.0, semispan=2.0, taper=0.6,
                       sweep_deg=25.0)
    plan = build_plan3d([block.with_kinds({"wall": "slip_wall" if model == "euler" else "no_slip_wall",
                                           "farfield": "far_field", "root": "symmetry", "tip": "symmetry"})])
    flow = FlowConditions(mach=0.6, alpha_deg=2.5, reynolds=None if model == "euler" else 1e5,
                          turbulence="sa_noft2" if model == "sa" else None)
    q_inf = np.array(freestream_primitive3(flow))
    mu = None if model == "euler" else flow.mu_inf
    args = (plan, q_inf, flow.gamma, "hllc", "van_albada_smooth", 0.0, mu, sutherland)
    return args, ImplicitConfig(krylov_subspace=5, krylov_restarts=1, max_relative_update=0.2)


def state(args, model):
    from oracle import numerics3d as n3
    plan = args[0]
    oracle = n3.Model3(*args, model == "sa", plan.distance)
    rng = np.random.default_rng(7)
    U = n3.initial_state(oracle)
    U = np.where(plan.interior, U * (1.0 + 0.02 * rng.uniform(-1.0, 1.0, U.shape)), U)
    U[2] = np.where(plan.interior, 0.05 * rng.uniform(-1.0, 1.0, plan.shape), U[2])   # off V.n = 0, a kink
    return oracle, U


@pytest.mark.parametrize("model,sutherland", [("euler", None), ("laminar", 0.38), ("sa", 0.38)])
def test_both_products_match_the_oracle(cuda, model, sutherland):
    from jaxrans_b200.native import JR_PRODUCT_DUAL, JR_PRODUCT_LINEARISED, JR_PRODUCT_NONE
    from jaxrans_b200.native3d import DevicePlan3
    from oracle import implicit as im
    from oracle import implicit3d as i3
    args, imp = wing(model, sutherland, (26, 8, 11, 5))
    oracle, U = state(args, model)
    step, norm = i3.newton_step(im.NewtonState(U, 10.0, np.inf), oracle, imp)
    dev = DevicePlan3(*args, imp)
    try:
        assert dev.product()[0] == JR_PRODUCT_NONE
        got = {}
        size = dev.product()[1]
        for limit, form in ((None, JR_PRODUCT_LINEARISED), (size - 1, JR_PRODUCT_DUAL), (0, JR_PRODUCT_DUAL),
                            (size, JR_PRODUCT_LINEARISED), (None, JR_PRODUCT_LINEARISED)):
            dev.product_limit(limit)
            new, cfl, _, hist = dev.newton_steps(U, 1, 10.0)
            assert dev.product() == (form, size)
            assert np.isclose(hist[0], norm, rtol=1e-12, atol=0.0) and cfl == step.cfl
            for v in range(U.shape[0]):   # the bound of the linearised product's own test
                d, ref = new[v] - U[v], step.U[v] - U[v]
                assert np.abs(d - ref).max() <= 1e-8 * np.abs(ref).max(), (limit, v)
            assert np.array_equal(got.setdefault(form, new), new)   # the same bits within a form
    finally:
        dev.close()


def test_another_plan_takes_the_factors_back(cuda):
    """With less free memory than a second plan needs, and more once the first plan's factors are
    given up, the second plan is made; the first steps without them, says so, and has them again
    once there is room."""
    import torch
    from jaxrans_b200.native import JR_PRODUCT_DUAL, JR_PRODUCT_LINEARISED
    from jaxrans_b200.native3d import DevicePlan3
    args, imp = wing("sa", None, (64, 16, 16, 16))
    _, U = state(args, "sa")

    def free():
        torch.cuda.empty_cache()
        return torch.cuda.mem_get_info()[0]

    first = DevicePlan3(*args, imp)
    before = free()
    second = DevicePlan3(*args, imp)
    need = before - free()
    second.close()
    ref = first.newton_steps(U, 1, 10.0)
    form, size = first.product()
    assert form == JR_PRODUCT_LINEARISED and size > (16 << 20) and need > size // 2
    hold = torch.empty(free() - (need - size // 2), dtype=torch.uint8, device="cuda")   # never written
    try:
        assert free() < need
        second = DevicePlan3(*args, imp)
        try:
            with pytest.warns(RuntimeWarning, match="dual-number"):
                U1 = first.newton_steps(U, 1, 10.0)[0]
            assert first.product()[0] == JR_PRODUCT_DUAL
            d = ref[0] - U
            assert all(np.abs(U1[v] - ref[0][v]).max() <= 1e-8 * np.abs(d[v]).max() for v in range(6))
        finally:
            second.close()
    finally:
        del hold
    free()
    again = first.newton_steps(U, 1, 10.0)
    assert first.product()[0] == JR_PRODUCT_LINEARISED and np.array_equal(again[0], ref[0])
    first.close()
