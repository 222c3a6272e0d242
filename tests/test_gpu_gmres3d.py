"""The 3D GMRES cycle with its scalars on the device: Newton steps against the oracle's for
subspaces either side of every register form of the orthogonalisation (8, 16, 32 vectors a
thread, then slices), an odd vector length (no 16-byte loads), a second cycle, and no
preconditioner."""

from __future__ import annotations

import numpy as np
import pytest

from jaxrans_b200.config import FlowConditions, ImplicitConfig, freestream_primitive3
from jaxrans_b200.grid3d import Block3, Rect3
from jaxrans_b200.plan3d import build_plan3d

pytestmark = pytest.mark.gpu


def box(ni, nj, nk):
    """A skewed box over a slip wall (j_min), far field elsewhere."""
    i, j, k = np.meshgrid(*(np.arange(n + 1, dtype=float) for n in (ni, nj, nk)), indexing="ij")
    nodes = np.stack([i + 0.2 * j, k + 0.1 * j, j + 0.3 * np.sin(0.7 * i) * (1.0 + 0.1 * k)])
    size = {"i": (nj, nk), "j": (ni, nk), "k": (ni, nj)}
    sides = {f"{a}_{e}": [Rect3("wall" if (a, e) == ("j", "min") else "farfield", (0, 0), size[a])]
             for a in "ijk" for e in ("min", "max")}
    return Block3(nodes, sides).with_kinds({"wall": "slip_wall", "farfield": "far_field"})


@pytest.mark.parametrize("cells,subspace,restarts,preconditioner",
                         [((8, 7, 6), 1, 1, "line_j"), ((9, 7, 5), 8, 1, "line_j"), ((9, 7, 5), 9, 2, "line_j"),
                          ((8, 7, 6), 17, 1, "line_j"), ((9, 7, 5), 33, 1, "line_j"), ((8, 7, 6), 40, 1, "none")])
def test_newton_step_matches_the_oracle(cuda, cells, subspace, restarts, preconditioner):
    from jaxrans_b200.native3d import DevicePlan3
    from oracle import implicit as im
    from oracle import implicit3d as i3
    from oracle import numerics3d as n3
    plan = build_plan3d([box(*cells)], with_distance=False)
    assert plan.n_canvas % 2 == (cells == (9, 7, 5))   # 5 variables: the odd canvas's vectors are odd too
    flow = FlowConditions(mach=0.6, alpha_deg=2.5)
    q_inf = np.array(freestream_primitive3(flow))
    imp = ImplicitConfig(krylov_subspace=subspace, krylov_restarts=restarts, krylov_tol=1e-9,
                         preconditioner=preconditioner)
    oracle = n3.Model3(plan, q_inf, flow.gamma, "roe", "van_albada_smooth", 0.0, None, None, False)
    rng = np.random.default_rng(3)
    U = n3.initial_state(oracle)
    U = np.where(plan.interior, U * (1.0 + 0.02 * rng.uniform(-1.0, 1.0, U.shape)), U)
    U[2] = np.where(plan.interior, 0.05 * rng.uniform(-1.0, 1.0, plan.shape), U[2])   # off V.n = 0, a kink
    step, norm = i3.newton_step(im.NewtonState(U, 10.0, np.inf), oracle, imp)
    dev = DevicePlan3(plan, q_inf, flow.gamma, "roe", "van_albada_smooth", 0.0, None, None, imp)
    try:
        got, cfl, _, hist = dev.newton_steps(U, 1, 10.0)
    finally:
        dev.close()
    assert np.isclose(hist[0], norm, rtol=1e-12, atol=0.0) and cfl == step.cfl
    for v in range(5):   # products within 1e-12 of their largest entry, amplified over the cycle
        d, ref = got[v] - U[v], step.U[v] - U[v]
        assert np.abs(d - ref).max() <= 1e-8 * np.abs(ref).max(), v
