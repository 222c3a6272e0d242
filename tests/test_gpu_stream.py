"""Newton steps on a caller's stream (jr_plan_set_stream), their graph captured over the plan's two
side streams: ordered after the caller's earlier work and before its later work, and bitwise the
steps on the plan's own stream, whichever stream the graph was captured on."""

from __future__ import annotations

import numpy as np
import pytest

from goldens import load
from jaxrans_b200.solver import freestream_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["o_euler", "c_sa"])
def test_steps_on_a_callers_stream(cuda, name):
    import torch
    from jaxrans_b200.native import DevicePlan
    z, case, plan = load(name)
    U0 = freestream_state(case, plan)
    own = DevicePlan(plan, case.flow, case.numerics, case.implicit)
    own.set_state(U0, case.implicit.cfl)
    hist = own.newton_steps(6)
    ref = own.get_state()[0]
    own.close()

    dev = DevicePlan(plan, case.flow, case.numerics, case.implicit)
    stream = torch.cuda.Stream()

    def steps_on(handle):
        """The state written and read in the stream's order, with nothing else waited for."""
        assert dev.lib.jr_plan_set_stream(dev.handle, handle) == 0
        with torch.cuda.stream(stream if handle else torch.cuda.ExternalStream(dev.stream_handle())):
            work = torch.randn(2048, 2048, device="cuda")
            for _ in range(20):   # the state is still to be written when the steps are queued
                work = torch.tanh(work @ work * 1e-3)
            u = torch.zeros(U0.shape, dtype=torch.float64, device="cuda")
            u.copy_(torch.as_tensor(U0), non_blocking=True)
            assert dev.lib.jr_state_set_device(dev.handle, u.data_ptr(), case.implicit.cfl, float("inf")) == 0
            got = torch.zeros(6, dtype=torch.float64, device="cuda")
            assert dev.lib.jr_newton_steps_async(dev.handle, 6, got.data_ptr()) == 0
            got = got.clone()
            torch.cuda.current_stream().synchronize()
        return got.cpu().numpy(), dev.get_state()[0]

    try:
        # captured on the caller's stream, then the same graph on the plan's own, and back
        for handle in (stream.cuda_stream, None, stream.cuda_stream):
            got, U = steps_on(handle)
            assert np.array_equal(got, hist.ravel()) and np.array_equal(U, ref)
        dev.enable(0, True)   # drops the graph: the next is captured on the plan's own stream
        got, U = steps_on(None)
        assert np.array_equal(got, hist.ravel()) and np.array_equal(U, ref)
    finally:
        dev.lib.jr_plan_set_stream(dev.handle, None)
        dev.close()


@pytest.mark.parametrize("many", [False, True])
def test_a_captured_residual_call_reads_what_is_there_at_replay(cuda, many):
    """jr_residual under a caller's stream capture, its ghosts by the tiles (one case) or by a launch
    (more than 5700 ghosts): nothing of the captured call lives on in host memory."""
    import torch
    from jaxrans_b200.native import DevicePlan
    z, case, plan = load("c_sa")
    flows = [case.flow] * (1 + 5700 // int((~plan.interior).sum()) * 2 if many else 1)
    dev = DevicePlan.batch(plan, flows, case.numerics, case.implicit) if many else \
        DevicePlan(plan, case.flow, case.numerics, case.implicit)
    rng = np.random.default_rng(9)
    U = [np.concatenate([(freestream_state(case, plan) * (1.0 + 0.01 * rng.uniform(-1.0, 1.0, (5,) + plan.shape))).ravel()
                         for _ in flows]) for _ in range(2)]
    if not many:
        U = [u.reshape((5,) + plan.shape) for u in U]
    ref = [dev.residual(u) for u in U]
    u, out = torch.as_tensor(U[0], device="cuda"), torch.zeros(U[0].shape, dtype=torch.float64, device="cuda")
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    torch.cuda.synchronize()
    assert dev.lib.jr_plan_set_stream(dev.handle, stream.cuda_stream) == 0
    with torch.cuda.graph(graph, stream=stream):
        assert dev.lib.jr_residual(dev.handle, u.data_ptr(), out.data_ptr(), 0) == 0
    assert dev.lib.jr_plan_set_stream(dev.handle, None) == 0
    for k in (0, 1, 0):
        u.copy_(torch.as_tensor(U[k]))
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy(), ref[k])
    del graph
    dev.close()
