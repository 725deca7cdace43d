"""Calls that wait for the context's stream, so that a caller may go on in a stream of its own:
gdfv_set_time (with a step of the other parity it moves the state to the other buffer) and
gdfv_get_time."""
import pytest
import torch

import cases

pytestmark = pytest.mark.gpu


def test_the_state_has_moved_when_set_time_returns():
    from gdfv.autograd import _state_view
    sim = cases.build_gpu(cases.c2_inflow_box(n=(32, 24, 20)))
    its, mine = torch.cuda.Stream(), torch.cuda.Stream()
    sim.set_stream(its.cuda_stream)
    first = _state_view(sim)                  # the buffer of even steps
    assert sim.run(max_step=1) == 1
    second = _state_view(sim)                 # and of odd ones
    assert first.data_ptr() != second.data_ptr()
    want = second.clone()
    out = torch.empty_like(want)
    first.zero_()
    torch.cuda.synchronize()
    with torch.cuda.stream(its):
        torch.cuda._sleep(100_000_000)        # some 50 ms of earlier work
    sim.set_time(0.0, 2, 1e-6)
    with torch.cuda.stream(mine):
        out.copy_(first)
    torch.cuda.synchronize()
    assert torch.equal(out, want)


def test_get_time_waits_for_the_contexts_stream():
    sim = cases.build_gpu(cases.c2_inflow_box(n=(32, 24, 20)))
    its, mine = torch.cuda.Stream(), torch.cuda.Stream()
    sim.set_stream(its.cuda_stream)
    assert sim.run(max_step=1) == 1
    there, out = torch.zeros(1000, device="cuda"), torch.zeros(1000, device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.stream(its):
        torch.cuda._sleep(100_000_000)
        there.fill_(1.0)
    assert sim.time()["step"] == 1
    with torch.cuda.stream(mine):
        out.copy_(there)
    torch.cuda.synchronize()
    assert torch.all(out == 1.0)
