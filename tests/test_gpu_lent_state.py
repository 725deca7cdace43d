"""The state lent by gdfv_state_device_ptr is the caller's to write until the next gdfv_run, also when
the stages have been timed in between: the run starts from what was written, in every form of the
stages (the line sweeps and the float kernel keep decoded primitives).  Compared with the same
state set by gdfv_block_set_conserved: equality."""
import numpy as np
import pytest
import torch

import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("config", [dict(line_sweeps=0), dict(line_sweeps=1), dict(flux_precision="fp32")])
@pytest.mark.parametrize("timed", [False, True])
def test_a_state_written_through_the_pointer(config, timed):
    from gdfv.autograd import _state_view
    out = []
    for through in (True, False):
        sim = cases.build_gpu(cases.c2_inflow_box(n=(24, 18, 14), noise_all=True), **config)
        assert sim.run(max_step=2) == 2
        U = sim.get_conserved(0)
        U[:] = U[:, ::-1] * 1.01
        view = _state_view(sim)
        if timed:
            sim.time_stages(2)
        if through:
            view.copy_(torch.from_numpy(U.copy()))
            torch.cuda.synchronize()
            sim.set_time(0.0, 2, 1e-6)   # (and the signal's maxima are taken again)
        else:
            sim.set_time(0.0, 2, 1e-6)
            sim.set_conserved(0, U)
        assert sim.run(max_step=2) == 2
        out.append((sim.get_conserved(0), sim.time()))
    assert np.array_equal(out[0][0], out[1][0]) and out[0][1] == out[1][1]


@pytest.mark.parametrize("config", [dict(line_sweeps=0), dict(line_sweeps=1), dict(flux_precision="fp32")])
def test_a_state_written_after_the_stages_were_timed(config):
    from gdfv.autograd import _state_view
    out = []
    for through in (True, False):
        sim = cases.build_gpu(cases.c2_inflow_box(n=(24, 18, 14), noise_all=True), **config)
        assert sim.run(max_step=2) == 2
        U = sim.get_conserved(0) * 1.02
        view = _state_view(sim)
        sim.time_stages(2)   # (takes the signal's maxima again as well)
        if through:
            view.copy_(torch.from_numpy(U))
            torch.cuda.synchronize()
        else:
            sim.set_conserved(0, U)
        assert sim.run(max_step=2) == 2
        out.append((sim.get_conserved(0), sim.time()))
    assert np.array_equal(out[0][0], out[1][0]) and out[0][1] == out[1][1]
