"""A schedule of the fused FP64 launch that the configuration asks for is the one that runs, at
sizes whose default is the line sweeps; results do not depend on it (equality)."""
import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu


def _run(**config):
    sim = cases.build_gpu(cases.c2_inflow_box(n=(64, 60, 56), noise_all=True), **config)
    assert sim.run(max_step=2) == 2
    return sim, sim.get_conserved(0)


@pytest.mark.parametrize("config, sweeps", [
    (dict(persistent=True), 0),
    (dict(tile_kchunk=7), 0),
    (dict(persistent=True, line_sweeps=1), 1),   # asked for as well
    (dict(line_sweeps=0), 0),
])
def test_the_schedule_asked_for_runs(config, sweeps):
    default, U0 = _run()
    assert default.option("line_sweeps") == 1
    sim, U = _run(**config)
    assert sim.option("line_sweeps") == sweeps
    for key, value in config.items():
        assert sim.option(key) == value
    assert np.array_equal(U0, U)


def test_the_tuner_weighs_the_sweeps_whatever_was_asked_for():
    sim = cases.build_gpu(cases.c2_inflow_box(n=(64, 60, 56), noise_all=True), autotune=True, persistent=True,
                          tile_kchunk=7)
    assert sim.option("line_sweeps") == 1   # on trial until the first run
    assert sim.run(max_step=2) == 2
    assert np.array_equal(sim.get_conserved(0), _run()[1])
