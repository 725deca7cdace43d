"""Runs in which a CUDA call fails after the first step was to begin (the call answered by a
fake): the next run goes on from the last completed step with the dt, c_h and states of runs in
which nothing failed.  Same kernels on the same numbers: the bound is equality."""
import pytest

from cuda_fakes import run_with_fakes

pytestmark = pytest.mark.gpu

BODY = """
    import numpy as np
    import cases
    from gdfv._lib import GDFV_ERR_CUDA, ffi
    make = dict(euler=lambda: cases.c1_shock_box(n=8), mhd=lambda: cases.orszag_tang(n=(16, 12, 4)))[%r]
    case = make()
    config = dict(cfl_count=1, dt_max=1.0)
    bad, good = cases.build_gpu(case, **config), cases.build_gpu(case, **config)
    state = lambda sim: sim.get_conserved(0)
    def record(sim, n):
        none = ffi.new("double*[]", [ffi.NULL] * n)
        return sim.L.gdfv_run_record(sim.ctx, n, none, none, ffi.new("double[]", n))
    def run(sim, n):
        return sim.L.gdfv_run(sim.ctx, n, 0.0, ffi.new("int*"))
    assert bad.run(max_step=3) == 3
    %s
    done = bad.time()["step"]
    assert done == %d
    assert good.run(max_step=done) == done
    assert bad.time()["time"] == good.time()["time"] and bad.time()["dt"] == good.time()["dt"]
    assert np.array_equal(state(bad), state(good))
    for n in (1, 9):
        assert bad.run(max_step=n) == n and good.run(max_step=n) == n
        assert bad.time() == good.time() and np.array_equal(state(bad), state(good))
"""


@pytest.mark.parametrize("form", ["euler", "mhd"])
@pytest.mark.parametrize("call, done", [
    ("fakes.fake_fail_malloc(0, 0); assert record(bad, 5) == GDFV_ERR_CUDA; fakes.fake_fail_malloc(-1, 0)", 3),
    ("fakes.fake_fail_graph_launch(0); assert run(bad, 5) == GDFV_ERR_CUDA; fakes.fake_fail_graph_launch(-1)", 3),
    ("fakes.fake_fail_graph_launch(2); assert run(bad, 5) == GDFV_ERR_CUDA; fakes.fake_fail_graph_launch(-1)", 5),
    ("fakes.fake_fail_graph_launch(2); assert record(bad, 5) == GDFV_ERR_CUDA; fakes.fake_fail_graph_launch(-1)", 5),
])
def test_a_run_goes_on_after_a_failed_call(tmp_path, form, call, done):
    run_with_fakes(tmp_path, BODY % (form, call, done))
