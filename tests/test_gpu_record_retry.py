"""A recorded run (gdfv_run_record) in which a step is retried: it ends a step short of its limit
with GDFV_ERR_STATE, and gdfv_run goes on from there.  Every number it leaves -- state, time,
dt, c_h, the CFL numbers and the last predictor state -- is what gdfv_run alone leaves after the same
steps, and so is every later step.  Same kernels on the same numbers: the bound is equality."""
import numpy as np
import pytest
import torch

import cases

pytestmark = pytest.mark.gpu

UNSTABLE = dict(dt_init=1.0, dt_max=1.0)
FORMS = {   # (case, configuration, steps to record): the step that fails is the first unless noted
    "euler": (lambda: cases.c1_shock_box(n=8), dict(UNSTABLE, cfl_value=3.0, cfl_count=1), 4),
    "euler_third": (lambda: cases.c1_shock_box(n=8), dict(UNSTABLE, cfl_value=3.0, cfl_count=3), 3),
    "euler_float": (lambda: cases.c1_shock_box(n=8), dict(UNSTABLE, cfl_value=3.0, cfl_count=1, flux_precision="fp32"), 4),
    "euler_sweeps": (lambda: cases.c1_shock_box(n=8), dict(UNSTABLE, cfl_value=3.0, cfl_count=1, line_sweeps=1), 4),
    "lattice": (lambda: cases.multiblock_lattice(nb=(2, 2, 1), sizes=(8,)), dict(UNSTABLE, cfl_value=8.0, cfl_count=1), 4),
    "mhd": (lambda: cases.orszag_tang(n=(16, 12, 4)), dict(UNSTABLE, cfl_value=3.0), 4),
    "mhd_every_step": (lambda: cases.orszag_tang(n=(16, 12, 4)), dict(UNSTABLE, cfl_value=3.0, cfl_count=1), 4),
    # the step that fails takes the last slot: the retry is still to come
    "mhd_fixed_last": (lambda: cases.orszag_tang(n=(16, 12, 4)),
                       dict(fixed_time_step=True, dt_init=0.03, dt_max=1.0), 3),
}


def _record(sim, n):
    from gdfv._lib import ffi
    none = ffi.new("double*[]", [ffi.NULL] * n)
    return sim.L.gdfv_run_record(sim.ctx, n, none, none, ffi.new("double[]", n))


def _predictor(sim, U0):
    from gdfv._lib import check
    from gdfv.autograd import _p
    U1 = torch.empty_like(U0)
    check(sim.ctx, sim.L.gdfv_last_predictor_state(sim.ctx, _p(U0), _p(U1)))
    torch.cuda.synchronize()
    return U1.cpu().numpy()


def _state(sim, case):
    return np.concatenate([sim.get_conserved(b) for b in range(len(case.blocks))], axis=1)


@pytest.mark.parametrize("form", sorted(FORMS))
def test_a_run_goes_on_after_an_incomplete_record(form):
    from gdfv._lib import GDFV_ERR_STATE
    make, config, n = FORMS[form]
    case = make()
    rec = cases.build_gpu(case, **config)
    plain = cases.build_gpu(case, **config)
    assert _record(rec, n) == GDFV_ERR_STATE
    done = rec.time()["step"]
    assert done == n - 1   # one step was tried twice
    assert plain.run(max_step=done) == done
    assert np.array_equal(_state(rec, case), _state(plain, case))
    if not form.endswith("_last"):   # (there dt is the coming retry's)
        assert rec.time() == plain.time()
        U0 = torch.zeros((case.nq, case.total_cells()), dtype=torch.float64, device="cuda")
        assert np.array_equal(_predictor(rec, U0), _predictor(plain, U0))
    for more in (1, 3):
        assert rec.run(max_step=more) == more and plain.run(max_step=more) == more
        assert rec.time() == plain.time()
        assert np.array_equal(_state(rec, case), _state(plain, case))
        assert np.all(np.isfinite(_state(rec, case)))


@pytest.mark.parametrize("form", ["euler", "mhd"])
def test_a_complete_record_is_the_run(form):
    case = FORMS[form][0]()
    rec, plain = cases.build_gpu(case), cases.build_gpu(case)
    for n in (1, 4):
        assert _record(rec, n) == 0 and plain.run(max_step=n) == n
        assert rec.time() == plain.time() and np.array_equal(_state(rec, case), _state(plain, case))
    assert rec.run(max_step=2) == 2 and plain.run(max_step=2) == 2
    assert rec.time() == plain.time() and np.array_equal(_state(rec, case), _state(plain, case))
