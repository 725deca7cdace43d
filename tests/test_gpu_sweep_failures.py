"""Steps that fail in the FP64 line sweeps: the predictor's failing cell, the retry at a fifth of
the dt, and the end after the last attempt are stage_kernel's.  No CTA of a predictor leaves
early, so the least failing cell does not depend on their order."""
import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu

FORMS = {
    "euler": lambda: cases.c1_shock_box(n=16),
    "lattice": lambda: cases.multiblock_lattice(nb=(2, 2, 1), sizes=(8, 12)),
    "mhd": lambda: cases.orszag_tang(n=(16, 12, 4)),
}


@pytest.mark.parametrize("form", sorted(FORMS))
@pytest.mark.parametrize("attempts", [1, 2])
def test_a_step_that_fails_in_the_predictor(form, attempts):
    from gdfv._lib import GDFV_ERR_STEP_FAILED, GdfvError
    seen = []
    for sweeps in (0, 1):
        sim = cases.build_gpu(FORMS[form](), line_sweeps=sweeps, fixed_time_step=True, dt_init=10.0, dt_max=10.0,
                              max_attempts_for_step=attempts)
        with pytest.raises(GdfvError) as e:
            sim.run(max_step=3)
        assert e.value.code == GDFV_ERR_STEP_FAILED
        assert sim.time()["step"] == 0 and sim.time()["dt"] == pytest.approx(10.0 * 0.2 ** attempts, rel=1e-12)
        seen.append((str(e.value), sim.last_bad_cell()))
    assert seen[0] == seen[1]


@pytest.mark.parametrize("form, cfl", [("euler", 3.0), ("mhd", 3.0)])
def test_a_step_that_is_retried_and_succeeds(form, cfl):
    out = []
    for sweeps in (0, 1):
        sim = cases.build_gpu(FORMS[form](), line_sweeps=sweeps, cfl_value=cfl, dt_init=1.0, dt_max=1.0)
        assert sim.run(max_step=1) == 1
        t = sim.time()
        assert t["dt"] == pytest.approx(0.2 * t["dt_allow"], rel=1e-12)   # the first attempt failed
        assert sim.run(max_step=3) == 3
        out.append((sim.get_conserved(0), sim.time()))
    assert np.array_equal(out[0][0], out[1][0]) and out[0][1] == out[1][1]
