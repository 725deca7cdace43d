"""The FP64 line sweeps (gdfv_sweep.cuh) against stage_kernel, which the parity tests hold to
the CPU oracle: the same functions per cell and face in the same order of the sums, so states,
time and R(U) are equal bit for bit, over the forms the stages take and at sizes where the
warps' windows and the threads' stretches end on, before and after the ends of the lines."""
import numpy as np
import pytest
import torch

import cases

pytestmark = pytest.mark.gpu

EXT = {f: ("outflow_simple_extrapolate", dict(x_order=1)) for f in ("west", "east", "south", "north", "bottom", "top")}


def _outflows():
    """Every outflow rule of its own: SimpleFlux, FixedP, FixedPT and linear extrapolation."""
    c = cases.c1_shock_box(n=14)
    c.blocks[0]["bcs"].update(west=("outflow_simple_flux", {}), east=("outflow_fixed_p", dict(p_outside=9.0e3)),
                              south=("outflow_fixed_p_and_t", dict(p_outside=6.0e4, T_outside=310.0)),
                              north=("outflow_simple_extrapolate", dict(x_order=1)))
    return c


def _lmr():
    c = cases.c2_inflow_box(n=(19, 8, 9), noise_all=True)
    c.config["van_albada_variant"] = "lmr"
    return c


FORMS = {
    "box": lambda: cases.c2_inflow_box(n=(37, 19, 23), noise_all=True),
    "small": lambda: cases.c2_inflow_box(n=(2, 2, 2)),
    "window_252": lambda: cases.c2_inflow_box(n=(250, 3, 6), noise_all=True),
    "window_254": lambda: cases.c2_inflow_box(n=(254, 2, 7), noise_all=True),
    "stretches": lambda: cases.c2_inflow_box(n=(33, 15, 14), flux="hllc"),
    "lattice": lambda: cases.multiblock_lattice(nb=(2, 2, 2)),
    "tube": cases.sod_eilmer,
    "graded": cases.graded_lattice,
    "exchange": lambda: cases.exchange_pair(1),
    "exchange_graded": lambda: cases.exchange_pair(3, graded=True),
    "rotating": lambda: cases.quarter_rotational(seed=3),
    "outflows": _outflows,
    "lmr": _lmr,
    "mhd": lambda: cases.orszag_tang(n=(34, 9, 3)),
    "mhd_rotating": lambda: cases.quarter_rotational(seed=3, mhd=True),
    "mhd_dipole": lambda: cases.mhd_slip_dipole(n=(32, 24, 4)),
    "mhd_2d": lambda: cases.mhd_shock_tube(N=128),
}


def _march(case, sweeps, **config):
    from gdfv.autograd import residual_eval
    sim = cases.build_gpu(case, line_sweeps=sweeps, **config)
    assert sim.run(max_step=4) == 4 and sim.option("line_sweeps") == sweeps
    U = np.concatenate([sim.get_conserved(b) for b in range(len(case.blocks))], axis=1)
    R = residual_eval(sim, torch.from_numpy(U).cuda()).cpu().numpy()
    return U, R, sim.time(), sim.residual_norms()


@pytest.mark.parametrize("form", sorted(FORMS))
def test_sweeps_equal_stage_kernel(form):
    U0, R0, t0, n0 = _march(FORMS[form](), 0)
    U1, R1, t1, n1 = _march(FORMS[form](), 1)
    assert np.array_equal(U0, U1) and np.array_equal(R0, R1) and t0 == t1
    assert np.array_equal(n0[0], n1[0]) and n0[1] == n1[1]


def test_sweeps_after_the_state_is_set_again_and_tuned():
    """A state written from outside a stage is decoded before the next step, and the tuner
    leaves results alone whichever form it keeps."""
    out = []
    for sweeps, tuned in ((0, False), (1, False), (1, True), (2, True)):
        sim = cases.build_gpu(cases.c2_inflow_box(n=(40, 24, 20)), line_sweeps=sweeps, autotune=tuned)
        U0 = sim.get_conserved(0)
        sim.run(max_step=3)
        sim.set_time(0.0, 0, sim.config.dt_init)
        sim.set_conserved(0, U0 * 1.0)
        sim.run(max_step=3)
        out.append(sim.get_conserved(0))
    assert all(np.array_equal(out[0], u) for u in out[1:])


def test_sweeps_report_the_failing_cell_and_retry_as_stage_kernel():
    """An unstable CFL number: the same status, steps and cell."""
    from gdfv._lib import GdfvError
    seen = []
    for sweeps in (0, 1):
        sim = cases.build_gpu(cases.c1_shock_box(n=16), line_sweeps=sweeps, cfl_value=12.0, dt_init=1.0, dt_max=1.0)
        try:
            seen.append(("ok", sim.run(max_step=6), sim.time(), sim.get_conserved(0).tobytes()))
        except GdfvError as e:
            seen.append((str(e), sim.time()["step"], sim.last_bad_cell()))
    assert seen[0] == seen[1]
