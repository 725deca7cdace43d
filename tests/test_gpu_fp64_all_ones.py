"""Densities one unit in the last place below a power of two: their reciprocals lie next to the
midpoint of two numbers (decode forms 1 / rho), where the branch-free quotient of
gdfv_device.cuh is hardest to round.  The FP64 residual and steps perform the oracle's IEEE
operations, so the bound is equality."""
import numpy as np
import pytest
import torch

import cases
from test_gpu_adjoint import _gpu_to_oracle_layout

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["ausmdv", "hllc", "graded", "mhd"])
@pytest.mark.parametrize("sweeps", [0, 1])
def test_density_just_below_a_power_of_two(form, sweeps):
    from gdfv.autograd import residual_eval
    if form == "mhd":
        case = cases.orszag_tang(n=(34, 9, 3))
    elif form == "graded":
        case = cases.graded_inflow_box(n=(13, 9, 7))
    else:
        case = cases.c2_inflow_box(n=(11, 9, 8), flux=form, noise_all=True)
    orc, sim = cases.build_pair(case, line_sweeps=sweeps)
    if case.mhd:   # a step on both sides: the same c_h
        assert orc.run(1) == 0 and sim.run(max_step=1) == 1
    U = sim.get_conserved(0)
    rng = np.random.default_rng(5)
    rho = np.nextafter(2.0 ** rng.integers(-3, 4, U.shape[1]), 0.0)
    U[:5] *= rho / U[0]
    U[0] = rho
    R = residual_eval(sim, torch.from_numpy(U).cuda()).cpu().numpy()
    assert np.all(np.isfinite(R)) and np.any(R != 0.0)
    assert np.array_equal(_gpu_to_oracle_layout(case, R), orc.residual(_gpu_to_oracle_layout(case, U)))
