"""Operands far outside the range of the branch-free FP64 quotients (gdfv_device.cuh): single
cells with energies, densities, momenta or fields of 1e100 and more, whose squares and
differences overflow, and Mach numbers whose u - a rounds to u.  There the kernels divide as the
reference does, and the residual performs the oracle's IEEE operations: equality, with cells
that are not a number in the same places."""
import numpy as np
import pytest
import torch

import cases
from test_gpu_adjoint import _gpu_to_oracle_layout

pytestmark = pytest.mark.gpu

CELL = 349


def _case(form):
    if form == "mhd":
        return cases.orszag_tang(n=(10, 9, 8))
    if form == "graded":
        return cases.graded_inflow_box(n=(11, 9, 7))
    case = cases.c2_inflow_box(n=(11, 9, 7), noise_all=True)
    if form == "hllc":
        case.config["flux_calculator"] = "hllc"
    if form == "lmr":
        case.config["van_albada_variant"] = "lmr"
    if form == "unclipped":
        case.config["extrema_clipping"] = False
    return case


def _extreme(U, kind):
    U = U.copy()
    if kind == "energy":
        U[4, CELL] = 1e160
    elif kind == "all energies":
        U[4] *= 1e200 / U[4].mean()
    elif kind == "density":
        U[0, CELL] = 1e160
    elif kind == "momentum":
        U[1, CELL] = 1e100
        U[4, CELL] += U[1, CELL] ** 2 / U[0, CELL]
    elif kind == "field":
        U[5, CELL] = 1e100
        U[4, CELL] += U[5, CELL] ** 2
    elif kind == "speed":
        u = 1e19
        U[4] += 0.5 * U[0] * u * u * (1.0 + 4e-16)
        U[1] = U[0] * u
    return U


@pytest.mark.parametrize("sweeps", [0, 1])
@pytest.mark.parametrize("form, kind", [(f, k) for f in ("ausmdv", "hllc", "lmr", "unclipped", "graded", "mhd")
                                        for k in ("energy", "all energies", "density", "momentum")] +
                         [("hllc", "speed"), ("mhd", "field")])
def test_residual_bit_for_bit_with_extreme_cells(form, kind, sweeps):
    from gdfv.autograd import residual_eval
    case = _case(form)
    orc, sim = cases.build_pair(case, line_sweeps=sweeps)
    if case.mhd:   # a step on both sides: the same c_h
        assert orc.run(1) == 0 and sim.run(max_step=1) == 1
    U = _extreme(sim.get_conserved(0), kind)
    R = residual_eval(sim, torch.from_numpy(U).cuda()).cpu().numpy()
    assert np.array_equal(_gpu_to_oracle_layout(case, R), orc.residual(_gpu_to_oracle_layout(case, U)), equal_nan=True)
