"""The branch-free FP64 quotient and root of the flux kernels (gdfv_device.cuh: quot, root)
round as the division and square root of IEEE arithmetic do, and operands outside their
range take the compiler's own: the FP64 residual equals the CPU oracle's bit for bit in
and out of that range.  Both sides perform the same IEEE operations, so the bound is
equality."""
import numpy as np
import pytest

import cases
from test_gpu_adjoint import _gpu_to_oracle_layout

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["ausmdv", "hllc", "lmr", "graded", "mhd"])
@pytest.mark.parametrize("scale, eps", [(0, 1e-12), (-90, 1e-12), (-120, 1e-12), (120, 1e-12), (0, 1e-250)])
def test_residual_bit_for_bit_over_the_operand_range(form, scale, eps):
    """Densities and energies times 2^scale (pressures and densities of 1e-36 and 1e36 at
    the ends, sound speeds unchanged), and a limiter epsilon below quot's range."""
    import torch
    from gdfv.autograd import residual_eval
    if form == "mhd":
        case = cases.orszag_tang(n=(34, 9, 3))
    elif form == "graded":
        case = cases.graded_lattice()
    else:
        case = cases.c1_shock_box(n=13)
    case.config["epsilon_van_albada"] = eps
    if form == "hllc":
        case.config["flux_calculator"] = "hllc"
    if form == "lmr":
        case.config["van_albada_variant"] = "lmr"
    orc, sim = cases.build_pair(case)
    if case.mhd:   # two steps on both sides: the same c_h
        assert orc.run(2) == 0 and sim.run(max_step=2) == 2
    rng = np.random.default_rng(11)
    Us = []
    for b in range(len(case.blocks)):
        U = sim.get_conserved(b)
        n = U.shape[1]
        dm = U[0] * rng.standard_normal((3, n)) * (0.05 if case.mhd else 30.0)
        U[4] += ((U[1:4] + dm) ** 2 - U[1:4] ** 2).sum(axis=0) / (2.0 * U[0])   # the same internal energy
        U[1:4] += dm
        U[:5] *= 2.0 ** scale
        if case.mhd:   # the magnetic energy scales with the square of B
            U[5:9] *= 2.0 ** (scale // 2)
        Us.append(U)
    U = np.concatenate(Us, axis=1)
    R = residual_eval(sim, torch.from_numpy(U).cuda()).cpu().numpy()
    assert np.all(np.isfinite(R)) and np.any(R != 0.0)
    assert np.array_equal(_gpu_to_oracle_layout(case, R), orc.residual(_gpu_to_oracle_layout(case, U)))
