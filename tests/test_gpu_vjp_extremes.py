"""The VJP with operands outside the range of its branch-free reciprocals (gdfv_adjoint.cu).

* At a subnormal limiter epsilon it is what it is at 1e-300: the epsilon matters only where both
  differences are 0, and there the limiter is 1 either way.
* It is finite beside a cell of energy 1e150, and four cells away along some axis it is what it
  is without that cell.

Bound: 1e-12 of the quantity's largest entry (the order of the atomic sums, 1e-13)."""
import numpy as np
import pytest
import torch

import cases
from test_gpu_fp64_extremes import CELL, _case

pytestmark = pytest.mark.gpu


def _vjp(case, kind=None):
    from gdfv.autograd import vjp
    sim = cases.build_gpu(case)
    if case.mhd:
        assert sim.run(max_step=1) == 1
    U = sim.get_conserved(0)
    if kind:
        U[4, CELL] = 1e150
    W = np.random.default_rng(1).standard_normal(U.shape)
    return vjp(sim, torch.from_numpy(U).cuda(), torch.from_numpy(W).cuda())[0].cpu().numpy()


@pytest.mark.parametrize("form", ["ausmdv", "hllc", "graded", "mhd"])
def test_vjp_with_a_subnormal_epsilon(form):
    out = []
    for eps in (1e-308, 1e-300):
        case = _case(form)
        case.config["epsilon_van_albada"] = eps
        out.append(_vjp(case))
    assert np.all(np.isfinite(out[0]))
    assert np.all(np.abs(out[0] - out[1]) <= 1e-12 * np.abs(out[1]).max(axis=1, keepdims=True))


@pytest.mark.parametrize("form", ["ausmdv", "hllc", "lmr", "graded"])
def test_vjp_beside_a_cell_of_extreme_energy(form):
    case = _case(form)
    n = case.blocks[0]["n"]
    G0, G1 = _vjp(case), _vjp(case, "energy")
    assert np.all(np.isfinite(G1))
    at = np.array(np.unravel_index(CELL, n[::-1]))
    where = np.stack(np.unravel_index(np.arange(G0.shape[1]), n[::-1]))
    far = (np.abs(where - at[:, None]) >= 4).any(axis=0)
    assert far.sum() > 100
    assert np.all(np.abs(G1 - G0)[:, far] <= 1e-12 * np.abs(G0).max(axis=1, keepdims=True))
