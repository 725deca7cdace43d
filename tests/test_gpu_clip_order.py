"""The order of the clipping bounds (src/nm/limiters.d:41-50: lower = A if A <= B, upper = A if
A > B) where it is not a question of magnitude: bounds +0 and -0, as a slip wall's ghost and a
cell without normal velocity have them, and bounds that are not a number.

* VJP against the CPU oracle's complex-step JVP column by column (one unit vector at a time, so
  that each entry takes the one-sided branch of its own value), at states whose velocity
  components are exactly zero.  Bound: 1e-10 of the row's largest entry, as for the other
  products (rounding of some tens of terms, each to about 1e-15).
* The residual with one cell's energy not a number, of either sign bit: the same operations
  as the oracle's, so the same numbers in all cells it does not reach."""
import numpy as np
import pytest
import torch

import cases

pytestmark = pytest.mark.gpu


def _walled_box(flux, moving):
    """3x4x3 cells, slip walls all round; random velocities along the axes in `moving`."""
    n = (3, 4, 3)
    case = cases.Case("walled", dict(flux_calculator=flux), cases.R_AIR_CHICKEN, 1.4)
    rng = np.random.default_rng(3)
    shape = n[::-1]
    rho = 1.0 + 0.1 * rng.standard_normal(shape)
    T = 300.0 * (1.0 + 0.05 * rng.standard_normal(shape))
    vel = tuple(30.0 * rng.standard_normal(shape) if axis in moving else np.zeros(shape) for axis in range(3))
    case.add_block(n, (1e-3, 1e-3, 1e-3), (0, 0, 0), {}, rho, vel, T)
    return case


@pytest.mark.parametrize("flux", ["ausmdv", "hllc"])
@pytest.mark.parametrize("moving", [(), (0,), (0, 2), (0, 1, 2)])
def test_vjp_columns_with_velocities_of_zero(flux, moving):
    from gdfv.autograd import vjp
    orc, sim = cases.build_pair(_walled_box(flux, moving))
    U = sim.get_conserved(0)
    assert orc.set_U(0, U) == 0
    N = U.size
    unit = np.eye(N)
    J = np.stack([orc.jvp_complex(U.ravel(), unit[k]) for k in range(N)], axis=1)
    Ud = torch.from_numpy(U).cuda()
    G = np.stack([vjp(sim, Ud, torch.from_numpy(unit[k].reshape(U.shape)).cuda())[0].cpu().numpy().ravel()
                  for k in range(N)])
    assert np.all(np.abs(G - J) <= 1e-10 * np.abs(J).max(axis=1, keepdims=True))


@pytest.mark.parametrize("sweeps", [0, 1])
@pytest.mark.parametrize("flux", ["ausmdv", "hllc"])
@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_residual_beside_a_cell_that_is_not_a_number(sign, flux, sweeps):
    from gdfv.autograd import residual_eval
    case = cases.c2_inflow_box(n=(9, 8, 7), noise_all=True)
    case.config["flux_calculator"] = flux
    orc, sim = cases.build_pair(case, line_sweeps=sweeps)
    U = sim.get_conserved(0)
    U[4, 250] = np.copysign(np.nan, sign)
    R = residual_eval(sim, torch.from_numpy(U).cuda()).cpu().numpy()
    Ro = orc.residual(U.ravel()).reshape(R.shape)
    assert np.isnan(R).any() and np.isfinite(R).sum() > 0.9 * R.size
    assert np.array_equal(R, Ro, equal_nan=True)
