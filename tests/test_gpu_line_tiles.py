"""The adjoint's line tiles (gdfv_adjoint.cu: 256 slots along i, 32 lines by 8 cells along j and
k) at the sizes where their ends fall on, before and after the ends of the lines, and the
tile depth chosen from the block sizes.

The VJP against the CPU oracle's complex-step JVP by the dot test, with the bound the other
VJP tests hold (1e-10: the products' own rounding, about 1e-14, times the few thousand terms
of the dot product with headroom); FP64 steps do not depend on the tile depth (equality)."""
import numpy as np
import pytest

import cases
from test_gpu_adjoint import _dot_check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flux", ["ausmdv", "hllc"])
@pytest.mark.parametrize("n", [(2, 2, 2), (33, 6, 7), (31, 7, 15), (251, 2, 8), (252, 3, 2), (255, 2, 13), (5, 64, 14)])
def test_vjp_at_tile_ends(flux, n):
    case = cases.c2_inflow_box(n=n, flux=flux, noise_all=True)
    _dot_check(case, 2, 1e-10)


@pytest.mark.parametrize("n", [(33, 6, 7), (252, 3, 2), (8, 14, 13)])
def test_mhd_vjp_at_tile_ends(n):
    _dot_check(cases.orszag_tang(n=n), 2, 1e-10)


@pytest.mark.parametrize("n", [(20, 9, 33), (40, 7, 2), (64, 48, 10), (33, 5, 61)])
def test_tile_depth_from_the_sizes_does_not_change_results(n):
    out = []
    for kc in (0, 32, 5):
        sim = cases.build_gpu(cases.c2_inflow_box(n=n), tile_kchunk=kc, line_sweeps=0)
        assert sim.run(max_step=3) == 3
        out.append(sim.get_conserved(0))
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])
