"""The MHD adjoint's line tiles (gdfv_adjoint.cu: 192 slots along i, which step by 191; 32 lines by
6 cells along j and k, which step by 5) at sizes where their ends fall on, before and after the
ends of the lines.  The VJP against the CPU oracle's complex-step JVP by the dot test, with the
bound the other VJP tests hold."""
import pytest

import cases
from test_gpu_adjoint import _dot_check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(4, 4, 4), (33, 5, 9), (31, 10, 14), (187, 3, 2), (188, 2, 3), (189, 4, 2), (5, 9, 15)])
def test_mhd_vjp_at_its_tile_ends(n):
    _dot_check(cases.orszag_tang(n=n), 2, 1e-10)
