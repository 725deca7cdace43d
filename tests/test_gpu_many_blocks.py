"""Contexts of many small blocks: the tiles of the FP64 line sweeps and of the adjoint find their
block among thousands.  Results are stage_kernel's bit for bit, the VJP is the transpose of the
oracle's JVP (bound as in the other VJP tests), and the sweeps, which such a context takes by its
number of cells, are not slower than stage_kernel (they take half its time; the bound of 1.25
leaves room for a noisy clock)."""
import numpy as np
import pytest

import cases
from test_gpu_adjoint import _dot_check

pytestmark = pytest.mark.gpu


def _lattice(nb, sizes):
    rng = np.random.default_rng(2)
    return cases.multiblock_lattice(nb=nb, choices=[rng.choice(sizes, nb[a]) for a in range(3)])


@pytest.mark.parametrize("nb", [(1, 1, 2), (3, 1, 1), (5, 7, 3), (13, 11, 9)])
def test_sweeps_equal_stage_kernel_on_many_blocks(nb):
    case = _lattice(nb, (2, 3, 5))
    out = []
    for sweeps in (0, 1):
        sim = cases.build_gpu(case, line_sweeps=sweeps)
        assert sim.run(max_step=3) == 3
        out.append((np.concatenate([sim.get_conserved(b) for b in range(len(case.blocks))], axis=1), sim.time()))
    assert np.array_equal(out[0][0], out[1][0]) and out[0][1] == out[1][1]


def test_vjp_on_many_blocks():
    case = _lattice((5, 4, 3), (2, 3, 5))
    rng = np.random.default_rng(4)
    for b in case.blocks:   # no reconstructed field exactly uniform
        shape = b["n"][::-1]
        b["T"] = 220.0 * (1.0 + 0.01 * rng.standard_normal(shape))
        b["vel"] = tuple(v + 9.0 * rng.standard_normal(shape) for v in b["vel"])
    _dot_check(case, 2, 1e-10)


def test_sweeps_are_not_slower_on_many_small_blocks():
    ms = []
    for sweeps in (0, 2):
        sim = cases.build_gpu(cases.multiblock_lattice(nb=(32, 16, 16), sizes=(4,)), line_sweeps=sweeps)
        assert sim.option("line_sweeps") == (sweeps == 2)
        sim.run(max_step=2)
        ms.append(sum(sim.time_stages(5)))
    assert ms[1] < 1.25 * ms[0], ms
