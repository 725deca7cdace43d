"""gdfv_residual from several threads on one context, and beside a recorded run: each call's R(U) is
that of its own state and the run is not changed, although the line sweeps hold primitives and
residual sums in buffers of the context.  Same kernels on the same numbers: equality."""
import threading

import numpy as np
import pytest
import torch

import cases

pytestmark = pytest.mark.gpu


def _together(*jobs):
    errors = []

    def guarded(job):
        try:
            job()
        except Exception as e:   # (a thread's own failure is not the test's otherwise)
            errors.append(repr(e))

    threads = [threading.Thread(target=guarded, args=(job,)) for job in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120.0)
    assert not any(t.is_alive() for t in threads) and not errors, errors


def _states(sim, count):
    U = sim.get_conserved(0)
    rng = np.random.default_rng(3)
    return [torch.from_numpy(U * (1.0 + 1e-3 * rng.standard_normal(U.shape[1]))).cuda() for _ in range(count)]


@pytest.mark.parametrize("form", ["euler", "mhd"])
@pytest.mark.parametrize("sweeps", [0, 1])
def test_residuals_of_several_threads(form, sweeps):
    case = (cases.c2_inflow_box(n=(40, 33, 21), noise_all=True) if form == "euler" else cases.orszag_tang(n=(48, 40, 4)))
    sim = cases.build_gpu(case, line_sweeps=sweeps)
    assert sim.run(max_step=1) == 1
    Us = _states(sim, 4)
    want = []
    for U in Us:
        R = torch.empty_like(U)
        sim.residual(U.data_ptr(), R.data_ptr())
        want.append(R.clone())
    outs = [torch.empty_like(U) for U in Us]
    torch.cuda.synchronize()
    wrong = []

    def again(m):
        for _ in range(150):
            sim.residual(Us[m].data_ptr(), outs[m].data_ptr())
            if not torch.equal(outs[m], want[m]):
                wrong.append(m)

    _together(*(lambda m=m: again(m) for m in range(4)))
    assert not wrong, len(wrong)


def test_residuals_beside_a_recorded_run():
    from gdfv._lib import ffi
    case = cases.c2_inflow_box(n=(40, 33, 21), noise_all=True)
    sims = [cases.build_gpu(case, line_sweeps=1) for _ in range(2)]
    for sim in sims:   # the steps are captured once, by the first run
        assert sim.run(max_step=1) == 1
    U = _states(sims[0], 1)[0]
    R = torch.empty_like(U)
    done = threading.Event()
    none = ffi.new("double*[]", [ffi.NULL] * 2)

    def record(sim):
        for _ in range(60):
            assert sim.L.gdfv_run_record(sim.ctx, 2, none, none, ffi.new("double[]", 2)) == 0
        done.set()

    def residuals(sim):
        while not done.is_set():
            sim.residual(U.data_ptr(), R.data_ptr())

    record(sims[1])
    done.clear()
    _together(lambda: record(sims[0]), lambda: residuals(sims[0]))
    assert np.array_equal(sims[0].get_conserved(0), sims[1].get_conserved(0))
    assert sims[0].time() == sims[1].time()
