"""The device memory of the FP64 line sweeps, on a device whose free memory a fake sets: what fits
beside stage_kernel fits in a context that would take the sweeps, and the tuner that keeps
stage_kernel gives their memory back.  Results do not depend on it (equality)."""
import pytest

from cuda_fakes import run_with_fakes

pytestmark = pytest.mark.gpu

HEAD = """
    import numpy as np, torch
    import cases
    from gdfv.autograd import vjp, residual_eval
    make = dict(euler=lambda: cases.c2_inflow_box(n=(64, 64, 60), noise_all=True),
                mhd=lambda: cases.orszag_tang(n=(256, 208, 4)))[%r]
    case = make()
    total = case.total_cells()
    U = torch.rand((case.nq, total), dtype=torch.float64, device="cuda")
    out = [torch.empty_like(U) for _ in range(2)]
    from gdfv._lib import check, ffi
    from gdfv.autograd import _p
    sigma = ffi.new("double*")
"""

# every call of a context that takes device memory of its own, in the room of `room` bytes
CALLS = """
    def calls(sweeps, room):
        fakes.fake_room(room)
        sim = cases.build_gpu(case, line_sweeps=sweeps)
        took = sim.option("line_sweeps")
        least = fakes.fake_room_left()
        assert sim.run(max_step=2) == 2
        U.copy_(torch.from_numpy(sim.get_conserved(0)))
        check(sim.ctx, sim.L.gdfv_residual_jvp(sim.ctx, _p(U), _p(U), ffi.NULL, 0.0, _p(out[0]), sigma))
        R = out[0].cpu().numpy()
        check(sim.ctx, sim.L.gdfv_residual_vjp(sim.ctx, _p(U), _p(U), _p(out[1]), ffi.NULL))
        flow = np.concatenate([np.ravel(v) for v in sim.get_flow(0).values()])
        sim.run(max_step=3)
        norms = sim.residual_norms()
        left = fakes.fake_room_left()
        state = sim.get_conserved(0)
        sim.close()
        fakes.fake_room(-1)
        return took, left, (R, state, flow, norms[0])
    took, left, want = calls(0, 1 << 40)
    need = (1 << 40) - left
    assert took == 0
    for sweeps in (1, 2):
        for room in (need + 4096, int(1.3 * need), 2 * need, 1 << 40):
            took, left, got = calls(sweeps, room)
            print("room", room, "of", need, "sweeps", took, "left", left)
            assert all(np.array_equal(a, b) for a, b in zip(want, got))
"""


@pytest.mark.parametrize("form", ["euler", "mhd"])
def test_what_fits_beside_stage_kernel_fits(tmp_path, form):
    """By size, and with the sweeps asked for: rooms from the least that stage_kernel needs (and a
    little for the sweeps' tile offsets) up."""
    run_with_fakes(tmp_path, HEAD % form + CALLS)


def test_prepare_fits_where_the_sweeps_leave_nothing(tmp_path):
    run_with_fakes(tmp_path, HEAD % "euler" + """
    fakes.fake_room(1 << 40)
    sim = cases.build_gpu(case, line_sweeps=0)
    need = (1 << 40) - fakes.fake_room_left()
    sim.close()
    # around the room where the sweeps fit and what follows them in gdfv_prepare would not
    for more in [0, 1 << 10] + [184 * total + 512 * m for m in range(-8, 9)]:
        fakes.fake_room(need + more)
        sim = cases.build_gpu(case, line_sweeps=1)
        assert sim.run(max_step=1) == 1
        sim.close()
    """)


def test_the_tuner_gives_the_memory_back(tmp_path):
    run_with_fakes(tmp_path, HEAD % "euler" + """
    left = []
    for slow in (0, 2):   # two times of the sweeps, a thousand times longer
        fakes.fake_room(1 << 40)
        sim = cases.build_gpu(case, autotune=True)
        assert sim.option("line_sweeps") == 1
        fakes.fake_slow_events(slow)
        assert sim.run(max_step=2) == 2
        assert sim.option("line_sweeps") == (slow == 0)
        left.append(fakes.fake_room_left())
        sim.close()
        fakes.fake_room(-1)
    assert left[1] - left[0] >= 184 * total
    """)


def test_the_kept_flow_buffer_gives_way(tmp_path):
    """After flow states have been read, products whose scratch needs the buffer's room."""
    run_with_fakes(tmp_path, HEAD % "euler" + """
    def calls(room, flow):
        fakes.fake_room(room)
        sim = cases.build_gpu(case, line_sweeps=0)
        if flow:
            sim.get_flow(0)
        check(sim.ctx, sim.L.gdfv_residual_jvp(sim.ctx, _p(U), _p(U), ffi.NULL, 0.0, _p(out[0]), sigma))
        check(sim.ctx, sim.L.gdfv_residual_vjp(sim.ctx, _p(U), _p(U), _p(out[1]), ffi.NULL))
        left = fakes.fake_room_left()
        sim.close()
        return left
    least = (1 << 40) - calls(1 << 40, False) - 9 * 8 * total   # without the buffer of the state's way in
    calls(least + 4096, False)
    calls(least + 4096, True)
    """)


def test_memory_is_not_taken_from_a_run_of_another_thread(tmp_path):
    """Products that find no memory while another thread steps the context: they fail or, between
    runs, take the sweeps' memory; the run's states are those of a run alone."""
    run_with_fakes(tmp_path, HEAD % "euler" + """
    import threading
    alone, sim = cases.build_gpu(case), cases.build_gpu(case)
    assert sim.option("line_sweeps") == 1
    for s in (alone, sim):
        assert s.run(max_step=1) == 1   # the steps are captured
    U.copy_(torch.from_numpy(sim.get_conserved(0)))
    torch.cuda.synchronize()
    errors = []
    def steps():
        try:
            for _ in range(10):
                assert sim.run(max_step=17) == 17
        except Exception as e:
            errors.append(repr(e))
    fakes.fake_room(0)
    t = threading.Thread(target=steps)
    t.start()
    refused = 0
    while t.is_alive():
        refused += sim.L.gdfv_residual_jvp(sim.ctx, _p(U), _p(U), ffi.NULL, 1e-3, _p(out[0]), sigma) != 0
    t.join()
    fakes.fake_room(-1)
    assert not errors, errors
    print("refused", refused, "sweeps", sim.option("line_sweeps"))
    assert alone.run(max_step=170) == 170
    assert np.array_equal(alone.get_conserved(0), sim.get_conserved(0))
    """)
