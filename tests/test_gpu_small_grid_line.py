"""Where the time loop leaves the cooperative kernel, for the solver whose record leaves it
half a tile (28 x 4 written of 32 x 8 cells): a split step of the loop against the same
two sweeps issued one step at a time, by the events around them, and against the unsplit
loop with a marching shape forced.  The sweeps are the marching loop's kernels, whose
attempts add one launch of 4 to 8 us; the half tile on the wrong side of the line costs
1.3 times (measured 147 against 111 us at 1000 x 858, 578 against 405 at 2000 x 1715,
unsplit with minmod 66 against 50 at 450 x 386): the bound is 1.15 and 10 us (unsplit 3).  Results of both forms agree as in the marching tests."""
import time

import pytest

from helpers import max_rel
from pyclaw_b200 import riemann, tune
from test_gpu_launch_shapes import _make

pytestmark = pytest.mark.gpu


def _split(mx, my, device_loop=True):
    claw = _make("euler5", mx, my, 0, 2, 0)
    s = claw.solver
    s._dev.close()
    s.dimensional_split, s.dt_variable, s.device_time_loop = True, False, device_loop
    s.dt = 0.05 / mx
    s.setup(claw.solution)
    return s, claw.solution


def _us(s, sol, steps):
    def run():
        tend = sol.t + steps * s.dt
        t0 = time.perf_counter()
        s.evolve_to_time(sol, tend)
        return (time.perf_counter() - t0) / steps * 1e6
    run()
    return min(run() for _ in range(4))


@pytest.mark.parametrize("mx,my", [(1000, 858), (2000, 1715)])
def test_split_loop_is_no_slower_than_its_sweeps(mx, my):
    s, sol = _split(mx, my)
    loop = _us(s, sol, 20)
    s._dev.set_timing(True)
    ms = []
    for _ in range(8):
        s._dev.step(s.dt, want_cfl=False)
        s._dev.accept(False)
        ms.append(s._dev.kernel_ms())
    assert loop <= 1.15 * min(ms) * 1e3 + 10.0, (loop, min(ms) * 1e3)


@pytest.mark.parametrize("mx,my", [(450, 386), (470, 388)])  # 11 tiles per SM
def test_unsplit_loop_is_no_slower_than_a_march(mx, my):
    claw = _make("euler5", mx, my, 0, 2, 1)
    s, sol, rid = claw.solver, claw.solution, riemann.euler_5wave_2D.rp_id
    s._dev.close()
    s.dt_variable, s.dt, s.limiters = False, 0.05 / mx, 1
    s.setup(sol)
    loop = _us(s, sol, 20)
    march = []
    try:
        for rows in (6, 8, 9, 10, 12, 16):
            tune.set_shape(rid, 0, rows)
            march.append(_us(s, sol, 20))
    finally:
        tune.set_shape(rid, 0, 0)
    assert loop <= 1.15 * min(march) + 3.0, (loop, march)


@pytest.mark.parametrize("mx,my", [(530, 472), (560, 480)])  # 118 x 19 and 120 x 20 tiles: either side of 16 per SM
def test_split_results_on_both_sides(mx, my):
    out = []
    for device_loop in (True, False):
        s, sol = _split(mx, my, device_loop)
        s.evolve_to_time(sol, 12 * s.dt)
        out.append((s.status["numsteps"], sol.state.q.copy()))
    assert out[0][0] == out[1][0] == 12
    assert max_rel(out[0][1], out[1][1]) <= 1e-12
