"""Tiles at rest in the device time loop (passed over while they and their
neighbours do not change): a disturbance that starts in one tile of a grid at
rest, crosses the others and meets every kind of boundary, on small row
blocks (so there are many tiles), with ragged last strips and blocks, cells
holding -0.0, a moving uniform state and a rejected first dt, against the host
loop, which computes every tile every step.  Two instantiations of the same
tile source: 1e-13 as in the device-loop tests, counts exactly; and the part
that is still at rest is returned bit for bit."""
import numpy as np
import pytest

import pyclaw_b200 as pyclaw
from helpers import max_rel
from pyclaw_b200 import _lib, riemann, tune
from pyclaw_b200.geometry import Dimension, Domain
from pyclaw_b200.solution import Solution
from pyclaw_b200.state import State

pytestmark = pytest.mark.gpu
E, P, W = pyclaw.BC.extrap, pyclaw.BC.periodic, pyclaw.BC.wall


def _solve(rp, rid, data, q, lower, upper, shape, device_loop, tend, dt):
    tune.set_shape(rid, *shape)
    try:
        s = pyclaw.ClawSolver2D(rp)
        s.dimensional_split, s.transverse_waves, s.limiters = False, 2, pyclaw.limiters.tvd.MC
        s.bc_lower, s.bc_upper = list(lower), list(upper)
        s.device_time_loop = device_loop
        mx, my = q.shape[1:]
        state = State(Domain([Dimension(0.0, mx * 1.0, mx, name="x"), Dimension(0.0, my * 1.0, my, name="y")]),
                      q.shape[0])
        state.problem_data.update(data)
        state.q = q.copy()
        sol = Solution(state, Domain(state.grid.dimensions))
        s.setup(sol)
        s.dt = dt
        for t in (0.4 * tend, tend):  # two calls: the flags of the first must not outlive it
            s.evolve_to_time(sol, t)
        return s, sol
    finally:
        tune.set_shape(rid, 0, 0)


def _both(name, mx, my, at, lower, upper, shape, tend, dt=0.3, base=(0.0, 0.0)):
    if name == "shallow":
        rp, rid, data = riemann.shallow_roe_with_efix_2D, _lib.RP_SHALLOW_ROE, {"grav": 1.0}
        q = np.empty((3, mx, my))
        q[0], q[1], q[2] = 1.0, base[0], base[1]
        q[0, at[0]:at[0] + 3, at[1]:at[1] + 2] = 2.0
    else:
        rp, rid, data = riemann.euler_4wave_2D, _lib.RP_EULER_ROE, {"gamma": 1.4}
        q = np.empty((4, mx, my))
        q[0], q[1], q[2] = 1.0, base[0], base[1]
        q[3] = 2.5 + 0.5 * (base[0] ** 2 + base[1] ** 2)
        q[3, at[0]:at[0] + 3, at[1]:at[1] + 2] += 2.0
    (a, sa), (b, sb) = (_solve(rp, rid, data, q, lower, upper, shape, loop, tend, dt) for loop in (True, False))
    assert a.status["numsteps"] == b.status["numsteps"] >= 6
    assert abs(a.cfl.get_cached_max() - b.cfl.get_cached_max()) <= 1e-13 * b.cfl.get_cached_max()
    assert abs(a.dt - b.dt) <= 1e-13 * b.dt
    assert max_rel(sa.state.q, sb.state.q) <= 1e-13
    rest = (sb.state.q == q).all(0)
    assert (sa.state.q[:, rest] == q[:, rest]).all()
    return rest


@pytest.mark.parametrize("name", ["shallow", "euler"])
@pytest.mark.parametrize("variant", [0, 1, 3])
@pytest.mark.parametrize("mx,my,at", [(300, 61, (122, 7)), (249, 40, (0, 39)), (374, 33, (371, 0))])
@pytest.mark.parametrize("lower,upper", [((E, W), (W, E)), ((P, P), (P, P)), ((W, P), (E, P))])
def test_disturbance_crosses_tiles(name, variant, mx, my, at, lower, upper):
    at = (min(at[0], mx - 3), min(at[1], my - 2))
    rest = _both(name, mx, my, at, lower, upper, (variant, 4), 12.0)
    assert rest.any() and not rest.all()


def test_uniform_motion_and_negative_zero():
    # a uniform stream (at rest in the sense of the tiles), then cells of -0.0
    _both("shallow", 260, 50, (130, 20), (E, E), (E, E), (1, 4), 8.0, base=(0.3, -0.2))
    _both("shallow", 260, 50, (130, 20), (P, P), (P, P), (1, 4), 8.0, base=(-0.0, 0.0))


def test_rejected_first_step():
    _both("euler", 260, 50, (130, 20), (E, E), (W, W), (1, 4), 8.0, dt=5.0)


def test_one_row_blocks_are_all_computed():
    _both("shallow", 200, 30, (100, 10), (P, P), (P, P), (0, 1), 6.0)
