"""The small-grid form of the device time loop (one cooperative kernel, tiles
of 28 x 12 written cells, or 28 x 4 for the largest records): sizes at and
around the edges of a tile, every boundary rule, both splittings, solvers with
and without aux data, a run longer than one launch's budget of attempts, and
rejected steps, against the host loop (the marching kernels, which the parity
tests hold to the oracle).

Tolerance: the two evaluate the same formulas with other orders of summation,
a few ulps of O(1) data per step and growing by at most the CFL's factor of
order one per step: 1e-13 over the few steps taken, as in the device-loop
tests; counts exactly."""
import numpy as np
import pytest

import pyclaw_b200 as pyclaw
from helpers import max_rel
from pyclaw_b200 import riemann
from pyclaw_b200.geometry import Dimension, Domain
from pyclaw_b200.solution import Solution
from pyclaw_b200.state import State

pytestmark = pytest.mark.gpu
RTOL = 1e-13

SOLVERS = {  # solver, waves, aux components
    "advection": (riemann.advection_2D, 1, 0),
    "acoustics": (riemann.acoustics_2D, 2, 0),
    "euler": (riemann.euler_4wave_2D, 4, 0),
    "euler5": (riemann.euler_5wave_2D, 5, 0),
    "shallow": (riemann.shallow_roe_with_efix_2D, 3, 0),
    "hlle": (riemann.shallow_hlle_2D, 2, 0),
    "vc_acoustics": (riemann.vc_acoustics_2D, 2, 2),
    "vc_advection": (riemann.vc_advection_2D, 1, 2),
    "psystem": (riemann.psystem_2D, 2, 4),
}
DATA = {"u": 0.5, "v": -1.0, "rho": 1.0, "bulk": 4.0, "cc": 2.0, "zz": 2.0, "gamma": 1.4, "grav": 1.0}


def _make(name, mx, my, split, trans, limiter, lower, upper, device_loop, dt):
    rp, mwaves, naux = SOLVERS[name]
    rng = np.random.default_rng(mx * 1000 + my)
    s = pyclaw.ClawSolver2D(rp)
    s.num_waves = mwaves
    s.dimensional_split, s.transverse_waves, s.limiters = split, trans, limiter
    s.bc_lower, s.bc_upper = list(lower), list(upper)
    s.aux_bc_lower = [b for b in lower]
    s.aux_bc_upper = [b for b in upper]
    s.device_time_loop = device_loop
    s.dt_initial = dt
    state = State(Domain([Dimension(0.0, 1.0, mx, name="x"), Dimension(0.0, 1.3, my, name="y")]), rp.num_eqn, naux)
    state.problem_data.update(DATA)

    def field(lo, hi):  # constant in the left half, rough in the right
        f = rng.uniform(lo, hi, (mx, my))
        f[: mx // 2] = 0.5 * (lo + hi)
        return f

    if name in ("euler", "euler5"):
        r, u, v, p = field(0.8, 1.2), field(-0.3, 0.3), field(-0.3, 0.3), field(0.8, 1.2)
        q = [r, r * u, r * v, p / 0.4 + 0.5 * r * (u * u + v * v)] + ([field(0, 1)] if name == "euler5" else [])
    elif name in ("shallow", "hlle"):
        h = field(0.8, 1.2)
        q = [h, h * field(-0.3, 0.3), h * field(-0.3, 0.3)]
    else:
        q = [field(-0.2, 0.3) for _ in range(rp.num_eqn)]
    state.q = np.stack(q)
    if naux == 2:
        state.aux[...] = rng.uniform(0.5, 2.0, state.aux.shape)
    if naux == 4:
        state.aux[...] = np.stack([field(1, 4), field(1, 4), np.where(rng.random((mx, my)) < 0.5, 1.0, 2.0), q[0]])
    return s, Solution(state, state.patch and Domain(state.grid.dimensions))


def _run(tend, *args):
    out = []
    for device_loop in (True, False):
        s, sol = _make(*args[:-1], device_loop, args[-1])
        s.setup(sol)
        s.dt = s.dt_initial
        s.evolve_to_time(sol, tend)
        out.append((s, sol))
    (a, sa), (b, sb) = out
    assert a.status["numsteps"] == b.status["numsteps"]
    assert abs(sa.t - sb.t) <= RTOL * sb.t and abs(a.dt - b.dt) <= RTOL * b.dt
    assert abs(a.cfl.get_cached_max() - b.cfl.get_cached_max()) <= RTOL * b.cfl.get_cached_max()
    assert max_rel(sa.state.q, sb.state.q) <= RTOL
    return a.status["numsteps"]


E, P, W = pyclaw.BC.extrap, pyclaw.BC.periodic, pyclaw.BC.wall


@pytest.mark.parametrize("mx,my", [(28, 12), (29, 13), (27, 11), (56, 4), (57, 25), (300, 3), (3, 150), (2, 2)])
@pytest.mark.parametrize("name,split", [("acoustics", False), ("acoustics", True), ("euler", False), ("euler", True)])
@pytest.mark.parametrize("lower,upper", [((E, W), (W, E)), ((P, W), (P, W)), ((W, P), (E, P))])
def test_tile_edges_and_boundaries(name, split, mx, my, lower, upper):
    h = min(1.0 / mx, 1.3 / my)
    assert _run(1.2 * h, name, mx, my, split, 2, pyclaw.limiters.tvd.MC, lower, upper, 0.2 * h) >= 3


@pytest.mark.parametrize("name", sorted(SOLVERS))
@pytest.mark.parametrize("split,trans,limiter", [(True, 0, 1), (True, 0, 3), (False, 1, 2), (False, 2, 4)])
def test_solvers(name, split, trans, limiter):
    if name == "hlle" and not split:
        trans = 0  # has no transverse solver
    h = 1.0 / 61
    # (the slowest, at speed 1, take two steps)
    assert _run(1.0 * h, name, 61, 45, split, trans, limiter, (E, W), (E, E), 0.15 * h) >= 2


def test_one_cell():
    assert _run(2.0, "euler", 1, 1, False, 2, 4, (E, E), (E, E), 0.1) >= 3


def test_first_dt_rejected():
    assert _run(0.05, "shallow", 70, 50, False, 2, 4, (E, E), (E, E), 0.5) >= 3


def test_more_attempts_than_one_launch():
    # advection at a fixed speed on 8 x 8 cells: 1600 attempts, the budget of a launch is 1024
    s, sol = _make("advection", 8, 8, True, 0, 1, (P, P), (P, P), True, 0.01)
    s.dt_variable = False
    s.setup(sol)
    s.dt = s.dt_initial
    s.evolve_to_time(sol, 16.0)
    assert s.status["numsteps"] == 1600 and abs(sol.t - 16.0) < 1e-9
    assert np.isfinite(sol.state.q).all()
