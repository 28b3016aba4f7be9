"""The marching form of the device time loop at small sizes, where a patch's default is the
cooperative kernel: every solver family with and without aux data, both splittings, the
default launch shape and one with many row blocks, against the host loop.  Two calls: the
first from the caller's own dt (four attempts, then the captured graph from the first
record), the second from a Courant number that makes its first dt nearly twice too large,
so that one attempt is rejected and the attempts issued ahead, nine, run out in the middle:
the graph continues from the second record.  Then a fixed dt over more attempts than one
chunk holds, and its Courant failure.

Tolerance: the loop's kernels are other instantiations of the same source, a few ulps per
step on O(1) data, growing by at most a factor of order one over the thirty steps: 1e-12;
counts exactly.  Sixteen hundred steps of a monotone advection step do not amplify what
they are given and add at most eight roundings each: 1600 * 8 * 2^-53 = 1.5e-12."""
import numpy as np
import pytest

import pyclaw_b200 as pyclaw
from helpers import max_rel
from pyclaw_b200 import tune
from pyclaw_b200._lib import NonFiniteError
from pyclaw_b200.solver import CFLError
from test_gpu_small_grid import SOLVERS, _make

pytestmark = pytest.mark.gpu
RTOL = 1e-12
E, P, W = pyclaw.BC.extrap, pyclaw.BC.periodic, pyclaw.BC.wall


def _setup(device_loop, name, mx, my, split, trans, limiter, dt, lower=(E, W), upper=(E, E)):
    s, sol = _make(name, mx, my, split, trans, limiter, lower, upper, device_loop, dt)
    s.setup(sol)
    s._dev.set_marching(True)
    s.dt = dt
    return s, sol


def _same(a, sa, b, sb, rtol=RTOL):
    assert a.status["numsteps"] == b.status["numsteps"]
    assert abs(sa.t - sb.t) <= rtol * sb.t and abs(a.dt - b.dt) <= rtol * b.dt
    assert abs(a.cfl.get_cached_max() - b.cfl.get_cached_max()) <= rtol * b.cfl.get_cached_max()
    assert max_rel(sa.state.q, sb.state.q) <= rtol


@pytest.mark.parametrize("name", sorted(SOLVERS))
@pytest.mark.parametrize("split,trans,limiter", [(True, 0, 1), (False, 1, 2), (False, 2, 4)])
@pytest.mark.parametrize("shape", [(0, 0), (1, 8)])
def test_marching_loop_equals_host_loop(name, split, trans, limiter, shape):
    if name == "hlle" and not split:
        pytest.skip("has no transverse solver: unstable at this Courant number")
    if split and shape != (0, 0):
        pytest.skip("the shape is the unsplit step's")
    mx, my = 130, 61
    rid = SOLVERS[name][0].rp_id
    tune.set_shape(rid, *shape)
    try:
        out = []
        for device_loop in (True, False):
            s, sol = _setup(device_loop, name, mx, my, split, trans, limiter, 0.0003)
            s.evolve_to_time(sol, 0.07)
            first = s.status["numsteps"]
            big = 1.9 * s.dt * s.cfl_desired / s.cfl.get_cached_max()
            s.cfl.set_global_max(s.cfl.get_cached_max() / 1.9)
            s.evolve_to_time(sol, sol.t + 7.9 * big)
            out.append((s, sol, first))
    finally:
        tune.set_shape(rid, 0, 0)
    (a, sa, na), (b, sb, nb) = out
    assert na == nb >= 4
    assert b.status["numsteps"] - nb >= 13  # more than the nine attempts issued ahead
    _same(a, sa, b, sb)


@pytest.mark.parametrize("name", ["acoustics", "vc_acoustics", "vc_advection", "euler5"])
@pytest.mark.parametrize("split", [True, False])
def test_fixed_dt(name, split):
    mx, my = 130, 61
    out = []
    for device_loop in (True, False):
        s, sol = _setup(device_loop, name, mx, my, split, 0 if split else 2, 4, 0.0)
        s.dt_variable, s.dt = False, 0.05 / mx / 4.0
        s.evolve_to_time(sol, 75 * s.dt)
        out.append((s, sol))
    (a, sa), (b, sb) = out
    assert a.status["numsteps"] == 75
    _same(a, sa, b, sb)
    # a dt far above the limit: the loop fails as the host's does (a Courant number too
    # large, or before it a state that is not finite), its step dropped
    q, raised = sa.state.q.copy(), []
    for s, sol in out:
        s.dt = 50.0 / mx
        with pytest.raises((CFLError, NonFiniteError)) as e:
            s.evolve_to_time(sol, sol.t + 4 * s.dt)
        raised.append(e.type)
    assert raised[0] is raised[1] and (name == "euler5" or raised[0] is CFLError)
    assert np.array_equal(sa.state.q, q)


def test_switching_a_patch_between_the_forms():
    # the same patch: cooperative, marching, cooperative, against one that stays marching
    out = []
    for switch in (True, False):
        s, sol = _setup(True, "shallow", 130, 61, False, 2, 4, 0.001)
        for k in range(3):
            s._dev.set_marching(k == 1 or not switch)
            s.evolve_to_time(sol, 0.02 * (k + 1))
        out.append((s, sol))
    _same(*out[0], *out[1])


def test_more_attempts_than_a_cooperative_launch_takes():
    out = []
    for device_loop in (True, False):
        s, sol = _make("advection", 8, 8, True, 0, 1, (P, P), (P, P), device_loop, 0.01)
        s.dt_variable = False
        s.setup(sol)
        s.dt = s.dt_initial
        s.evolve_to_time(sol, 16.0)
        out.append((s, sol))
    (a, sa), (b, sb) = out
    assert a.status["numsteps"] == b.status["numsteps"] == 1600
    assert max_rel(sa.state.q, sb.state.q) <= 1.5e-12
