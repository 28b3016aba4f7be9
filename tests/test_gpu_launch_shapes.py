"""The default launch shape of the unsplit step (CTAs per SM, row height) against the best
of forced ones, by the step kernel's own time: a tiling that counts CTAs an SM cannot hold
runs a second, half-empty wave, and a register cap for them spills for nothing.  The solver
whose tile is too large for three CTAs, the capacity forms (compiled without the cap) and
the solvers whose tiles leave room for more.

Bound: half a wave too many costs a third to a half of the step (1.4 to 1.9 times measured
where it happened); between that and the few per cent that rounding a height costs lies
1.25.  A batch of one problem adds its ghost fill and its record's update, 10 us."""
import numpy as np
import pytest

import pyclaw_b200 as pyclaw
from pyclaw_b200 import batch, riemann, tune
from pyclaw_b200.geometry import Dimension, Domain
from pyclaw_b200.solution import Solution
from pyclaw_b200.state import State

pytestmark = pytest.mark.gpu
E = pyclaw.BC.extrap
SOLVERS = {  # solver, waves, aux components
    "euler5": (riemann.euler_5wave_2D, 5, 0),
    "euler": (riemann.euler_4wave_2D, 4, 0),
    "shallow": (riemann.shallow_roe_with_efix_2D, 3, 0),
    "acoustics": (riemann.acoustics_2D, 2, 0),
    "vc_acoustics": (riemann.vc_acoustics_2D, 2, 2),
    "advection": (riemann.advection_2D, 1, 0),
}


class _Claw(object):
    pass


def _make(name, mx, my, capa, order, trans):
    rp, mwaves, naux = SOLVERS[name]
    s = pyclaw.ClawSolver2D(rp)
    s.num_waves, s.order, s.dimensional_split, s.transverse_waves, s.limiters = mwaves, order, False, trans, 4
    s.all_bcs, s.aux_bc_lower, s.aux_bc_upper = E, [E, E], [E, E]
    state = State(Domain([Dimension(0.0, 1.0, mx, name="x"), Dimension(0.0, 1.0, my, name="y")]), rp.num_eqn,
                  naux + capa)
    state.problem_data.update({"u": 0.5, "v": -1.0, "rho": 1.0, "bulk": 4.0, "cc": 2.0, "zz": 2.0, "gamma": 1.4,
                               "grav": 1.0})
    x, y = np.arange(mx)[:, None] / mx, np.arange(my)[None, :] / my
    f = [0.5 + 0.3 * np.sin((5 + k) * x + 3 * y) * np.cos(4 * y + k * x) for k in range(5)]
    if name in ("euler", "euler5"):
        r, u, v, p = 0.8 + f[0], f[1] - 0.5, f[2] - 0.5, 0.8 + f[3]
        q = [r, r * u, r * v, p / 0.4 + 0.5 * r * (u * u + v * v), f[4]]
    elif name == "shallow":
        q = [0.8 + f[0], f[1] - 0.5, f[2] - 0.5]
    else:
        q = f
    state.q = np.stack(q[:rp.num_eqn])
    if naux + capa:
        state.aux[...] = 0.7 + np.stack(f[:naux + capa])
    if capa:
        state.index_capa = naux
    claw = _Claw()
    claw.solver, claw.solution = s, Solution(state, Domain(state.grid.dimensions))
    s.setup(claw.solution)
    s.dt_initial = 0.1 / max(mx, my)
    return claw


def _ms(dev, dt):
    t = []
    for _ in range(8):
        dev.step(dt, want_cfl=False)
        dev.accept(False)
        t.append(dev.kernel_ms())
    return min(t[2:])


def _best_and_default(name, claw):
    rid, dev, dt = SOLVERS[name][0].rp_id, claw.solver._dev, claw.solver.dt_initial
    dev.set_timing(True)
    try:
        default = _ms(dev, dt)
        best = {}
        for variant in (0, 1):
            for rows in (4, 6, 8, 9, 10, 12, 14, 16, 18, 20, 24, 28, 32, 40, 48, 64):
                tune.set_shape(rid, variant, rows)
                best[variant, rows] = _ms(dev, dt)
    finally:
        tune.set_shape(rid, 0, 0)
    return min(best.values()), default, min(best, key=best.get)


@pytest.mark.parametrize("name,capa,order,trans", [
    ("euler5", 0, 2, 2), ("euler5", 0, 2, 1), ("euler", 0, 2, 2), ("shallow", 0, 2, 2), ("acoustics", 0, 2, 2),
    ("vc_acoustics", 0, 2, 2), ("advection", 0, 2, 2), ("advection", 0, 1, 0), ("euler5", 1, 2, 2),
    ("euler", 1, 2, 2), ("vc_acoustics", 1, 2, 2), ("acoustics", 1, 2, 2)])
@pytest.mark.parametrize("mx,my", [(600, 515), (1000, 858), (2000, 1715)])
def test_default_shape(name, capa, order, trans, mx, my):
    best, default, shape = _best_and_default(name, _make(name, mx, my, capa, order, trans))
    assert default <= 1.25 * best, (default, best, shape)


@pytest.mark.parametrize("name", ["euler5", "euler", "acoustics"])
def test_batch_of_one(name):
    claw = _make(name, 1000, 858, 0, 2, 2)
    best, _, shape = _best_and_default(name, claw)
    b = batch.Batch([claw])
    b.upload()
    b.set_time([claw.solver.dt_initial], 0.0, 1e99, 0.9, 1.0, 1e99)
    b.run(3, mode=1)
    ms = min(b.run(10, mode=1) for _ in range(3)) / 10
    assert ms <= 1.25 * best + 0.010, (ms, best, shape)
