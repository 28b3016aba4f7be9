"""The Roe solvers' eigenvector-coordinate forms where they can go wrong: the
root-free transonic test of the entropy fix on data full of transonic
rarefactions in both directions, and limiter ratios whose squared norms leave
the range of a double (a tiny shear wave beside an ordinary one), against the
oracle at 1e-12 (rounding of a step of O(1) data, as in the parity tests)."""
import numpy as np
import pytest

from helpers import PARITY_RTOL, RP_INFO, max_rel, method_vector, set_cparam
from pyclaw_b200 import _lib, classic2

pytestmark = pytest.mark.gpu

ROE = [_lib.RP_EULER_ROE, _lib.RP_SHALLOW_ROE]


def _compare(oracle, rp, qbc, lim, split, dt_cfl=0.4):
    name, meqn, mwaves, cp = RP_INFO[rp]
    mx, my = qbc.shape[1] - 4, qbc.shape[2] - 4
    mthlim = np.full(mwaves, lim, dtype=np.intc)
    set_cparam(classic2, rp)
    dx = dy = 0.01
    dt = dt_cfl * dx / 6.0  # speeds stay below 6
    for ids in (1, 2) if split else (0,):
        method = method_vector(2, 0 if split else 2, split=split)
        q_o = qbc.copy(order="F")
        if split:
            cfl_o = oracle.step2ds(qbc, q_o, dx, dy, dt, method, mthlim, ids, rp, cp)
            q_g, cfl_g = classic2.step2ds(max(mx, my), 2, mx, my, qbc, qbc.copy(order="F"), None, dx, dy, dt, method,
                                          mthlim, ids=ids, rpn2=rp)
        else:
            cfl_o = oracle.step2(qbc, q_o, dx, dy, dt, method, mthlim, rp, cp)
            q_g, cfl_g = classic2.step2(max(mx, my), 2, mx, my, qbc, qbc.copy(order="F"), None, dx, dy, dt, method,
                                        mthlim, rpn2=rp)
        assert np.isfinite(q_o).all()
        assert abs(cfl_g - cfl_o) <= PARITY_RTOL * cfl_o
        assert max_rel(q_g[:, 2:-2, 2:-2], q_o[:, 2:-2, 2:-2]) <= PARITY_RTOL


@pytest.mark.parametrize("rp", ROE)
@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("mx,my", [(130, 37), (41, 67)])
def test_transonic_rarefactions(oracle, rp, split, mx, my):
    rng = np.random.default_rng(mx + my)
    shape = (mx + 4, my + 4)
    # smooth-ish states whose u - c and u + c change sign again and again
    u, v = (rng.choice([-1.0, 1.0], shape) * rng.uniform(0.7, 1.4, shape) for _ in range(2))
    h = rng.uniform(0.8, 1.3, shape)
    if rp == _lib.RP_EULER_ROE:
        p = rng.uniform(0.6, 1.1, shape)
        q = np.stack([h, h * u, h * v, p / 0.4 + 0.5 * h * (u * u + v * v)])
    else:
        q = np.stack([h, h * u, h * v])
    _compare(oracle, rp, np.asfortranarray(q), 4, split)


@pytest.mark.parametrize("rp", ROE)
@pytest.mark.parametrize("lim", [1, 2, 3, 4])
@pytest.mark.parametrize("split", [False, True])
def test_waves_out_of_squared_range(oracle, rp, lim, split):
    rng = np.random.default_rng(lim)
    mx, my = 133, 21
    shape = (mx + 4, my + 4)
    h = 1.0 + 0.1 * rng.random(shape)
    # shear strengths from 1e-3 down to 1e-300 from one column to the next, and exact zeros
    mag = 10.0 ** -rng.choice([3.0, 60.0, 154.0, 162.0, 200.0, 300.0], shape)
    hv = np.where(rng.random(shape) < 0.2, 0.0, mag * rng.choice([-1.0, 1.0], shape))
    hu = np.zeros(shape)
    if rp == _lib.RP_EULER_ROE:
        q = np.stack([np.ones(shape), hu, hv, 2.5 * h])
    else:
        q = np.stack([h, hu, hv])
    _compare(oracle, rp, np.asfortranarray(q), lim, split)
