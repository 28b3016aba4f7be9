"""Rounding of the variable-coefficient acoustics solver's strengths, whose divisions by the
sum of two impedances are reciprocal products on the device: one first-order step of data
that vary in x only, from zero pressure, so that the new pressure is the fluctuations alone
(no final sum hides their rounding), against extended precision on the scale of its two
terms.  The yardstick is the same expressions with divisions in double precision: the
device's rms error may be at most that, and 2% for the sampling of 200000 cells (0.2% each)."""
import numpy as np
import pytest

from pyclaw_b200 import classic2, riemann

pytestmark = pytest.mark.gpu


def _pressure(t, u, rho, c, r):
    u, rho, c, r = (np.asarray(z, dtype=t) for z in (u, rho, c, r))
    z = rho * c
    zl, zr, cl, cr = z[:-1], z[1:], c[:-1], c[1:]
    d2 = u[1:] - u[:-1]
    left = cl * (zr * d2 / (zl + zr)) * zl    # -c_l times the pressure of the left-going wave
    right = cr * (zl * d2 / (zl + zr)) * zr
    a, b = right[1:-2], left[2:-1]            # of cells 2 .. : what enters from the left, and from the right
    return -r * (a + b), r * (abs(a) + abs(b))


def test_strengths_round_as_divisions_do():
    if np.finfo(np.longdouble).nmant < 63:
        pytest.skip("no extended precision here")
    mx, my, r = 200000, 1, np.random.default_rng(7)
    u, rho, c = r.uniform(-1, 1, mx + 4), r.uniform(0.5, 2.0, mx + 4), r.uniform(0.5, 2.0, mx + 4)
    q, aux = np.zeros((3, mx + 4, my + 4), order="F"), np.empty((2, mx + 4, my + 4), order="F")
    q[1], aux[0], aux[1] = u[:, None], rho[:, None], c[:, None]
    dx = 0.01
    dt = 0.3 * dx / 2.0
    out, _ = classic2.step2(mx, 2, mx, my, q, q.copy(order="F"), aux, dx, 1.0, dt,
                            np.array([1, 1, 0, 0, 0, 0, 2], dtype=np.intc), np.zeros(2, dtype=np.intc),
                            rpn2=riemann.vc_acoustics_2D)
    got = out[0, 2:-2, 2]
    ref, scale = _pressure(np.longdouble, u, rho, c, np.longdouble(dt / dx))
    plain, _ = _pressure(np.float64, u, rho, c, dt / dx)

    def rms(x):
        return float(np.sqrt(np.mean(((x - ref) / scale).astype(float) ** 2)))

    assert len(got) == len(ref) == mx
    assert rms(got) <= 1.02 * rms(plain), (rms(got), rms(plain))
