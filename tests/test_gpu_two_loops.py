"""Cooperative time loops of several patches, and a network's training, at the same time:
each launch wants every SM to itself, and its CTAs wait for one another (with a limit).
Three threads on their own streams, many launches each; the results are those of the
same calls one after another, bit for bit."""
import threading

import numpy as np
import pytest

from pyclaw_b200.learned import Network
from test_gpu_launch_shapes import _make

pytestmark = pytest.mark.gpu


def _loop(name, mx, my, calls):
    claw = _make(name, mx, my, 0, 2, 2)
    s, sol = claw.solver, claw.solution
    s.dt_variable, s.dt = False, 0.02 / mx

    def run():
        for _ in range(calls):
            s.evolve_to_time(sol, sol.t + 25 * s.dt)
        return sol.state.q.copy()
    return run


def _train():
    net = Network(seed=3)
    net.generate(1 << 18, seed=4)

    def run():
        net.train(20, 4096, 1e-3)
        return net.params.copy()
    return run


def _all():
    return [_loop("euler", 420, 390, 40), _loop("shallow", 400, 410, 40), _train()]


def test_loops_side_by_side():
    alone = [run() for run in _all()]
    together, errors, start = [None] * 3, [], threading.Barrier(3)

    def call(k, run):
        try:
            start.wait()
            together[k] = run()
        except Exception as e:  # (shown by the main thread)
            errors.append((k, e))
    threads = [threading.Thread(target=call, args=x) for x in enumerate(_all())]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for a, b in zip(alone, together):
        assert np.array_equal(a, b)
