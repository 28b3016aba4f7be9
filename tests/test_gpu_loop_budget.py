"""A launch of the cooperative time loop holds every SM, so it is bounded in time: while
a split Euler run of 1500 steps at 2500 x 2000 (0.36 ms a step) goes on in one thread,
a small kernel on another stream has to get through between two launches.  Bounded at
about 20 ms of work a launch; unbounded, 1024 attempts, it was 0.37 s.  The test allows
0.15 s, for the host's scheduling on top."""
import threading
import time

import numpy as np
import pytest
import torch

from test_gpu_launch_shapes import _make

pytestmark = pytest.mark.gpu


def test_other_streams_get_through():
    claw = _make("euler", 2500, 2000, 0, 2, 0)
    s, sol = claw.solver, claw.solution
    s._dev.close()
    s.dimensional_split, s.dt_variable, s.dt = True, False, 0.01 / 2500
    s.setup(sol)
    s.evolve_to_time(sol, 2 * s.dt)  # (buffers, launch attributes)
    other, x = torch.cuda.Stream(), torch.zeros(1024, device="cuda")
    with torch.cuda.stream(other):
        x += 1.0
    other.synchronize()
    steps, t0 = 1500, sol.t
    run = threading.Thread(target=s.evolve_to_time, args=(sol, t0 + steps * s.dt))
    waits = []
    run.start()
    time.sleep(0.02)
    while run.is_alive():
        t = time.perf_counter()
        with torch.cuda.stream(other):
            x += 1.0
        other.synchronize()
        waits.append(time.perf_counter() - t)
        time.sleep(0.002)
    run.join()
    assert s.status["numsteps"] == steps + 2
    assert np.isfinite(sol.state.q).all()
    assert len(waits) >= 3 and max(waits) <= 0.15, (len(waits), max(waits))
