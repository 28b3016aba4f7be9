"""A launch of the training kernel holds every SM, so it is bounded in time as the time
loop's: while an epoch over 2^28 samples in minibatches of 65536 goes on in one thread,
a small kernel on another stream has to get through between two launches (about 20 ms
each; 4096 minibatches a launch were 0.15 s).  The test allows 0.08 s."""
import threading
import time

import numpy as np
import pytest
import torch

from pyclaw_b200.learned import Network

pytestmark = pytest.mark.gpu


def test_other_streams_get_through():
    net = Network(seed=2)
    net.generate(1 << 28, seed=6)
    net.train(1, 1 << 28, 1e-3)  # (one minibatch: the kernel is loaded)
    other, x = torch.cuda.Stream(), torch.zeros(1024, device="cuda")
    with torch.cuda.stream(other):
        x += 1.0
    other.synchronize()
    loss, waits = [], []
    run = threading.Thread(target=lambda: loss.append(net.train(2, 65536, 1e-3)))
    run.start()
    time.sleep(0.002)
    while run.is_alive():
        t = time.perf_counter()
        with torch.cuda.stream(other):
            x += 1.0
        other.synchronize()
        waits.append(time.perf_counter() - t)
        time.sleep(0.002)
    run.join()
    assert np.isfinite(net.params).all() and loss[0] < 0.2
    assert len(waits) >= 3 and max(waits) <= 0.08, (len(waits), max(waits))
    net.close()
