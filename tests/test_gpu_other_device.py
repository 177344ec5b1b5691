"""States and velocities of a handle are set and read from whichever device is
current in the calling thread (needs two devices; skipped on one).

Bound (written here): the bits that were set; the same bits read on either device.
"""
import threading

import numpy as np
import pytest

from rigidfibers_b200.generate import sphere_layout

pytestmark = pytest.mark.gpu


def test_state_is_set_and_read_with_another_device_current():
    import torch
    from rigidfibers_b200 import Config, Simulation
    if torch.cuda.device_count() < 2:
        pytest.skip("one device")
    pos, ori = sphere_layout(40, 5.0, 0.2, seed=3)
    with torch.cuda.device(1):
        sim = Simulation(Config(), pos, ori)
        sim.step(0)
        here = sim.state() + sim.velocities()
    with torch.cuda.device(0):
        there = sim.state() + sim.velocities()
        sim.set_state(pos, ori)
        assert torch.cuda.current_device() == 0
    got = []
    t = threading.Thread(target=lambda: got.append(sim.state()))   # a thread of its own: device 0
    t.start()
    t.join()
    for a, b in zip(here, there):
        assert np.array_equal(a, b)
    assert np.array_equal(got[0][0], pos) and np.array_equal(got[0][1], ori)
    with torch.cuda.device(1):
        sim.close()
