"""States and results across the bus: one chunk, and the edges of several
(5461 fibers or 65536 solution entries fill the page-locked block).

Bounds (written here): states come back as they were set, bit for bit; after a
first step every position is the one before plus timestep times its velocity
to 1e-12 (FP64 update, FP32 velocities); the fetched solution satisfies the
fetched right-hand side to 1e-5 relative (solved to 1e-6, FP32 products).
"""
import numpy as np
import pytest

from rigidfibers_b200.generate import sphere_layout

pytestmark = pytest.mark.gpu


def _layout(n):
    return sphere_layout(n, (n / 0.1) ** (1.0 / 3.0) + 1.0, 0.2, seed=50 + n)


@pytest.mark.parametrize("n", [1, 2, 43, 5461, 5462, 10923])
def test_state_round_trip(n):
    from rigidfibers_b200 import Config, Simulation
    rng = np.random.default_rng(n)
    s = Simulation(Config(precision="matrix_free"), np.zeros((n, 3)), np.tile([1.0, 0.0, 0.0], (n, 1)))
    pos, ori = rng.standard_normal((n, 3)), rng.standard_normal((n, 3))
    s.set_state(pos, ori)
    p, o = s.state()
    s.close()
    assert np.array_equal(p, pos) and np.array_equal(o, ori)


@pytest.mark.parametrize("n", [3, 4369, 4370, 5600])
def test_results_of_a_first_step(n):
    from rigidfibers_b200 import Config, Simulation
    pos, ori = _layout(n)
    s = Simulation(Config(precision="mixed_fp16", timestep=0.1), pos, ori)
    s.assembleSystem()
    s.solveSystem()
    x = s.solution()
    _, b = s.system(with_matrix=False)
    assert np.abs(s.apply_operator(x) - b).max() <= 1e-5 * np.abs(b).max()
    s.set_state(pos, ori)
    s.step(0)
    p1, _ = s.state()
    tvel, _ = s.velocities()
    s.close()
    assert np.abs(p1 - (pos + 0.1 * tvel)).max() <= 1e-12 * np.abs(pos).max()
    assert np.abs(tvel).max() > 0
