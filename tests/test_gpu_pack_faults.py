"""A bounded wait of the packed solve that runs out (forced by a zero wait
limit: the wait gives up before the copy it waits for is looked at, and the
copy is then waited for) is reported as RF_E_TIMEOUT by every member, leaves
the states as they were, and the next step gives the bits it would have given.

Members: one storage tile, a single CTA, a cluster with a ragged last tile.
"""
import numpy as np
import pytest

from rigidfibers_b200.generate import sphere_layout

pytestmark = pytest.mark.gpu


@pytest.fixture
def lib():
    from rigidfibers_b200 import _capi as C
    lib = C.load()
    yield lib
    lib.rf_debug_set_device_wait_limit(-1)


def _sims():
    from rigidfibers_b200 import Config, Simulation
    lays = [sphere_layout(n, (n / 0.5) ** (1.0 / 3.0) + 1.0, 0.2, seed=60 + n) for n in (5, 40, 201)]
    return [Simulation(Config(precision="mixed_bf16"), pos, ori) for pos, ori in lays]


def test_packed_step_reports_a_lost_copy_and_goes_on(lib):
    from rigidfibers_b200 import _capi as C
    from rigidfibers_b200.simulation import step_packed
    sims, want = _sims(), _sims()
    assert step_packed(sims, [0] * 3) == [C.RF_OK] * 3
    step_packed(want, [0] * 3)
    before = [s.state() for s in sims]
    lib.rf_debug_set_device_wait_limit(0)
    assert step_packed(sims, [1] * 3) == [C.RF_E_TIMEOUT] * 3
    lib.rf_debug_set_device_wait_limit(-1)
    for s, (p, o) in zip(sims, before):
        assert np.array_equal(s.state()[0], p) and np.array_equal(s.state()[1], o)
    assert step_packed(sims, [1] * 3) == [C.RF_OK] * 3
    step_packed(want, [1] * 3)
    for s, w in zip(sims, want):
        assert np.array_equal(s.state()[0], w.state()[0]) and np.array_equal(s.solution(), w.solution())


def test_packed_solve_reports_a_lost_copy(lib):
    from rigidfibers_b200 import _capi as C
    from rigidfibers_b200.simulation import solve_packed
    sims = _sims()
    for s in sims:
        s.assembleSystem()
    lib.rf_debug_set_device_wait_limit(0)
    with pytest.raises(C.RigidFibersError) as e:
        solve_packed(sims)
    assert e.value.status == C.RF_E_TIMEOUT
    lib.rf_debug_set_device_wait_limit(-1)
    solve_packed(sims)
    assert all(np.isfinite(s.solution()).all() for s in sims)
