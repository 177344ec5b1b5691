"""Distances at which the far pairs' rule must not be used: centres that are not
numbers, and distances whose squares overflow FP32.

A single fiber sinks by itself wherever it is, infinitely far from the origin or
nowhere (its position is not read).  Two fibers on one axis 1e20 apart, or 1e18
(where squares are still finite), do not feel each other: the kernel's FP32
values are 0, or below 1e-17 of the fibers' own terms.  Either way the
velocities are the single fiber's, to the last bit or two (4 roundings of 6e-8
relative to the largest component).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MODES = {"fp32": {}, "mixed_fp16": dict(precision="mixed_fp16"), "recompute": dict(precision="mixed_fp16_recompute"),
         "matrix_free": dict(precision="matrix_free"), "analytical": dict(integration="analytical")}


def _velocities(pos, ori, kw):
    from rigidfibers_b200 import Config, Simulation
    with Simulation(Config(**kw), np.asarray(pos, float), np.asarray(ori, float)) as s:
        s.step(0)
        return s.velocities()


@pytest.mark.parametrize("where", [np.nan, np.inf, 1e30])
@pytest.mark.parametrize("mode", sorted(MODES))
def test_single_fiber_anywhere(mode, where):
    t = [[0.6, 0.0, 0.8]]
    got = _velocities([[where, 0.0, 1.0]], t, MODES[mode])
    want = _velocities([[0.0, 0.0, 0.0]], t, MODES[mode])
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])


# the closed form divides by the distance from the other fiber's axis: not for fibers on one axis
@pytest.mark.parametrize("mode", sorted(set(MODES) - {"analytical"}))
@pytest.mark.parametrize("dist", [1e18, 1e20, 1e30])
def test_two_fibers_out_of_reach(mode, dist):
    got = _velocities([[0.0, 0.0, 0.0], [0.0, 0.0, dist]], [[0.0, 0.0, 1.0]] * 2, MODES[mode])
    want = _velocities([[0.0, 0.0, 0.0]], [[0.0, 0.0, 1.0]], MODES[mode])
    for g, w in zip(got, want):
        assert np.abs(g - w).max() <= 2.4e-7 * np.abs(want[0]).max()
