"""The far pairs' quadrature rule (8 points per fiber, the Gauss rule of the
full rule's discrete measure) against the FP64 oracle's full rule.

Bounds (written here): a block entry is a sum of 8 x 8 kernel values of FP32
accuracy, about 30 roundings of 6e-8 relative to the block's largest entry, so
dense entries within 4e-6 of the largest off-diagonal one (the rule itself is
within 3e-10).  The right-hand side of a dilute suspension sums T^{ij}[k][P0] ~
1/D^(k+1) of blocks whose largest entry is ~1/D: 6e-8 D relative per pair, 5e-6
for distances up to ~70.
"""
import numpy as np
import pytest

from oracle import oracle as O
from rigidfibers_b200.generate import sphere_layout

pytestmark = pytest.mark.gpu


def _sim(pos, ori, **kw):
    from rigidfibers_b200 import Config, Simulation
    return Simulation(Config(**kw), pos, ori)


def _pairs(m, intervals, collinear=True):
    # fiber 0 against fibers on both sides of the limits and far away; radial,
    # collinear (not for the closed form, whose formulas divide by the distance
    # from the other fiber's axis) and random orientations; 19 fibers fill no tile
    rng = np.random.default_rng(100 * m + intervals)
    dist = [3.0, 3.9999, 4.0001, 4.5, 5.0, 6.9999, 7.0001, 8.0, 40.0]
    pos, ori = [np.zeros(3)], [np.array([0.0, 0.0, 1.0])]
    for k, d in enumerate(dist * 2):
        u = np.array([0.0, 0.0, 1.0]) if collinear and k % 9 == 2 else rng.standard_normal(3)
        u /= np.linalg.norm(u)
        t = u if collinear and k < 9 else rng.standard_normal(3)
        pos.append(d * u)
        ori.append(t / np.linalg.norm(t))
    return np.array(pos), np.array(ori)


@pytest.mark.parametrize("integration", ["numerical", "analytical"])
@pytest.mark.parametrize("m,intervals", [(1, 8), (2, 8), (3, 8), (4, 8), (5, 8), (6, 8), (7, 8), (8, 8), (5, 4), (5, 16)])
def test_pairs_on_both_sides_of_the_distance_limit(m, intervals, integration):
    pos, ori = _pairs(m, intervals, integration == "numerical")
    A64, _ = O.assemble(pos, ori, O.Params(M=m, intervals=intervals), integration == "analytical", np.float64)
    sim = _sim(pos, ori, number_of_terms_in_force_expansion=m, number_of_quadrature_intervals=intervals,
               integration=integration)
    sim.assembleSystem()
    A, _ = sim.system()
    r = 3 * m
    for f in range(1, len(pos)):
        here, there = slice(0, r), slice(f * r, f * r + r)
        for blk in ((here, there), (there, here)):
            # a block's largest entry is about 1/D times its coefficients (0.1 .. 1)
            big = max(np.abs(A64[blk]).max(), 0.1 / np.linalg.norm(pos[f]))
            assert np.abs(A[blk] - A64[blk]).max() <= 4e-6 * big, (f, blk)
    sim.close()


@pytest.mark.parametrize("prec", ["fp32", "mixed_fp16", "matrix_free"])
def test_right_hand_side_of_a_dilute_suspension(prec):
    pos, ori = sphere_layout(300, (100.0 * 300) ** (1.0 / 3.0), 0.2, seed=77)
    _, b64 = O.assemble(pos, ori, O.Params(), False, np.float64)
    sim = _sim(pos, ori, precision=prec)
    sim.assembleSystem()
    _, b = sim.system(with_matrix=False)
    assert np.linalg.norm(b - b64) <= 5e-6 * np.linalg.norm(b64)
    sim.close()


@pytest.mark.parametrize("integration", ["numerical", "analytical"])
@pytest.mark.parametrize("m,intervals", [(5, 8), (8, 8), (2, 8), (5, 4), (5, 16)])
def test_velocities_on_both_sides_of_the_distance_limit(m, intervals, integration):
    """The velocity kernels' far and near parts (and their split into chunks and
    segments) for a given force density, against the FP64 oracle on the same
    forces: a sum of ~20 sources of FP32 accuracy, 2e-6 of the largest velocity."""
    pos, ori = _pairs(m, intervals, integration == "numerical")
    p = O.Params(M=m, intervals=intervals)
    sim = _sim(pos, ori, number_of_terms_in_force_expansion=m, number_of_quadrature_intervals=intervals,
               integration=integration)
    sim.assembleSystem()
    sim.solveSystem()
    sim.updateVelocities()
    x = sim.solution()
    want = O.update_velocities(pos, ori, x, p, dtype=np.float64, analytical=integration == "analytical")
    for got, ref in zip(sim.velocities(), want):
        assert np.abs(got - ref).max() <= 2e-6 * np.abs(ref).max()
    sim.close()
