"""Packed solves at the sizes and lengths where the dot products change form:
one partial sum per slice up to 32 fibers, two up to 64; 4, 8 or 16 values at a
time (a restart of 3, 7, 8 or 20 keeps a cycle's widest product on either side
of each).

Bounds (written here): GMRES-IR to a relative residual of 1e-6 on a dilute
system, whose condition number is below 10: 1e-5 of the largest force against
the FP64 oracle's direct solution, plus 1e-6 for the FP32 operator; a member
bit for bit the same alone and among others.
"""
import numpy as np
import pytest

from oracle import oracle as O
from rigidfibers_b200.generate import sphere_layout

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("restart", [3, 7, 8, 20])
def test_packed_solutions_at_the_edges_of_the_dot_products(restart):
    from rigidfibers_b200 import Config, Simulation
    from rigidfibers_b200.simulation import solve_packed
    sizes = [2, 16, 17, 32, 33, 64, 65]
    lays = [sphere_layout(n, (100.0 * n) ** (1.0 / 3.0), 0.2, seed=500 + n) for n in sizes]

    def solved(which):
        sims = [Simulation(Config(precision="mixed_fp16", gmres_restart=restart, refinement_restart=restart), *lays[k])
                for k in which]
        for s in sims:
            s.assembleSystem()
        solve_packed(sims)
        out = [s.solution() for s in sims]
        for s in sims:
            s.close()
        return out

    together = solved(range(len(sizes)))
    for k, (pos, ori) in enumerate(lays):
        A, b = O.assemble(pos, ori, O.Params(), False, np.float64)
        want = np.linalg.solve(A, b)
        assert np.abs(together[k] - want).max() <= 1.1e-5 * np.abs(want).max()
        assert np.array_equal(solved([k])[0], together[k])
