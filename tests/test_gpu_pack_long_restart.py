"""Packed solves at the longest restart: the shared memory of a member is at
its largest there, and the dot products of one CTA's slices no longer fit in
one pass.

Bound (written here): the same bits and the same iteration counts on one CTA
(two for 256 fibers) as on eight; the inner iterations run past the 32 basis
vectors above which a single CTA takes its slices in several passes.
"""
import numpy as np
import pytest

from rigidfibers_b200.generate import sphere_layout

pytestmark = pytest.mark.gpu


def _solve(lays, n_keep):
    from rigidfibers_b200 import Config, Simulation
    from rigidfibers_b200.simulation import solve_packed
    sims = []
    for k, (pos, ori) in enumerate(lays):
        kw = dict(precision="mixed_fp16", gmres_restart=64, refinement_restart=64, gmres_max_iterations=64)
        # a tolerance out of reach: the cycle runs on until its estimate has
        # fallen by 30 digits
        kw["refinement_tolerance"] = 1e-30
        sims.append(Simulation(Config(**kw), pos, ori))
        sims[-1].assembleSystem()
    solve_packed(sims, allow_noconv=True)
    out = [(sims[k].solution(), sims[k].stats()["iterations"]) for k in range(n_keep)]
    for s in sims:
        s.close()
    return out


@pytest.mark.parametrize("n", [97, 128, 256])
def test_long_restart_is_the_same_for_every_cluster_size(n):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    lay = sphere_layout(n, (n / 0.5) ** (1.0 / 3.0) + 1.0, 0.2, seed=700 + n)
    small = [sphere_layout(3, 3.0, 0.2, seed=k) for k in range(max(148, sms))]
    (alone, it1), = _solve([lay], 1)
    (packed, it2), = _solve([lay] + small, 1)
    assert np.isfinite(alone).all()
    assert it1 == it2 and it1 > 32
    assert np.array_equal(alone, packed)
