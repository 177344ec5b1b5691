"""Roundings of the right-hand side of dilute suspensions: with the far pairs' rule
no more than with the full rule.

Bound (written here): a block of P_k against P_0 of two fibers D apart carries,
rule by rule, roundings n_k / D rms; an FP32 emulation of the full rule (24 points
a fiber, every operation rounded, random pairs 4 to 40 apart) gives n_k = 3.9, 5.6,
2.3, 2.9 and 1.8 e-8 for k = 1 .. 5.  Half of the pairs enter a fiber's sum by the
transposed block, P_0 against P_k, with 1.5, 1.2, 0.6, 0.7 and 0.4 e-8.  Times
|F/2| = 1/2 and gamma_k, summed in squares over the other fibers, that is b's
expected error; the measured one, rms over all rows of several layouts (4800 of
them: the rms of that many is within 5 % of its expectation), is at most that.
"""
import numpy as np
import pytest

from oracle import oracle as O
from rigidfibers_b200.generate import sphere_layout

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp32", "mixed_fp16", "mixed_bf16"])
def test_right_hand_side_rounds_no_worse_than_with_the_full_rule(prec):
    from rigidfibers_b200 import Config, Simulation
    d = -np.log(0.01 * 0.01 * np.e)
    lam = [2.0]
    for k in range(1, 5):
        lam.append(lam[-1] + 2.0 / (k + 1))
    gamma = np.array([0.75 / (d - 2.0)] + [0.5 * (2.0 * (k + 1) + 1.0) / (d + 2.0 - lam[k]) for k in range(1, 5)])
    col, row = np.array([3.9, 5.6, 2.3, 2.9, 1.8]) * 1e-8, np.array([1.5, 1.2, 0.6, 0.7, 0.4]) * 1e-8
    per_pair = 0.5 * gamma * np.sqrt(0.5 * (col ** 2 + row ** 2))
    got, want = 0.0, 0.0
    for seed in range(4):
        n = 80
        pos, ori = sphere_layout(n, (100.0 * n) ** (1.0 / 3.0), 4.0, seed=900 + seed)
        pos, ori = pos.astype(np.float32).astype(float), ori.astype(np.float32).astype(float)
        _, b64 = O.assemble(pos, ori, O.Params(), False, np.float64)
        with Simulation(Config(precision=prec), pos, ori) as sim:
            sim.assembleSystem()
            _, b = sim.system(with_matrix=False)
        dist = np.linalg.norm(pos[:, None] - pos[None], axis=2)
        np.fill_diagonal(dist, np.inf)
        got += ((b - b64) ** 2).sum()
        want += 3 * ((dist ** -2.0).sum(1)[:, None] * per_pair[None, :] ** 2).sum()
    print(prec, np.sqrt(got / want))
    assert got <= want
