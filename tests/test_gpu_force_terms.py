"""Right-hand sides and whole steps for every number of force terms.

b of fiber i, force index k is -C_k sum_j T^{ij}[k + 1][P_0] F/2, one partial sum
per batch of pairs and thread: 37 fibers are more than two tiles of 16 (every
row of a batch and every Legendre index has its own partial sum), 19 fill none.

Bounds (written here): a kernel value is at most 2/r, so the 4 points' worth of
weight of two fibers D apart make block entries up to 8/D, times |F/2| = 1/2; an
entry carries about 30 roundings of 6e-8 relative to the block's largest one,
hence |b - b64| <= gamma_k 2e-6 sum_j 4/D_ij for every index k (gamma_k: D1 and
the gamma of the system, at most 2).  Steps are solved to 1e-6 of the
right-hand side, and the system's condition number is below 50 for a dilute
suspension: 5e-5 of the largest force; velocities add the forces' sums to the
fibers' own, 1e-5 of the largest.
"""
import numpy as np
import pytest

from oracle import oracle as O
from rigidfibers_b200.generate import sphere_layout

pytestmark = pytest.mark.gpu

MQ = [(1, 8), (2, 8), (3, 8), (4, 8), (5, 8), (6, 8), (7, 8), (8, 8), (5, 4), (5, 16)]
MODES = {"fp32": {}, "mixed_fp16": dict(precision="mixed_fp16"), "mixed_bf16": dict(precision="mixed_bf16"),
         "recompute": dict(precision="mixed_fp16_recompute"), "matrix_free": dict(precision="matrix_free"),
         "analytical": dict(integration="analytical")}


def _sim(pos, ori, m, intervals, **kw):
    from rigidfibers_b200 import Config, Simulation
    return Simulation(Config(number_of_terms_in_force_expansion=m, number_of_quadrature_intervals=intervals, **kw),
                      pos, ori)


def _gammas(m, eps=0.01):
    d = -np.log(eps * eps * np.e)
    lam = [2.0]
    for k in range(1, m):
        lam.append(lam[-1] + 2.0 / (k + 1))
    return np.array([0.75 / (d - 2.0)] + [0.5 * (2.0 * (k + 1) + 1.0) / abs(d + 2.0 - lam[k]) for k in range(1, m)])


# the mixed modes are built for 8 intervals
CASES = [(m, iv, mode) for m, iv in MQ for mode in sorted(MODES)
         if iv == 8 or not (mode.startswith("mixed") or mode == "recompute")]


@pytest.mark.parametrize("m,intervals,mode", CASES)
def test_right_hand_side_per_force_index(m, intervals, mode):
    for n in (19, 37):
        pos, ori = sphere_layout(n, (n / 0.1) ** (1.0 / 3.0), 0.5, seed=300 + n)
        _, b64 = O.assemble(pos, ori, O.Params(M=m, intervals=intervals), mode == "analytical", np.float64)
        sim = _sim(pos, ori, m, intervals, **MODES[mode])
        sim.assembleSystem()
        _, b = sim.system(with_matrix=False)
        sim.close()
        dist = np.linalg.norm(pos[:, None] - pos[None], axis=2)
        np.fill_diagonal(dist, np.inf)
        bound = 2e-6 * (4.0 / dist).sum(1)[:, None] * _gammas(m)[None, :]
        err = np.abs(b - b64).reshape(n, m, 3).max(2)
        assert (err <= bound).all(), (n, np.argwhere(err > bound)[:4].tolist(), (err / bound).max())


@pytest.mark.parametrize("mode", ["fp32", "direct", "bicgstab", "mixed_fp16", "recompute", "matrix_free"])
@pytest.mark.parametrize("m", [7, 8])
def test_whole_step_with_many_force_terms(m, mode):
    n = 37
    pos, ori = sphere_layout(n, (n / 0.1) ** (1.0 / 3.0), 0.5, seed=400 + m)
    kw = dict(MODES[mode] if mode in MODES else dict(solver=mode))
    kw.update(gmres_tolerance=1e-6, bicgstab_tolerance=1e-6)
    sim = _sim(pos, ori, m, 8, **kw)
    sim.step(0)
    ref = O.run_steps(pos, ori, O.Params(M=m), 1, solver="direct", dtype=np.float64)[0]
    x, (tv, rv) = sim.solution(), sim.velocities()
    sim.close()
    assert np.abs(x - ref["x"].reshape(-1)).max() <= 5e-5 * np.abs(ref["x"]).max()
    for got, want in ((tv, ref["tvel"]), (rv, ref["rvel"])):
        want = want.reshape(got.shape)
        assert np.abs(got - want).max() <= 1e-5 * max(np.abs(want).max(), 1e-3)
