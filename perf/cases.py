"""Performance cases: whole time steps of fiber suspensions through the public API.

A case is one suspension (or a pack of small ones) and a number of time steps.
A pass sets the fibers' initial state, takes the steps and reads back what a
program saves after them: the force coefficients, the velocities and the new
positions and orientations.  The handle (device memory, stream, captured
graphs) is made once in `prepare`, as a program keeps it over its run.

Layouts: centres uniform in a ball with a minimum centre distance of 0.2,
orientations uniform on the sphere (the layouts of bench.py).  Two densities:
"dense" suspensions have N / radius^3 about 0.7 (100 fibers in radius 5, 2000 in
14, 4000 in 18, 8000 in 23), "dilute" ones 0.01 (the served ensembles).

Results are returned in single precision: the solver's vectors and velocities
are single-precision values on the device, and states are saved in it.
"""
import math

import numpy as np
import torch

from rigidfibers_b200 import Config, Simulation
from rigidfibers_b200.simulation import step_packed

M, INTERVALS, DT = 5, 8, 0.1
MIN_DISTANCE = 0.2


def _case(name, kind, n, density, eps, steps, **kw):
    c = {"name": name, "kind": kind, "n": n, "density": density, "eps": eps, "steps": steps}
    c.update(kw)
    return c


def listed():
    return [
        # the headline run: mixed precision, FP16 blocks
        _case("mixed_fp16_4000", "mixed_fp16", 4000, 0.686, 0.01, 1),
        # the largest single suspension of the benchmark's configurations
        _case("mixed_fp16_8000", "mixed_fp16", 8000, 0.657, 0.01, 1),
        # the largest served request: BF16 blocks, dilute, a few steps between state reads
        _case("mixed_bf16_1000", "mixed_bf16", 1000, 0.01, 0.005, 4),
        # the smallest call: the reference's own 100-fiber configuration, FP32, GMRES(10)
        _case("fp32_100", "fp32", 100, 0.8, 0.01, 1),
        # the plain method at the thesis' scale, dense FP32 matrix
        _case("fp32_2000", "fp32", 2000, 0.729, 0.01, 1),
        # analytical inner integrals (--analytical), a size that fills no tile
        _case("analytical_777", "analytical", 777, 0.729, 0.01, 1),
        # the direct solver (--magma): blocked LU
        _case("direct_1000", "direct", 1000, 0.7, 0.01, 1),
        # --bicgstab on the 16-bit operator
        _case("bicgstab_1501", "bicgstab", 1501, 0.7, 0.01, 1),
        # a serving pack: a few small requests stepping together
        _case("pack_12", "pack", 12, 0.01, 0.01, 10, lo=16, hi=128),
        # no stored operator: the mode for suspensions beyond device memory
        _case("matrix_free_2500", "matrix_free", 2500, 0.7, 0.01, 1),
        # only the 16-bit records stored: the mode between the two
        _case("recompute_3001", "recompute", 3001, 0.7, 0.01, 1),
        # the near-field preconditioner (opt-in) on the headline suspension
        _case("near_field_4000", "near_field", 4000, 0.686, 0.01, 1),
    ]


# kind: smallest and largest size, densities, steps per pass
_RANGES = {
    "mixed_fp16": (130, 7000, "dense"),
    "mixed_bf16": (130, 1000, "dilute"),
    "fp32": (20, 2000, "dense"),
    "analytical": (50, 777, "dense"),
    "direct": (100, 1000, "dense"),
    "bicgstab": (100, 2000, "dense"),
    "pack": (1, 24, "dilute"),
    "matrix_free": (100, 2500, "dense"),
    "recompute": (200, 3001, "dense"),
    "near_field": (200, 4000, "dense"),
}


def draw(rng):
    kind = rng.choice(sorted(_RANGES))
    lo, hi, density = _RANGES[kind]
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    dense = density == "dense"
    c = {"kind": kind, "n": n, "density": round(rng.uniform(0.5, 0.8), 3) if dense else 0.01,
         "eps": 0.01 if dense else rng.choice([0.01, 0.005]), "steps": 1 if dense else rng.randint(2, 6)}
    if kind == "pack":
        c["lo"], c["hi"] = 16, rng.choice([64, 100, 128, 200])
    return c


def _sizes(case):
    """Fiber counts of the case's suspensions (a pack's: spread over [lo, hi] on a log scale)."""
    if case["kind"] != "pack":
        return [case["n"]]
    n, lo, hi = case["n"], case["lo"], case["hi"]
    return [int(round(lo * (hi / lo) ** ((k + 0.5) / n))) for k in range(n)]


def _layouts(case, seed):
    """(positions, orientations) of every suspension of the case."""
    rng = np.random.Generator(np.random.PCG64(seed))
    device = "cuda" if torch.cuda.is_available() else "cpu"
    out = []
    for n in _sizes(case):
        radius = (n / case["density"]) ** (1.0 / 3.0)

        def ball(k):
            v = rng.standard_normal((k, 3))
            return v / np.linalg.norm(v, axis=1, keepdims=True) * radius * rng.random((k, 1)) ** (1.0 / 3.0)

        pos = ball(n)
        while True:   # redraw the later fiber of every pair that is too close
            p = torch.from_numpy(pos).to(device)
            bad = np.zeros(n, bool)
            for i in range(0, n, 2048):
                d2 = ((p[i:i + 2048, None, :] - p[None, :, :]) ** 2).sum(-1)
                earlier = torch.arange(n, device=device)[None, :] < torch.arange(i, min(n, i + 2048), device=device)[:, None]
                bad[i:i + 2048] = ((d2 < MIN_DISTANCE ** 2) & earlier).any(1).cpu().numpy()
            if not bad.any():
                break
            pos[bad] = ball(int(bad.sum()))
        ori = rng.standard_normal((n, 3))
        out.append((pos, ori / np.linalg.norm(ori, axis=1, keepdims=True)))
    return out


def _config(case):
    kind = case["kind"]
    kw = {"slenderness": case["eps"], "timestep": DT}
    if kind in ("mixed_fp16", "mixed_bf16"):
        kw["precision"] = kind
    elif kind == "matrix_free":
        # every iteration recomputes the operator: a longer restart than the plain method's 10
        kw.update(precision="matrix_free", gmres_restart=20, gmres_tolerance=1e-6)
    elif kind == "near_field":
        kw["precision"] = "mixed_fp16"
    elif kind == "bicgstab":
        kw.update(precision="mixed_fp16", solver="bicgstab")
    elif kind == "pack":
        kw["precision"] = "mixed_bf16"
    elif kind == "recompute":
        kw.update(precision="mixed_fp16_recompute", refinement_restart=40)
    elif kind == "analytical":
        kw["integration"] = "analytical"
    elif kind == "direct":
        kw["solver"] = "direct"
    return Config(**kw)


def prepare(case, seed):
    layouts = _layouts(case, seed)
    sims = [Simulation(_config(case), pos, ori) for pos, ori in layouts]
    if case["kind"] == "near_field":
        sims[0].set_near_field_preconditioner(4)
    return {"sims": sims, "layouts": layouts, "steps": case["steps"], "pack": case["kind"] == "pack"}


def _results(sim):
    pos, ori = sim.state()
    tvel, rvel = sim.velocities()
    return {"x": sim.solution().astype(np.float32), "tvel": tvel.astype(np.float32), "rvel": rvel.astype(np.float32),
            "pos": pos.astype(np.float32), "ori": ori.astype(np.float32)}


def run(state):
    sims = state["sims"]
    for sim, (pos, ori) in zip(sims, state["layouts"]):
        sim.set_state(pos, ori)
    for t in range(state["steps"]):
        if state["pack"]:
            codes = step_packed(sims, [t] * len(sims))
            if any(codes):
                raise RuntimeError("step_packed: %r" % codes)
        else:
            sims[0].step(t)
    res = [_results(sim) for sim in sims]
    if not state["pack"]:
        return res[0]
    # one array per field over the pack's members
    return {k: np.concatenate([r[k].reshape(-1) for r in res]) for k in res[0]}


def work(case):
    """Per step: the state in and out, the stored operator written and read once, and one
    product with the system (the direct solver: its factorization)."""
    by, fl = 0.0, 0.0
    for n in _sizes(case):
        rows, pairs = 3 * M * n, n * (n - 1) / 2
        stored = {"fp32": 4.0 * rows * rows, "analytical": 4.0 * rows * rows, "direct": 4.0 * rows * rows,
                  "matrix_free": 0.0, "recompute": 300.0 * pairs}.get(case["kind"], (300.0 + 864.0) * pairs)
        by += case["steps"] * (2.0 * stored + 2.0 * 4 * rows + n * 2 * (2 * 48 + 2 * 24))
        fl += case["steps"] * (2.0 * rows * rows + (2.0 / 3.0 * rows ** 3 if case["kind"] == "direct" else 0.0))
    return {"bytes": by, "flops": fl}


# ---- the same steps in 64 bits -----------------------------------------------
def _legendre(s, k):
    return np.polynomial.legendre.Legendre.basis(k)(s)


def _rule():
    """Composite three-point Gauss rule on [-1, 1]; weights of the Legendre moments P_0..P_M."""
    h = 2.0 / INTERVALS
    p = np.array([-math.sqrt(0.6), 0.0, math.sqrt(0.6)]) * h / 2
    pts = np.concatenate([-1 + h * (k + 0.5) + p for k in range(INTERVALS)])
    w = np.tile(np.array([5.0, 8.0, 5.0]) / 9.0 * h / 2, INTERVALS)
    return pts, np.stack([w * _legendre(pts, k) for k in range(M + 1)])


_COMP = [(0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)]


class _Fp64:
    """One suspension's system in 64 bits, formed in chunks of fibers."""

    def __init__(self, n, eps, analytical):
        self.n, self.eps, self.analytical = n, eps, analytical
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        pts, wk = _rule()
        self.pts = torch.tensor(pts, device=self.dev)
        self.wk = torch.tensor(wk, device=self.dev)
        d = -math.log(eps * eps * math.e)
        self.d = d
        lam = [2.0]
        for k in range(1, M):
            lam.append(lam[-1] + 2.0 / (k + 1))
        eig = [((d - 2.0 - v) / 2.0) / (d - v) for v in lam]
        gam = [0.75 / (d - 2.0)] + [0.5 * (2.0 * (k + 1) + 1.0) / (d + 2.0 - lam[k]) for k in range(1, M)]
        self.eig = torch.tensor([1.0] + eig[1:], device=self.dev, dtype=torch.float64)
        self.gam = torch.tensor(gam, device=self.dev, dtype=torch.float64)
        # sinh-substituted rule for the closed inner integral
        u, w = np.polynomial.legendre.leggauss(160)
        self.u, self.uw = torch.tensor(u, device=self.dev), torch.tensor(w, device=self.dev)

    def chunk(self):
        per = 160 if self.analytical else 24
        return max(1, int(1.5e8 / (self.n * 24 * per)))

    def blocks(self, pos, ori, i0, i1):
        """T[i, j, k, l, 3, 3] of fibers i0..i1 against all, zero for i = j (k on i, l on j)."""
        n, e2 = self.n, 2.0 * self.eps ** 2
        rel = pos[i0:i1, None, :] - pos[None, :, :]
        p = rel[:, :, None, :] + self.pts[None, None, :, None] * ori[i0:i1, None, None, :]   # points of i, from j's centre
        idx = torch.arange(i0, i1, device=self.dev)
        p[idx - i0, idx] = 3.0   # any regular value: zeroed below
        t = ori[None, :, None, :]
        if not self.analytical:
            sep = [p[..., a, None] - self.pts * t[..., a, None] for a in range(3)]
            inv = (sep[0] ** 2 + sep[1] ** 2 + sep[2] ** 2).rsqrt()
            kern = None
        else:
            # s - s* = h sinh(u): |r| = h cosh(u) on the interval that maps to [-1, 1]
            ss = (p * t).sum(-1)
            perp = p - ss[..., None] * t
            h = (perp ** 2).sum(-1).sqrt().clamp_min(1e-9)
            ua, ub = torch.asinh((-1.0 - ss) / h), torch.asinh((1.0 - ss) / h)
            u = 0.5 * (ua + ub)[..., None] + 0.5 * (ub - ua)[..., None] * self.u
            du = 0.5 * (ub - ua)[..., None] * self.uw * h[..., None] * torch.cosh(u)
            s = ss[..., None] + h[..., None] * torch.sinh(u)
            sep = [p[..., a, None] - s * t[..., a, None] for a in range(3)]
            inv = (sep[0] ** 2 + sep[1] ** 2 + sep[2] ** 2).rsqrt()
            leg = [torch.ones_like(s), s]
            for k in range(1, M):
                leg.append(((2 * k + 1) * s * leg[k] - k * leg[k - 1]) / (k + 1))
            kern = torch.stack([v * du for v in leg], -2)   # [i,j,q,k,u]
        inv3 = inv ** 3
        a = inv + e2 * inv3
        b = inv3 - 3.0 * e2 * inv3 * inv * inv
        out = torch.empty(i1 - i0, n, M + 1, M + 1, 3, 3, device=self.dev, dtype=torch.float64)
        for c, (x, y) in enumerate(_COMP):
            val = b * sep[x] * sep[y]
            if x == y:
                val = val + a
            if kern is None:
                g = val @ self.wk.T                                   # [i,j,q,l]
            else:
                g = (kern @ val[..., None])[..., 0]
            tb = torch.einsum("kq,ijql->ijkl", self.wk, g)
            out[..., x, y] = tb
            out[..., y, x] = tb
        out[idx - i0, idx] = 0.0
        return out

    def project(self, z, ori):
        """C z: z[..., k, 3] of the force indices of fibers with orientation ori[..., 3]."""
        t = ori[..., None, :]
        tz = (t * z).sum(-1, keepdim=True)
        full = z - self.eig[:, None] * t * tz
        full[..., 0, :] = (t * tz)[..., 0, :]
        return self.gam[:, None] * full

    def solve_step(self, pos, ori):
        """(x, tvel, rvel) of one state."""
        n, rows = self.n, 3 * M * self.n
        A = torch.empty(rows, rows, device=self.dev, dtype=torch.float64)
        b = torch.empty(n, M, 3, device=self.dev, dtype=torch.float64)
        step = self.chunk()
        for i0 in range(0, n, step):
            i1 = min(n, i0 + step)
            T = self.blocks(pos, ori, i0, i1)
            b[i0:i1] = -self.project(T[:, :, 1:, 0, :, 2].sum(1) * -0.5, ori[i0:i1])
            t = ori[i0:i1]
            # C applied on the row side of every block: [i, j, k, l, d, e]
            S = T[:, :, 1:, 1:]
            tS = torch.einsum("id,ijklde->ijkle", t, S)
            ttS = t[:, None, None, None, :, None] * tS[..., None, :]
            blk = S - self.eig[None, None, :, None, None, None] * ttS
            blk[:, :, 0] = ttS[:, :, 0]
            blk = blk * self.gam[None, None, :, None, None, None]
            A[i0 * 3 * M:i1 * 3 * M] = blk.permute(0, 2, 4, 1, 3, 5).reshape((i1 - i0) * 3 * M, rows)
            del T, S, tS, ttS, blk
        A.diagonal().add_(1.0)
        x = self.gmres(A, b.reshape(-1))
        del A
        xf = x.reshape(n, M, 3)
        F = torch.tensor([0.0, 0.0, -1.0], device=self.dev, dtype=torch.float64)
        dens = torch.cat([(0.5 * F).expand(n, 1, 3), xf], 1)   # Legendre coefficients of the force density
        tv, rv = torch.empty_like(pos), torch.empty_like(pos)
        for i0 in range(0, n, step):
            i1 = min(n, i0 + step)
            T = self.blocks(pos, ori, i0, i1)
            s = torch.einsum("ijklde,jle->ikd", T[:, :, :2], dens)
            t = ori[i0:i1]
            tF = (t * F).sum(-1, keepdim=True)
            tv[i0:i1] = 0.5 / self.d * ((self.d + 2) * F + (self.d - 2) * tF * t + s[:, 0])
            rv[i0:i1] = 1.5 / self.d * (s[:, 1] - t * (t * s[:, 1]).sum(-1, keepdim=True))
            del T
        return x, tv, rv

    def gmres(self, A, b, tol=1e-12, most=240):
        norm = b.norm()
        V = torch.zeros(most + 1, b.numel(), device=self.dev, dtype=torch.float64)
        H = np.zeros((most + 1, most))
        V[0] = b / norm
        for j in range(most):
            w = A @ V[j]
            h = V[:j + 1] @ w
            w = w - V[:j + 1].T @ h
            g = V[:j + 1] @ w
            w = w - V[:j + 1].T @ g
            H[:j + 1, j] = (h + g).cpu().numpy()
            H[j + 1, j] = float(w.norm())
            rhs = np.zeros(j + 2)
            rhs[0] = 1.0
            y, *_ = np.linalg.lstsq(H[:j + 2, :j + 1], rhs, rcond=None)
            if np.linalg.norm(H[:j + 2, :j + 1] @ y - rhs) < tol or H[j + 1, j] == 0.0:
                break
            V[j + 1] = w / H[j + 1, j]
        return V[:j + 1].T @ torch.tensor(y, device=self.dev) * norm


def exact(case, seed):
    res = []
    for pos, ori in _layouts(case, seed):
        sys64 = _Fp64(pos.shape[0], case["eps"], case["kind"] == "analytical")
        x1 = torch.from_numpy(pos).to(sys64.dev)
        t1 = torch.from_numpy(ori).to(sys64.dev)
        x0, t0, u0, w0 = x1, t1, None, None
        for step in range(case["steps"]):
            x, u, w = sys64.solve_step(x1, t1)
            if step == 0:
                xn, tn = x1 + DT * u, t1 + DT * w
            else:
                xn = (4 * x1 - x0 + 2 * DT * (2 * u - u0)) / 3
                tn = (4 * t1 - t0 + 2 * DT * (2 * w - w0)) / 3
            tn = tn / tn.norm(dim=1, keepdim=True)
            x0, x1, t0, t1, u0, w0 = x1, xn, t1, tn, u, w
        res.append({k: v.cpu().numpy() for k, v in (("x", x), ("tvel", u), ("rvel", w), ("pos", x1), ("ori", t1))})
    if case["kind"] != "pack":
        return res[0]
    return {k: np.concatenate([r[k].reshape(-1) for r in res]) for k in res[0]}
