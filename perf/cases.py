"""The work that users of this library have it do, as cases that can be timed and compared.

A case is a dict of plain values.  Its `kind`:

  box        one time step of the plain method (lid-driven box, uniform or stretched grid)
  cylinder   one time step of a cylinder with an immersed-boundary method, fixed body
  moving     one time step of the embedded method with an oscillating cylinder (the body
             moves, is tagged again and changes both operators every step)
  batch      one step of many independent cases of uneven sizes advanced together
  adjoint    the gradient of the averaged drag over a short run (forward and reverse sweep)
  poisson    one pressure solve alone, as a coupling code calls it
  explicit   the explicit kernels alone: right-hand sides, projection, CFL

Linear solves run to 1e-12 or 1e-13, as the parity runs of this repository do, so that the
outputs are fixed by the discrete equations and not by where an iteration stopped: at the
looser tolerances of production runs (1e-5 to 1e-8) two correct solvers differ by the
tolerance itself (and the pressure's level, fixed by one pinned cell, by a hundred times it).  A step starts from a given state (device copies of u, N, p and the
velocity solve's starting vector are written into the solver first), as a restarted run,
an ensemble member or a coupled solver does it, so that every pass does the same work."""
import math
import os
import tempfile

import numpy as np
import torch

import cuibm_gb300 as cb
from cuibm_gb300 import cases as yaml_cases

D = 8  # bytes of a value: every field is FP64


# ---------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------
def listed():
    return [
        # the reference's own lid-driven cavity set-up, the smallest run: launches and latency
        {"name": "cavity_64", "kind": "box", "h": 1.0 / 64, "ratio": 1.0, "ax": 0.5, "ay": 0.5, "core": 0.5,
         "nu": 0.01, "dt": 0.01, "krylov": "CG", "precision": "FP64", "tol": 1e-13},
        # a stretched box with odd, unequal sides (103 x 63)
        {"name": "box_odd", "kind": "box", "h": 0.05, "ratio": 1.04, "ax": 5.0, "ay": 2.0, "core": 0.7, "nu": 0.02,
         "dt": 0.01, "krylov": "BICGSTAB", "precision": "FP64", "tol": 1e-12},
        # the largest cavity of the batched workload, alone, in mixed precision
        {"name": "cavity_512_mixed", "kind": "box", "h": 1.0 / 512, "ratio": 1.0, "ax": 0.5, "ay": 0.5, "core": 0.5,
         "nu": 0.002, "dt": 0.000625, "krylov": "BICGSTAB", "precision": "MIXED", "tol": 1e-12},
        # the benchmark's default workload: impulsively started cylinder, Re 40, external method (270 x 270)
        {"name": "cylinder_re40", "kind": "cylinder", "method": "LUO", "h": 0.02, "ratio": 1.03, "extent": 15.0,
         "points": 157, "nu": 0.025, "dt": 0.01, "precision": "FP64", "tol": 1e-13},
        # the same flow with the modified Fadlun method on a coarser, odd grid
        {"name": "fadlun_re40", "kind": "cylinder", "method": "FADLUN", "h": 0.03, "ratio": 1.05, "extent": 12.0,
         "points": 105, "nu": 0.025, "dt": 0.01, "precision": "FP64", "tol": 1e-12},
        # the large benchmark: cylinder at Re 550 (922 x 922)
        {"name": "cylinder_re550", "kind": "cylinder", "method": "LUO", "h": 0.005, "ratio": 1.01, "extent": 15.0,
         "points": 629, "nu": 1.0 / 550, "dt": 0.002, "precision": "FP64", "tol": 1e-13},
        # a cylinder at Re 100 in mixed precision (FP32 preconditioner, FP64 iteration; 270 x 270)
        {"name": "cylinder_mixed", "kind": "cylinder", "method": "LUO", "h": 0.02, "ratio": 1.03, "extent": 15.0,
         "points": 158, "nu": 0.01, "dt": 0.008, "precision": "MIXED", "tol": 1e-12},
        # the oscillating cylinder of the adjoint benchmark, forward (KC 10, 686 x 686)
        {"name": "oscillating_kc10", "kind": "moving", "h": 0.01, "ratio": 1.02, "extent": 10.0, "core": 2.0,
         "points": 314, "um": 1.0, "period": 10.0, "nu": 0.005, "dt": 0.0025, "tol": 1e-12},
        # sensitivities: forward and reverse sweep of the reduced oscillating cylinder
        {"name": "adjoint_reduced", "kind": "adjoint", "h": 0.05, "ratio": 1.1, "extent": 3.0, "core": 0.6,
         "points": 48, "um": 0.5, "period": 1.0, "nu": 0.02, "dt": 0.01, "steps": 6, "snapshots": 4, "tol": 1e-12},
        # an ensemble: uneven cavities and cylinders advanced together
        {"name": "batch_12", "kind": "batch", "count": 12, "sizes": 1, "tol": 1e-12},
        # a pressure solve alone on a long box (662 x 326)
        {"name": "poisson_long", "kind": "poisson", "h": 0.01, "ratio": 1.01, "ax": 12.0, "ay": 2.1, "core": 0.8,
         "nu": 0.005, "dt": 0.002, "krylov": "BICGSTAB", "precision": "FP64", "tol": 1e-12},
        # the explicit kernels at the large benchmark's size
        {"name": "explicit_re550", "kind": "explicit", "h": 0.005, "ratio": 1.01, "ax": 15.0, "ay": 15.0,
         "core": 0.6, "nu": 1.0 / 550, "dt": 0.002, "krylov": "BICGSTAB", "precision": "FP64", "tol": 1e-12},
    ]


def _log(rng, a, b):
    return math.exp(rng.uniform(math.log(a), math.log(b)))


def _box_draw(rng, n_lo, n_hi):
    """A box of about n cells along x and an aspect ratio between 1:3 and 3:1."""
    n = _log(rng, n_lo, n_hi)
    m = min(n_hi, max(20.0, n * _log(rng, 1 / 3, 3)))
    h = 1.0 / n
    if rng.random() < 0.5:
        return {"h": h, "ratio": 1.0, "ax": 0.5, "ay": 0.5 * m / n, "core": 0.5 * min(1.0, m / n)}
    ratio = 1 + min(0.06, 3.0 / min(n, m))
    reach = lambda k: h * (ratio ** (0.35 * k) - 1) / (ratio - 1) + 0.15 * k * h  # noqa: E731
    return {"h": h, "ratio": ratio, "ax": reach(n), "ay": reach(m), "core": 0.15 * min(n, m) * h}


def draw(rng):
    kind = rng.choice(["box", "box", "cylinder", "cylinder", "poisson", "explicit", "moving", "batch", "adjoint"])
    precision = rng.choice(["FP64", "FP64", "MIXED"])
    if kind in ("box", "poisson", "explicit"):
        c = {"kind": kind}
        c.update(_box_draw(rng, 24, 900))
        c.update({"nu": _log(rng, 1e-3, 2e-2), "dt": 0.3 * c["h"], "krylov": rng.choice(["BICGSTAB", "CG"]),
                  "precision": precision if kind != "explicit" else "FP64", "tol": 1e-12})
        return c
    if kind == "cylinder":
        h = _log(rng, 0.005 if precision == "FP64" else 0.02, 0.05)
        pts = int(round(math.pi / h / 2)) * 2 + rng.choice([0, 1])
        return {"kind": kind, "method": rng.choice(["LUO", "LUO", "FADLUN"]), "h": h, "ratio": 1 + max(0.01, 1.4 * h),
                "extent": rng.uniform(10, 15), "points": pts, "nu": 1 / _log(rng, 40, 550), "dt": 0.4 * h,
                "precision": precision, "tol": 1e-13 if precision == "FP64" else 1e-12}
    if kind == "moving":
        h = _log(rng, 0.012, 0.05)
        return {"kind": kind, "h": h, "ratio": 1.03, "extent": rng.uniform(5, 8), "core": 1.5,
                "points": int(round(math.pi / h)), "um": 1.0, "period": rng.uniform(3, 6), "nu": _log(rng, 0.005, 0.02),
                "dt": 0.25 * h, "tol": 1e-12}
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(3, 12), "sizes": rng.randint(2, 1 << 20), "tol": 1e-12}
    return {"kind": "adjoint", "h": rng.uniform(0.045, 0.06), "ratio": 1.1, "extent": rng.uniform(2.6, 3.4), "core": 0.6,
            "points": rng.randint(40, 60), "um": 0.5, "period": rng.uniform(0.8, 1.2), "nu": _log(rng, 0.01, 0.03),
            "dt": 0.01, "steps": rng.randint(3, 6), "snapshots": rng.randint(2, 4), "tol": 1e-12}


# ---------------------------------------------------------------------------------
# grids (the cell counts and widths that a domain.yaml entry means)
# ---------------------------------------------------------------------------------
def _axis_subs(a, core, ratio):
    return [(a, 1.0)] if ratio == 1.0 else [(-core, ratio), (core, 1.0), (a, ratio)]


def _widths(a, core, h, ratio):
    out, a0 = [], -a
    for a1, r in _axis_subs(a, core, ratio):
        if r == 1.0:
            m = int((a1 - a0) / h)
            out += [(a1 - a0) / m] * m
        else:
            m = int(math.log(1 / (h / ((a1 - a0) * (r - 1))) + 1) / math.log(r))
            h0 = (a1 - a0) * (r - 1) / (r ** m - 1)
            w = [h0 * r ** k for k in range(m)]
            out += w[::-1] if a1 < 0 else w
        a0 = a1
    return np.array(out)


def _count(a, core, h, ratio):
    return len(_widths(a, core, h, ratio))


def _sizes(case):
    """(nx, ny) of a case's grid."""
    k = case["kind"]
    if k in ("box", "poisson", "explicit"):
        return (_count(case["ax"], case["core"], case["h"], case["ratio"]),
                _count(case["ay"], case["core"], case["h"], case["ratio"]))
    n = _count(case["extent"], case.get("core", 0.6), case["h"], case["ratio"])
    return n, n


# ---------------------------------------------------------------------------------
# seeded inputs
# ---------------------------------------------------------------------------------
def _smooth(rng, x, y, modes=6):
    """A smooth random field on the points x (columns) and y (rows), of order 1."""
    sx = (x - x.min()) / max(x.max() - x.min(), 1e-30)
    sy = (y - y.min()) / max(y.max() - y.min(), 1e-30)
    f = np.zeros((len(y), len(x)))
    for _ in range(modes):
        kx, ky = rng.integers(1, 5, 2)
        f += rng.standard_normal() / modes ** 0.5 * np.outer(np.sin(math.pi * ky * sy + rng.uniform(0, 6)),
                                                             np.sin(math.pi * kx * sx + rng.uniform(0, 6)))
    return f


class _Box:
    """The plain method on a box in numpy: grids, seeded fields, and one step in 64 bits."""

    def __init__(self, case, seed):
        self.dx = _widths(case["ax"], case["core"], case["h"], case["ratio"])
        self.dy = _widths(case["ay"], case["core"], case["h"], case["ratio"])
        self.nx, self.ny = len(self.dx), len(self.dy)
        self.nu, self.dt = case["nu"], case["dt"]
        self.rng = np.random.default_rng(seed)
        self.lid = 1.0
        xe, ye = np.cumsum(self.dx) - case["ax"], np.cumsum(self.dy) - case["ay"]
        xc, yc = xe - self.dx / 2, ye - self.dy / 2
        self.xf, self.yf, self.xc, self.yc = xe[:-1], ye[:-1], xc, yc
        # the flow that a lid drives: a shear towards the lid and smooth eddies
        s = (yc - yc.min()) / (yc.max() - yc.min())
        self.U = self.lid * s[:, None] ** 4 + 0.2 * _smooth(self.rng, self.xf, yc)
        self.V = 0.2 * _smooth(self.rng, xc, self.yf)
        # the convection term and pressure of a step before: of a slightly different flow
        self.NU, self.NV = self.convection(0.97 * self.U, 0.97 * self.V)
        self.P = 0.05 * _smooth(self.rng, xc, yc)

    def fields(self):
        cat = lambda a, b: np.concatenate([a.ravel(), b.ravel()])  # noqa: E731
        return {"u": cat(self.U, self.V), "N": cat(self.NU, self.NV), "p": self.P.ravel(),
                "uhat": cat(self.U, self.V)}

    # boundary values: still walls, the lid at y+ moves with u = lid
    def _pad_u(self, U, top, bottom):
        """U with its x walls (0) and one row below and above, as given."""
        W = np.zeros((self.ny + 2, self.nx + 1))
        W[1:-1, 1:-1], W[0, 1:-1], W[-1, 1:-1] = U, bottom, top
        return W

    def _pad_v(self, V, left, right):
        W = np.zeros((self.ny + 1, self.nx + 2))
        W[1:-1, 1:-1], W[1:-1, 0], W[1:-1, -1] = V, left, right
        return W

    def convection(self, U, V):
        dx, dy = self.dx, self.dy
        a, b = dx[:-1][None, :], dx[1:][None, :]
        c = dy[:, None]
        n, s = np.append(dy[1:], dy[-1])[:, None], np.insert(dy[:-1], 0, dy[0])[:, None]
        xE, xW = a / (b * (a + b)), 1 / (a + b) - 1 / a
        yN, yS = 1 / (n + c), s / (c * (c + s)) - 1 / c
        W = self._pad_u(U, 2 * self.lid - U[-1], -U[0])
        Vw = np.zeros((self.ny + 1, self.nx))
        Vw[1:-1] = V
        hA = 0.5 * a / (a + b)
        vb = hA * (Vw[1:, 1:] + Vw[:-1, 1:]) + (0.5 - hA) * (Vw[1:, :-1] + Vw[:-1, :-1])
        NU = U * (W[1:-1, 2:] * xE + W[1:-1, :-2] * xW - U * (xE + xW)) + \
            vb * (W[2:, 1:-1] * yN + W[:-2, 1:-1] * yS - U * (yN + yS))
        a = dx[None, :]
        e, w = np.append(dx[1:], dx[-1])[None, :], np.insert(dx[:-1], 0, dx[0])[None, :]
        c, d = dy[:-1][:, None], dy[1:][:, None]
        xE, xW = 1 / (a + e), w / (a * (a + w)) - 1 / a
        yN, yS = c / (d * (d + c)), 1 / (d + c) - 1 / c
        Z = self._pad_v(V, -V[:, 0], -V[:, -1])
        Uw = np.zeros((self.ny, self.nx + 1))
        Uw[:, 1:-1] = U
        hA = 0.5 * c / (c + d)
        ub = hA * (Uw[1:, 1:] + Uw[1:, :-1]) + (0.5 - hA) * (Uw[:-1, 1:] + Uw[:-1, :-1])
        NV = ub * (Z[1:-1, 2:] * xE + Z[1:-1, :-2] * xW - V * (xE + xW)) + \
            V * (Z[2:, 1:-1] * yN + Z[:-2, 1:-1] * yS - V * (yN + yS))
        return NU, NV

    def _second(self, d, wall):
        """The 1-D second difference: coefficients to the next and previous node.  wall: nodes
        at the cell centres with walls half a cell away, else on the faces between the cells."""
        if wall:
            n = 2 / (d * (np.append(d[1:], d[-1]) + d))
            p = 2 / (d * (np.insert(d[:-1], 0, d[0]) + d))
            return n, p
        return 2 / (d[1:] * (d[1:] + d[:-1])), 2 / (d[:-1] * (d[1:] + d[:-1]))

    def rhs1(self, U, V, NU0, NV0):
        """(NU, NV), (LU, LV), (B1U, B1V), (RU, RV)."""
        hd = 0.5 * self.dt * self.nu
        NU, NV = self.convection(U, V)
        xE, xW = (t[None, :] for t in self._second(self.dx, False))
        yN, yS = (t[:, None].copy() for t in self._second(self.dy, True))
        yNl, ySl = yN.copy(), yS.copy()
        yNl[-1] *= 2
        ySl[0] *= 2  # the wall is half a cell away
        W = self._pad_u(U, self.lid, 0.0)
        LU = (W[1:-1, 2:] - U) * xE + (W[1:-1, :-2] - U) * xW + (W[2:, 1:-1] - U) * yNl + (W[:-2, 1:-1] - U) * ySl
        BU = np.zeros_like(U)
        BU[-1] += (2 * self.lid - U[-1]) * hd * yN[-1]
        BU[0] += -U[0] * hd * yS[0]
        xE, xW = (t[None, :].copy() for t in self._second(self.dx, True))
        yN, yS = (t[:, None] for t in self._second(self.dy, False))
        xEl, xWl = xE.copy(), xW.copy()
        xEl[0, -1] *= 2
        xWl[0, 0] *= 2
        Z = self._pad_v(V, 0.0, 0.0)
        LV = (Z[1:-1, 2:] - V) * xEl + (Z[1:-1, :-2] - V) * xWl + (Z[2:, 1:-1] - V) * yN + (Z[:-2, 1:-1] - V) * yS
        BV = np.zeros_like(V)
        BV[:, -1] += -V[:, -1] * hd * xE[0, -1]
        BV[:, 0] += -V[:, 0] * hd * xW[0, 0]
        dt = self.dt
        RU = U + 0.5 * dt * NU0 - 1.5 * dt * NU + hd * LU + BU
        RV = V + 0.5 * dt * NV0 - 1.5 * dt * NV + hd * LV + BV
        return (NU, NV), (self.nu * LU, self.nu * LV), (BU, BV), (RU, RV)

    @staticmethod
    def _modes(up, down, w):
        """Eigenpairs of the 1-D operator tridiag(-down, up + down, -up), symmetric in the weights w."""
        n = len(w)
        off = up[:-1] * w[:-1] / np.sqrt(w[:-1] * w[1:])
        T = np.diag(up + down) - np.diag(off, 1) - np.diag(off, -1)
        lam, Q = np.linalg.eigh(T)
        r = np.sqrt(w)
        return lam, Q / r[:, None], (Q * r[:, None]).T

    @staticmethod
    def _apply(x, X, Y, shift):
        """(shift + X + Y) x for the 1-D operators X = (up, down) along the rows and Y along the columns."""
        y = (shift + (X[0] + X[1])[None, :] + (Y[0] + Y[1])[:, None]) * x
        y[:, :-1] -= X[0][:-1] * x[:, 1:]
        y[:, 1:] -= X[1][1:] * x[:, :-1]
        y[:-1] -= Y[0][:-1, None] * x[1:]
        y[1:] -= Y[1][1:, None] * x[:-1]
        return y

    def _solver(self, X, wx, Y, wy, shift):
        lx, Vx, Wx = self._modes(X[0], X[1], wx)
        ly, Vy, Wy = self._modes(Y[0], Y[1], wy)
        S = shift + lx[None, :] + ly[:, None]
        if shift == 0:
            S[0, 0] = np.inf  # the constant: what is left of it is the caller's

        def once(b):
            return Vy @ ((Wy @ b @ Wx.T) / S) @ Vx.T

        return once

    def solve_velocity(self, RU, RV):
        h = 0.5 * self.dt * self.nu
        out = []
        for R, (X, wx), (Y, wy) in (
                (RU, (self._second(self.dx, False), self.dx[1:] + self.dx[:-1]), (self._second(self.dy, True), self.dy)),
                (RV, (self._second(self.dx, True), self.dx), (self._second(self.dy, False), self.dy[1:] + self.dy[:-1]))):
            X, Y = [h * t for t in X], [h * t for t in Y]
            once = self._solver(X, wx, Y, wy, 1.0)
            x = once(R)
            for _ in range(2):
                x = x + once(R - self._apply(x, X, Y, 1.0))
            out.append(x)
        return out

    def rhs2(self, U, V):
        Uw, Vw = np.zeros((self.ny, self.nx + 1)), np.zeros((self.ny + 1, self.nx))
        Uw[:, 1:-1], Vw[1:-1] = U, V
        return -(Uw[:, 1:] - Uw[:, :-1]) / self.dx[None, :] - (Vw[1:] - Vw[:-1]) / self.dy[:, None]

    def solve_pressure(self, b):
        """The pinned pressure system: the diagonal is doubled at cell 0 and, inside, at the centre cell."""
        def ops(d):
            up, down = np.zeros(len(d)), np.zeros(len(d))
            up[:-1] = self.dt * 2 / (d[:-1] * (d[:-1] + d[1:]))
            down[1:] = self.dt * 2 / (d[1:] * (d[1:] + d[:-1]))
            return up, down
        X, Y = ops(self.dx), ops(self.dy)
        once = self._solver(X, self.dx, Y, self.dy, 0.0)
        w = np.outer(self.dy, self.dx)
        pins = [(0, 0)]
        cI, cJ = self.nx // 2, self.ny // 2
        if 0 < cI < self.nx - 1 and 0 < cJ < self.ny - 1:
            pins.append((cJ, cI))
        delta = [(X[0] + X[1])[i] + (Y[0] + Y[1])[j] for j, i in pins]

        def apply(x):
            y = self._apply(x, X, Y, 0.0)
            for (j, i), d in zip(pins, delta):
                y[j, i] += d * x[j, i]
            return y

        # x = G b - sum_k f_k G e_k + c with f_k = delta_k x_k and sum_k w_k f_k = w . b
        E = []
        for j, i in pins:
            e = np.zeros_like(w)
            e[j, i] = 1.0
            E.append(once(e))
        m = len(pins)
        M = np.zeros((m + 1, m + 1))
        for r, (j, i) in enumerate(pins):
            M[r, r] = 1 / delta[r]
            M[r, :m] += [g[j, i] for g in E]
            M[r, m] = -1.0
            M[m, r] = w[j, i]

        def solve(r):
            y = once(r)
            q = np.linalg.solve(M, np.array([y[j, i] for j, i in pins] + [np.sum(w * r)]))
            for k in range(m):
                y = y - q[k] * E[k]
            return y + q[m]

        x = solve(b)
        for _ in range(2):
            x = x + solve(b - apply(x))
        return x

    def project(self, U, V, P):
        return (U - (P[:, 1:] - P[:, :-1]) * self.dt * 2 / (self.dx[1:] + self.dx[:-1])[None, :],
                V - (P[1:] - P[:-1]) * self.dt * 2 / (self.dy[1:] + self.dy[:-1])[:, None])

    def cfl(self, U, V):
        f = np.zeros((self.ny, self.nx))
        f[:-1, :-1] = self.dt * (np.abs(U[:-1]) / self.dx[None, :-1] + np.abs(V[:, :-1]) / self.dy[:-1, None])
        return f


# ---------------------------------------------------------------------------------
# solvers with their states
# ---------------------------------------------------------------------------------
def _precision(case):
    return "MIXED" if case.get("precision") == "MIXED" else None


def _box_folder(folder, case):
    sim = {"type": "simulation", "dt": float(case["dt"]), "nt": 1000000, "nsave": 1000000,
           "SolverType": "NAVIER_STOKES_SOLVER",
           "linearSolvers": yaml_cases.solvers("DIAGONAL", case["tol"], "SMOOTHED_AGGREGATION", case["tol"],
                                               pois_krylov=case["krylov"], precision=_precision(case))}
    flow = [{"type": "flow", "nu": float(case["nu"]), "initialVelocity": [0.0, 0.0],
             "initialPerturbation": [0.0, 0.0],
             "boundaryConditions": yaml_cases.bcs((0, 0), (0, 0), (0, 0), (1.0, 0))}]
    dom = [yaml_cases.axis(d, -case[a], case["h"], _axis_subs(case[a], case["core"], case["ratio"]))
           for d, a in (("x", "ax"), ("y", "ay"))]
    return yaml_cases.write_case(folder, [sim], flow, dom, [])


def _cylinder_folder(folder, case, nu):
    return yaml_cases.cylinder(folder, h=case["h"], ratio=case["ratio"], extent=case["extent"],
                               points=case["points"], nu=nu, dt=case["dt"], nt=1000000, method=case["method"],
                               vel_tol=case["tol"], pois_tol=case["tol"], precision=_precision(case))


def _moving_folder(folder, case, nu):
    w = 2 * math.pi / case["period"]
    motion = {"xCoefficient": case["um"] / w, "uCoefficient": case["um"], "xfrequency": 1.0 / case["period"],
              "xPhase": -math.pi / 2, "uPhase": -math.pi / 2}
    return yaml_cases.cylinder(folder, h=case["h"], ratio=case["ratio"], extent=case["extent"], core=case["core"],
                               points=case["points"], nu=nu, dt=case["dt"], nt=1000000, method="OSC_CYLINDER",
                               quiescent=True, motion=motion, vel_tol=case["tol"], pois_tol=case["tol"])


def _batch_folders(tmp, case, seed):
    """Cavities (96 to 512 cells a side) and cylinders (core h 0.02 to 0.04) in turn, the sizes
    drawn with the case's number, the Reynolds numbers with the seed."""
    sizes, values = np.random.default_rng(case["sizes"]), np.random.default_rng(seed)
    out = []
    for k in range(case["count"]):
        f = os.path.join(tmp, "m%02d" % k)
        if k % 2 == 0:
            n = int(sizes.choice(np.arange(96, 513, 32)))
            re = float(np.exp(values.uniform(np.log(100), np.log(1000))))
            yaml_cases.cavity(f, n=n, nu=1.0 / re, dt=0.01 * 32 / n, nt=1000000, vel_tol=case["tol"],
                              pois_tol=case["tol"], pois_krylov="CG")
        else:
            h = float(sizes.choice([0.04, 0.03, 0.02]))
            re = float(np.exp(values.uniform(np.log(40), np.log(300))))
            pts = int(round(math.pi / h))
            yaml_cases.cylinder(f, h=h, ratio=1.03, points=pts + pts % 2, nu=1.0 / re, dt=0.005, nt=1000000,
                                vel_tol=case["tol"], pois_tol=case["tol"])
        out.append(f)
    return out


def _solver(folder):
    s = cb.NavierStokesSolver(folder)
    s.set_option("write_output", 0)
    return s


def _buffer(s, name):
    return torch.empty(s.field_size(name), dtype=torch.float64, device="cuda")


def _snapshot(s, names):
    """Device copies of a solver's fields."""
    out = []
    for name in names:
        t = _buffer(s, name)
        s.get_into(name, t.data_ptr(), t.numel() * D, on_device=True)
        out.append((name, t))
    return out


def _write(s, fields):
    for name, t in fields:
        s.set_from(name, t.data_ptr(), t.numel() * D, on_device=True, asynchronous=True)


def _read(s, fields):
    for name, t in fields:
        s.get_into(name, t.data_ptr(), t.numel() * D, on_device=True, asynchronous=True)


def _disturb(s, seed, size):
    """A smooth disturbance of the solver's velocity (the first steps then settle it)."""
    i, rng = s.info, np.random.default_rng(seed)
    u = s.get("u")
    U = u[:i.numU].reshape(i.ny, i.nx - 1)
    V = u[i.numU:].reshape(i.ny - 1, i.nx)
    U += size * _smooth(rng, s.get("xu"), s.get("yu"))
    V += size * _smooth(rng, s.get("xv"), s.get("yv"))
    s.set("u", u)


def prepare(case, seed):
    kind = case["kind"]
    torch.cuda.init()
    with tempfile.TemporaryDirectory(prefix="cuibm_case_") as tmp:
        folder = os.path.join(tmp, "case")
        if kind in ("box", "poisson", "explicit"):
            box = _Box(case, seed)
            s = _solver(_box_folder(folder, case))
            s.initialise()
            f = {k: torch.from_numpy(v).cuda() for k, v in box.fields().items()}
            if kind == "box":
                ins, outs = ["u", "N", "p", "uhat"], ["u", "uhat", "p", "N"]
            elif kind == "poisson":
                f["rhs2"] = torch.from_numpy(box.rhs2(box.U, box.V).ravel()).cuda()
                ins, outs = ["rhs2", "p"], ["p"]
            else:
                f["Nold"] = f.pop("N")
                ins, outs = ["u", "Nold", "p", "uhat"], ["N", "L", "bc1", "rhs1", "rhs2", "u", "cfl"]
            state = {"solver": s, "in": [(k, f[k]) for k in ins], "out": [(k, _buffer(s, k)) for k in outs]}
        elif kind == "cylinder":
            rng = np.random.default_rng(seed)
            s = _solver(_cylinder_folder(folder, case, case["nu"] * rng.uniform(0.9, 1.1)))
            s.initialise()
            _disturb(s, seed, 0.01)
            s.stepTime(2)
            state = {"solver": s, "in": _snapshot(s, ["u", "N", "p", "uhat", "bc_xplus"]),
                     "out": [(k, _buffer(s, k)) for k in ("u", "p", "forces")]}
        elif kind == "moving":
            rng = np.random.default_rng(seed)
            s = _solver(_moving_folder(folder, case, case["nu"] * rng.uniform(0.9, 1.1)))
            s.initialise()
            s.stepTime(1)
            state = {"solver": s, "in": [], "out": [(k, _buffer(s, k)) for k in ("u", "p", "forces")]}
        elif kind == "batch":
            b = cb.Batch(_batch_folders(tmp, case, seed))
            for s in b.instances:
                s.set_option("write_output", 0)
            b.initialise()
            for k, s in enumerate(b.instances):
                _disturb(s, seed + k, 0.02)
            b.stepTime(2)
            state = {"batch": b, "members": []}
            for s in b.instances:
                names = ["u", "N", "p", "uhat"] + (["bc_xplus"] if s.info.total_points else [])
                state["members"].append({"solver": s, "in": _snapshot(s, names),
                                         "out": [(k, _buffer(s, k)) for k in ("u", "p")]})
        else:
            rng = np.random.default_rng(seed)
            s = _solver(_moving_folder(folder, case, case["nu"] * rng.uniform(0.9, 1.1)))
            s.set_option("adjoint_tolerance", case["tol"])
            s.initialise()
            state = {"solver": s}
    state["case"] = case
    torch.cuda.synchronize()
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "adjoint":
        J, grad, _ = state["solver"].adjoint(case["steps"], 2.0 / case["steps"], snapshots=case["snapshots"])
        return {"J": float(J), "grad": grad}
    if kind == "batch":
        for m in state["members"]:
            _write(m["solver"], m["in"])
        state["batch"].stepTime(1)
        out = {}
        for k, m in enumerate(state["members"]):
            _read(m["solver"], m["out"])
            out["m%02d" % k] = {name: t for name, t in m["out"]}
        return out
    s = state["solver"]
    _write(s, state["in"])
    if kind == "poisson":
        s.run("solve_poisson")
    elif kind == "explicit":
        for op in ("rhs1_terms", "rhs2", "project", "cfl"):
            s.run(op)
    else:
        s.stepTime(1)
    _read(s, state["out"])
    return {name: t for name, t in state["out"]}


# ---------------------------------------------------------------------------------
# what a pass cannot do without, and its outputs in 64 bits
# ---------------------------------------------------------------------------------
def _step_work(nx, ny):
    nuv, n = (nx - 1) * ny + nx * (ny - 1), nx * ny
    # u, N, the velocity solve's start and p in; u, uhat, N and p out.  Explicit terms, and for
    # each solve a residual, a correction and the residual that shows it small
    return D * (6 * nuv + 2 * n), 60.0 * nuv + 30.0 * nuv + 30.0 * n


def work(case):
    kind = case["kind"]
    if kind == "batch":
        sizes = np.random.default_rng(case["sizes"])
        total = np.zeros(2)
        for k in range(case["count"]):
            if k % 2 == 0:
                n = int(sizes.choice(np.arange(96, 513, 32)))
            else:
                n = _count(15.0, 0.6, float(sizes.choice([0.04, 0.03, 0.02])), 1.03)
            total += _step_work(n, n)
        return {"bytes": total[0], "flops": total[1]}
    nx, ny = _sizes(case)
    nuv, n = (nx - 1) * ny + nx * (ny - 1), nx * ny
    if kind == "poisson":
        return {"bytes": D * 3.0 * n, "flops": 30.0 * n}
    if kind == "explicit":  # u, Nold, uhat, p in; N, L, bc1, rhs1, u, uold, rhs2, cfl out
        return {"bytes": D * (9.0 * nuv + 3.0 * n), "flops": 70.0 * nuv + 10.0 * n}
    b, f = _step_work(nx, ny)
    steps = 2 * case["steps"] if kind == "adjoint" else 1
    return {"bytes": steps * b, "flops": steps * f}


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("box", "poisson", "explicit"):
        return None
    g = _Box(case, seed)
    cat = lambda a: np.concatenate([a[0].ravel(), a[1].ravel()])  # noqa: E731
    if kind == "poisson":
        return {"p": g.solve_pressure(g.rhs2(g.U, g.V)).ravel()}
    N, L, B, R = g.rhs1(g.U, g.V, g.NU, g.NV)
    if kind == "explicit":
        unew = g.project(g.U, g.V, g.P)
        return {"N": cat(N), "L": cat(L), "bc1": cat(B), "rhs1": cat(R), "rhs2": g.rhs2(g.U, g.V).ravel(),
                "u": cat(unew), "cfl": g.cfl(*unew).ravel()}
    uh = g.solve_velocity(*R)
    p = g.solve_pressure(g.rhs2(*uh))
    return {"u": cat(g.project(uh[0], uh[1], p)), "uhat": cat(uh), "p": p.ravel(), "N": cat(N)}
