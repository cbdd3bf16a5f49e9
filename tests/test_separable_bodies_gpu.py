"""Separable pressure solves with an embedded body's rows (csrc/separable.cu), whose last
correction uses a preconditioner that is only near the operator's inverse: whatever the
tolerance, the solution meets it in the assembled matrix's residual, and its level (fixed by
one pinned corner cell) is that of a direct solve.

The residual's bound is the tolerance and the rounding of x and of the operator (five terms a
row, a dozen in a body's): 60 eps || |A| |x| + |b| ||.  The level: a relative residual of
1e-12 left up to 2e-9 of the pressure before the correction; bound 1e-8."""
import numpy as np
import pytest

cb = pytest.importorskip("cuibm_gb300")
sp = pytest.importorskip("scipy.sparse")
from scipy.sparse.linalg import spsolve  # noqa: E402

from cuibm_gb300 import cases  # noqa: E402

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps


def solver(folder, tol, moving, graph=1):
    motion = {"xCoefficient": 0.05, "uCoefficient": 0.05 * 2 * np.pi, "xfrequency": 1.0, "xPhase": 0.0,
              "uPhase": 0.0} if moving else None
    f = cases.cylinder(folder, h=0.04, ratio=1.08, extent=4.0, core=0.7, points=78, nu=0.025, dt=0.01, nt=20,
                       vel_tol=tol, pois_tol=tol, method="OSC_CYLINDER", motion=motion)
    s = cb.NavierStokesSolver(f, ["-separable", "1"])
    s.set_option("write_output", 0)
    s.set_option("use_graph", graph)
    s.initialise()
    return s


def matrix(s):
    n = s.info.numP
    r, c, v = s.matrix(2)
    return sp.coo_matrix((v, (r, c)), shape=(n, n)).tocsr()


def residual(A, b, x, tol):
    """The residual's norm as a multiple of what the tolerance and rounding allow."""
    bound = tol * np.linalg.norm(b) + 60 * EPS * np.linalg.norm(abs(A) @ np.abs(x) + np.abs(b))
    return np.linalg.norm(b - A @ x) / bound


@pytest.mark.parametrize("moving", [False, True])
@pytest.mark.parametrize("tol", [1e-1, 3e-2, 1e-3, 2e-5, 1e-8, 1e-12])
def test_solves_meet_their_tolerance(tmp_path, tol, moving):
    with solver(str(tmp_path / "c"), tol, moving) as s:
        s.stepTime(3)
        A, rng = matrix(s), np.random.default_rng(7)
        n = A.shape[0]
        for k in range(24):
            b = rng.standard_normal(n) if k % 2 else A @ rng.standard_normal(n)
            s.set("rhs2", b)
            s.set("p", rng.standard_normal(n) * (k % 3))
            s.run("solve_poisson")
            assert residual(A, b, s.get("p"), tol) <= 1, k


@pytest.mark.parametrize("graph", [0, 1])
def test_steps_meet_their_tolerance(tmp_path, graph):
    """A fixed body's steps leave the right-hand side and the solution of their pressure solve."""
    with solver(str(tmp_path / "c"), 1e-3, False, graph) as s:
        A = matrix(s)
        for k in range(15):
            s.stepTime(1)
            assert residual(A, s.get("rhs2"), s.get("p"), 1e-3) <= 1, k


@pytest.mark.parametrize("moving", [False, True])
def test_the_level_is_a_direct_solves(tmp_path, moving):
    with solver(str(tmp_path / "c"), 1e-12, moving) as s:
        s.stepTime(3)
        A, b = matrix(s), s.get("rhs2")
        s.run("solve_poisson")
        p, ref = s.get("p"), spsolve(A.tocsc(), b)
        assert np.linalg.norm(p - ref) <= 1e-8 * np.linalg.norm(ref)
