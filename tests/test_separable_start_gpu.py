"""Separable solves whose starting vector meets the tolerance already, or just misses it: the
first leave it as it is, to the bit and with no iteration, and the second solve.  The residual
is set to a multiple of the tolerance, 1e-4 to either side of it (the kernels' early look at it
is good to 1e-5, and decides nothing by itself), and far from it."""
import numpy as np
import pytest

cb = pytest.importorskip("cuibm_gb300")
sp = pytest.importorskip("scipy.sparse")
from cuibm_gb300 import cases  # noqa: E402

pytestmark = pytest.mark.gpu
TOL = 1e-3
MOTION = {"xCoefficient": 0.05, "uCoefficient": 0.05 * 2 * np.pi, "xfrequency": 1.0, "xPhase": 0.0, "uPhase": 0.0}


def box(folder, nx, ny, krylov, precision=None):
    sim = {"type": "simulation", "dt": 0.003, "nt": 10, "nsave": 10, "SolverType": "NAVIER_STOKES_SOLVER",
           "linearSolvers": cases.solvers("DIAGONAL", TOL, "SMOOTHED_AGGREGATION", TOL, pois_krylov=krylov,
                                          vel_krylov=krylov, precision=precision)}
    flow = [{"type": "flow", "nu": 0.05, "initialVelocity": [0.0, 0.0],
             "boundaryConditions": cases.bcs((0, 0), (0, 0), (0, 0), (1.0, 0))}]
    return cases.write_case(folder, [sim], flow, [cases.axis("x", 0.0, 0.01, [((nx + 0.5) * 0.01, 1.0)]),
                                                  cases.axis("y", 0.0, 0.01, [((ny + 0.5) * 0.01, 1.0)])], [])


def cylinder(folder, method, **kw):
    return cases.cylinder(folder, h=0.05, ratio=1.1, extent=3.0, core=0.6, points=48, nu=0.025, dt=0.01, nt=10,
                          vel_tol=TOL, pois_tol=TOL, method=method, **kw)


KINDS = {"CG by rows": lambda f: box(f, 60, 64, "CG"), "BiCGSTAB by rows": lambda f: box(f, 60, 64, "BICGSTAB"),
         "CG": lambda f: box(f, 420, 430, "CG"), "BiCGSTAB": lambda f: box(f, 420, 430, "BICGSTAB"),
         "along y": lambda f: box(f, 70, 60, "BICGSTAB", "MIXED"), "Fadlun": lambda f: cylinder(f, "FADLUN"),
         "external": lambda f: cylinder(f, "LUO"), "embedded": lambda f: cylinder(f, "OSC_CYLINDER"),
         "embedded, moving": lambda f: cylinder(f, "OSC_CYLINDER", motion=MOTION)}


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("system", [1, 2])
def test_starts_beside_the_tolerance(tmp_path, kind, system):
    with cb.NavierStokesSolver(KINDS[kind](str(tmp_path / "c")), ["-separable", "1"]) as s:
        s.set_option("write_output", 0)
        s.initialise()
        n, rhs, sol, op = ((s.info.numP, "rhs2", "p", "solve_poisson") if system == 2 else
                           (s.info.numUV, "rhs1", "uhat", "solve_velocity"))
        r, c, v = s.matrix(system)
        A = sp.coo_matrix((v, (r, c)), shape=(n, n)).tocsr()
        rng = np.random.default_rng(n)
        x, d = rng.standard_normal(n), rng.standard_normal(n)
        d /= np.linalg.norm(d)
        Ax = A @ x

        def run(multiple, scale):
            """The solve from x with ||b - A x|| = multiple tol ||b||; everything times scale."""
            t = 0.0
            for _ in range(60):
                t = multiple * TOL * np.linalg.norm(Ax + t * d)
            s.set(rhs, scale * (Ax + t * d))
            s.set(sol, scale * x)
            s.run(op)
            b, y = s.get(rhs), s.get(sol)
            same = np.array_equal(y, scale * x)
            if not same:
                assert np.linalg.norm(b - A @ y) <= 1.001 * TOL * np.linalg.norm(b)
            return same

        for scale in (1.0, 1e-30, 1e40):
            for multiple, met in ((0.0, True), (1e-3, True), (0.5, True), (1 - 1e-4, True), (1 + 1e-4, False), (3.0, False),
                                  (1 - 1e-4, True), (100.0, False)):
                assert run(multiple, scale) == met, (scale, multiple)
                if met:
                    assert s.iterations()[system - 1] == 0
        s.set(rhs, np.zeros(n))
        s.set(sol, np.zeros(n))
        s.run(op)
        assert np.all(s.get(sol) == 0)


@pytest.mark.parametrize("krylov", ["CG", "BICGSTAB"])
@pytest.mark.parametrize("n", [64, 410])
def test_a_flow_comes_to_rest(tmp_path, krylov, n):
    """Steps with and without the step graph, through solves of no iteration and of some: same bits."""
    out = []
    for graph in (1, 0):
        with cb.NavierStokesSolver(box(str(tmp_path / ("c%d" % graph)), n, n, krylov), ["-separable", "1"]) as s:
            s.set_option("write_output", 0)
            s.set_option("use_graph", graph)
            s.initialise()
            its = []
            for _ in range(40):
                s.stepTime(5)
                its.append(s.iterations())
            out.append((s.get("u"), s.get("p"), its))
    assert out[0][2] == out[1][2] and np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
