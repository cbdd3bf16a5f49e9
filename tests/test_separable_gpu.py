"""The separable preconditioner (csrc/separable.cu): pressure and velocity solves on
grids at the edges of its tiles - chunks of 32 terms, product tiles of 32 x 32 and 32 x 64,
the splitting kernels' 256, 512 and 1024 places, the tridiagonal blocks of 4 and 8 modes -
along both transform directions, uniform and stretched, for both Krylov methods and
precisions, against the residual of the assembled matrix.

The bound: the solver stops at ||r|| <= tol ||b|| for the recursively updated r; x is the
sum of at most a few updates, each rounded to half an ulp, and each application of A (five
terms a row) rounds by at most 6 eps of |A| |x|, so the true residual is below
tol ||b|| + 40 eps || |A| |x| + |b| ||."""
import numpy as np
import pytest

cb = pytest.importorskip("cuibm_gb300")
sp = pytest.importorskip("scipy.sparse")
from cuibm_gb300 import cases  # noqa: E402

pytestmark = pytest.mark.gpu
TOL = 1e-12


def box(folder, nx, ny, ratio, krylov, precision, tol=TOL, nu=0.01):
    """nx x ny cells: uniform, or stretched away from the first corner (the counts of a
    stretched axis follow from its length)."""
    def axis(name, n):
        if ratio == 1.0:
            return cases.axis(name, 0.0, 0.01, [((n + 0.5) * 0.01, 1.0)])
        return cases.axis(name, 0.0, 0.01, [(0.01 * (ratio ** (n + 0.5) - 1) / (ratio - 1), ratio)])
    sim = {"type": "simulation", "dt": 0.003, "nt": 10, "nsave": 10, "SolverType": "NAVIER_STOKES_SOLVER",
           "linearSolvers": cases.solvers("DIAGONAL", tol, "SMOOTHED_AGGREGATION", tol, pois_krylov=krylov,
                                          vel_krylov=krylov, precision=precision)}
    flow = [{"type": "flow", "nu": nu, "initialVelocity": [0.0, 0.0], "initialPerturbation": [0.0, 0.0],
             "boundaryConditions": cases.bcs((0, 0), (0, 0), (0, 0), (1.0, 0))}]
    return cases.write_case(folder, [sim], flow, [axis("x", nx), axis("y", ny)], [])


def solver(folder, args=("-separable", "1")):
    s = cb.NavierStokesSolver(folder, args)
    s.set_option("write_output", 0)
    s.initialise()
    return s


def check(s, b, p0, system=2):
    n, rhs, sol, op = ((s.info.numP, "rhs2", "p", "solve_poisson") if system == 2 else
                       (s.info.numUV, "rhs1", "uhat", "solve_velocity"))
    s.set(rhs, b)
    s.set(sol, p0)
    s.run(op)
    p = s.get(sol)
    r, c, v = s.matrix(system)
    A = sp.coo_matrix((v, (r, c)), shape=(n, n)).tocsr()
    floor = np.linalg.norm(abs(A) @ np.abs(p) + np.abs(b))
    res = np.linalg.norm(b - A @ p)
    assert res <= TOL * np.linalg.norm(b) + 40 * np.finfo(float).eps * floor, (res, np.linalg.norm(b), floor)
    return p


SIZES = [(3, 3, 1.0), (5, 4, 1.3), (31, 40, 1.05), (32, 33, 1.0), (33, 32, 1.0), (64, 65, 1.02), (129, 63, 1.0),
         (257, 90, 1.01), (700, 24, 1.0), (24, 700, 1.0), (290, 1100, 1.0), (521, 530, 1.004), (610, 601, 1.0),
         (1033, 1040, 1.0), (40, 512, 1.0), (40, 513, 1.0), (40, 1024, 1.0), (40, 1025, 1.0)]


@pytest.mark.parametrize("nx,ny,ratio", SIZES)
@pytest.mark.parametrize("krylov,precision", [("BICGSTAB", None), ("CG", None), ("BICGSTAB", "MIXED")])
def test_solves_meet_the_residual_bound(tmp_path, nx, ny, ratio, krylov, precision):
    with solver(box(str(tmp_path / "c"), nx, ny, ratio, krylov, precision)) as s:
        i = s.info
        assert (i.nx, i.ny) == (nx, ny)
        rng = np.random.default_rng(nx * 1000 + ny)
        for b in (rng.standard_normal(i.numP), np.repeat(rng.standard_normal(ny), nx)):
            check(s, b, rng.standard_normal(i.numP))
            assert s.iterations()[1] <= 3  # the inverse to rounding
        check(s, rng.standard_normal(i.numUV), rng.standard_normal(i.numUV), system=1)


@pytest.mark.parametrize("nx,ny,ratio", [(3, 3, 1.0), (33, 32, 1.0), (65, 31, 1.03), (120, 257, 1.0), (514, 130, 1.0),
                                         (40, 512, 1.0), (40, 513, 1.0), (1024, 40, 1.0), (40, 1025, 1.0)])
@pytest.mark.parametrize("krylov,precision", [("BICGSTAB", None), ("CG", None), ("BICGSTAB", "MIXED")])
def test_velocity_solves_meet_the_residual_bound(tmp_path, nx, ny, ratio, krylov, precision):
    """nu large enough that the diagonal preconditioner would take tens of iterations."""
    with solver(box(str(tmp_path / "c"), nx, ny, ratio, krylov, precision, nu=1.0)) as s:
        rng = np.random.default_rng(nx + ny)
        check(s, rng.standard_normal(s.info.numUV), rng.standard_normal(s.info.numUV), system=1)
        assert s.iterations()[0] <= 2


def test_agrees_with_smoothed_aggregation_and_runs_in_steps(tmp_path):
    f = box(str(tmp_path / "c"), 90, 71, 1.02, "BICGSTAB", None)
    out = []
    for flag, graph in (("1", 1), ("1", 0), ("0", 1)):
        with solver(f, ["-separable", flag]) as s:
            s.set_option("use_graph", graph)
            s.stepTime(12)
            out.append((s.get("u"), s.get("p"), s.iterations()[1]))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
    (u, p, it), _, (us, ps, its) = out
    assert it <= 2 < its
    assert np.linalg.norm(u - us) <= 1e-9 * np.linalg.norm(us) and np.linalg.norm(p - ps) <= 1e-9 * np.linalg.norm(ps)


def test_zero_and_non_finite_right_hand_sides(tmp_path):
    with solver(box(str(tmp_path / "c"), 40, 36, 1.0, "BICGSTAB", None)) as s:
        n = s.info.numP
        assert np.all(check(s, np.zeros(n), np.zeros(n)) == 0)
        b = np.ones(n)
        b[77] = np.inf
        s.set("rhs2", b)
        with pytest.raises(cb.CuibmError) as e:
            s.run("solve_poisson")
        assert e.value.status == cb.ERR_NAN
        check(s, np.random.default_rng(1).standard_normal(n), np.zeros(n))  # and is usable again


@pytest.mark.parametrize("h,points,precision", [(0.05, 48, None), (0.05, 48, "MIXED"), (0.021, 150, None)])
def test_patched_rows_of_a_fixed_body(tmp_path, h, points, precision):
    """The modified Fadlun method's rows at the body: the capacitance matrix makes the
    preconditioner the patched operator's inverse, so one or two iterations are left."""
    f = cases.cylinder(str(tmp_path / "c"), h=h, ratio=1.1, extent=3.0, core=0.6, points=points, nu=0.025, dt=0.01,
                       nt=10, vel_tol=TOL, pois_tol=TOL, method="FADLUN", precision=precision)
    with solver(f) as s:
        rng = np.random.default_rng(points)
        check(s, rng.standard_normal(s.info.numP), rng.standard_normal(s.info.numP))
        assert s.iterations()[1] <= 3


@pytest.mark.parametrize("method,precision,moving", [("LUO", None, False), ("LUO", "MIXED", False),
                                                     ("FADLUN", None, False), ("FADLUN", "MIXED", False),
                                                     ("OSC_CYLINDER", None, False), ("OSC_CYLINDER", None, True)])
def test_body_methods_agree_with_smoothed_aggregation(tmp_path, method, precision, moving):
    """Each immersed-boundary method's steps with the separable preconditioner and with smoothed
    aggregation, both solved to 1e-12: u to 1e-9, p less its mean (one pinned corner cell fixes
    its level) to 1e-8, the forces to 1e-9 of their size."""
    motion = {"xCoefficient": 0.05, "uCoefficient": 0.05 * 2 * np.pi, "xfrequency": 1.0, "xPhase": 0.0,
              "uPhase": 0.0} if moving else None
    f = cases.cylinder(str(tmp_path / "c"), h=0.04, ratio=1.08, extent=4.0, core=0.7, points=78, nu=0.025, dt=0.01, nt=20,
                       vel_tol=TOL, pois_tol=TOL, method=method, precision=precision, motion=motion)
    out = []
    for flag in ("1", "0"):
        with solver(f, ["-separable", flag]) as s:
            s.stepTime(15)
            p = s.get("p")
            out.append((s.get("u"), p - p.mean(), np.array(s.forces())))
    (u, p, fo), (us, ps, fs) = out
    assert np.linalg.norm(u - us) <= 1e-9 * np.linalg.norm(us)
    assert np.linalg.norm(p - ps) <= 1e-8 * np.linalg.norm(ps)
    assert np.max(np.abs(fo - fs)) <= 1e-9 * max(1.0, np.max(np.abs(fs)))


@pytest.mark.parametrize("nx,ny,separable", [(30, 50, False), (38, 39, False), (19, 79, True), (39, 39, True)])
def test_one_level_systems_keep_their_dense_inverse(tmp_path, nx, ny, separable):
    """Up to 1500 pressure unknowns the default is the one-level hierarchy: the bits of -separable 0."""
    out = []
    for args in ((), ("-separable", "0")):
        with solver(box(str(tmp_path / ("c%d" % len(out))), nx, ny, 1.0, "BICGSTAB", None), args) as s:
            s.set("rhs2", np.random.default_rng(5).standard_normal(s.info.numP))
            s.run("solve_poisson")
            out.append(s.get("p"))
    assert np.array_equal(*out) == (not separable)
