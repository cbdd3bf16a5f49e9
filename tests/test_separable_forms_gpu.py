"""The separable solves' less common forms (csrc/separable.cu): the four-digit products of
mixed-precision Fadlun cases at the splitting kernels' and tiles' edges, bodies on both sides of
the capacitance matrices' limits, the longest transforms, and right-hand sides that are not
finite in every kind of solve.

Residual bound as in test_separable_gpu: tol ||b|| + 40 eps || |A| |x| + |b| || (six rounded
terms a row, a few updates of x)."""
import numpy as np
import pytest

cb = pytest.importorskip("cuibm_gb300")
sp = pytest.importorskip("scipy.sparse")
from cuibm_gb300 import cases  # noqa: E402

pytestmark = pytest.mark.gpu
TOL = 1e-12
EPS = np.finfo(float).eps


def solver(folder, *args):
    s = cb.NavierStokesSolver(folder, list(args) or ["-separable", "1"])
    s.set_option("write_output", 0)
    s.initialise()
    return s


def names(s, system):
    return (s.info.numP, "rhs2", "p", "solve_poisson") if system == 2 else (s.info.numUV, "rhs1", "uhat",
                                                                            "solve_velocity")


def check(s, b, x0, system):
    n, rhs, sol, op = names(s, system)
    s.set(rhs, b)
    s.set(sol, x0)
    s.run(op)
    x = s.get(sol)
    r, c, v = s.matrix(system)
    A = sp.coo_matrix((v, (r, c)), shape=(n, n)).tocsr()
    floor = np.linalg.norm(abs(A) @ np.abs(x) + np.abs(b))
    res = np.linalg.norm(b - A @ x)
    assert res <= TOL * np.linalg.norm(b) + 40 * EPS * floor, (res, np.linalg.norm(b), floor)


def cylinder(folder, h, ratio, extent, points, method="FADLUN", precision=None, core=0.6, **kw):
    return cases.cylinder(folder, h=h, ratio=ratio, extent=extent, core=core, points=points, nu=0.025, dt=0.01, nt=10,
                          vel_tol=TOL, pois_tol=TOL, method=method, precision=precision, **kw)


# cells a side on both sides of the splitting kernels' 256, 512 and 1024 places and of the row
# kernels' 400 (from where on there are enough 32 x 64 tiles, too)
FADLUN = [(0.02, 1.0293984, 256), (0.02, 1.029, 258), (0.015, 1.0161333, 400), (0.015, 1.016, 402),
          (0.012, 1.0123137, 512), (0.012, 1.0122198, 514), (0.008, 1.0046178, 1024), (0.008, 1.0045992, 1026)]


@pytest.mark.parametrize("precision", ["MIXED", None])
@pytest.mark.parametrize("h,ratio,cells", FADLUN)
def test_fadlun_sizes(tmp_path, h, ratio, cells, precision):
    f = cylinder(str(tmp_path / "c"), h, ratio, 11.9, int(round(np.pi / h)), precision=precision)
    with solver(f) as s:
        assert s.info.nx == s.info.ny == cells
        rng = np.random.default_rng(cells)
        for system in (2, 1):
            n = names(s, system)[0]
            check(s, rng.standard_normal(n), rng.standard_normal(n), system)


def patched_rows(s):
    """(velocity, pressure) rows that the Fadlun method patches, from the tags."""
    nx, ny = s.info.nx, s.info.ny
    nU = (nx - 1) * ny
    g, h = s.get("ghost_tags_uv"), s.get("hybrid_tags_uv")
    uv = ((h != -1) | (g != -1)) & (g != 0)
    u, v = uv[:nU].reshape(ny, nx - 1)[1:-1, 1:-1], uv[nU:].reshape(ny - 1, nx)[1:-1, 1:-1]
    p = ((s.get("hybrid_tags_p") != -1) | (s.get("ghost_tags_p") > 0)).reshape(ny, nx)[1:-1, 1:-1]
    return u.sum() + v.sum(), p.sum()


@pytest.mark.parametrize("h,above", [(0.013, (False, False)), (0.006, (True, False)), (0.0017, (True, True))])
def test_capacitance_limits(tmp_path, h, above):
    """Bodies of fewer and more rows than the capacitance matrices take (1024 velocity rows, 2048
    pressure rows): the larger systems keep their other preconditioner, with the bits of
    -separable 0."""
    f = cylinder(str(tmp_path / "c"), h, 1.2, 2.5, int(round(np.pi / h)))
    with solver(f) as s, solver(f, "-separable", "0") as other:
        rows = patched_rows(s)
        assert (rows[0] > 1024, rows[1] > 2048) == above, rows
        rng = np.random.default_rng(3)
        for system in (2, 1):
            n, rhs, sol, op = names(s, system)
            b, x0 = rng.standard_normal(n), rng.standard_normal(n)
            if not above[system - 1]:
                check(s, b, x0, system)
                continue
            for t in (s, other):
                t.set(rhs, b)
                t.set(sol, x0)
                t.run(op)
            assert np.array_equal(s.get(sol), other.get(sol))
            assert s.iterations()[system - 1] == other.iterations()[system - 1]


def box(folder, nx, ny, krylov, precision=None, nu=0.01):
    sim = {"type": "simulation", "dt": 0.003, "nt": 10, "nsave": 10, "SolverType": "NAVIER_STOKES_SOLVER",
           "linearSolvers": cases.solvers("DIAGONAL", TOL, "SMOOTHED_AGGREGATION", TOL, pois_krylov=krylov,
                                          vel_krylov=krylov, precision=precision)}
    flow = [{"type": "flow", "nu": nu, "initialVelocity": [0.0, 0.0],
             "boundaryConditions": cases.bcs((0, 0), (0, 0), (0, 0), (1.0, 0))}]
    return cases.write_case(folder, [sim], flow, [cases.axis("x", 0.0, 0.01, [((nx + 0.5) * 0.01, 1.0)]),
                                                  cases.axis("y", 0.0, 0.01, [((ny + 0.5) * 0.01, 1.0)])], [])


@pytest.mark.parametrize("nx,ny", [(1300, 1310), (2048, 2048), (2060, 2047)])
def test_longest_transforms(tmp_path, nx, ny):
    """Up to 2048 places, along both directions; the residual by the matrix-free operator."""
    with solver(box(str(tmp_path / "c"), nx, ny, "BICGSTAB")) as s:
        n, m = s.info.numP, s.info.numUV
        rng = np.random.default_rng(nx)
        b = rng.standard_normal(n)
        s.set("rhs2", b)
        s.set("p", np.zeros(n))
        s.run("solve_poisson")
        assert s.iterations()[1] <= 3
        x = s.get("p")

        def apply(v):
            s.set("work_x", np.concatenate([v, np.zeros(m - n)]))
            s.run("apply_lhs2")
            return s.get("work_y")[:n]

        # |A| |x| <= 8 dt / h^2 |x|'s largest neighbours: bounded by twice the diagonal times the norm
        floor = 2 * 2 * 4 * 0.003 / 1e-4 * np.linalg.norm(x) + np.linalg.norm(b)
        assert np.linalg.norm(b - apply(x)) <= TOL * np.linalg.norm(b) + 40 * EPS * floor


MOTION = {"xCoefficient": 0.05, "uCoefficient": 0.05 * 2 * np.pi, "xfrequency": 1.0, "xPhase": 0.0, "uPhase": 0.0}
KINDS = {"CG by rows": lambda f: box(f, 60, 64, "CG"), "BiCGSTAB by rows": lambda f: box(f, 60, 64, "BICGSTAB"),
         "CG": lambda f: box(f, 420, 430, "CG"), "BiCGSTAB": lambda f: box(f, 420, 430, "BICGSTAB"),
         "along y": lambda f: box(f, 70, 60, "BICGSTAB", "MIXED"),
         "Fadlun": lambda f: cylinder(f, 0.05, 1.1, 3.0, 48), "Fadlun mixed": lambda f: cylinder(
             f, 0.05, 1.1, 3.0, 48, precision="MIXED"),
         "embedded": lambda f: cylinder(f, 0.05, 1.1, 3.0, 48, "OSC_CYLINDER"),
         "embedded, moving": lambda f: cylinder(f, 0.05, 1.1, 3.0, 48, "OSC_CYLINDER", motion=MOTION)}


@pytest.mark.parametrize("bad", [np.nan, np.inf, 1e300])
@pytest.mark.parametrize("kind", KINDS)
def test_right_hand_sides_that_are_not_finite(tmp_path, kind, bad):
    """Reported as such (1e300: the norm overflows), and the solver is usable again."""
    with solver(KINDS[kind](str(tmp_path / "c"))) as s:
        rng = np.random.default_rng(5)
        for system in (2, 1):
            n, rhs, sol, op = names(s, system)
            b = rng.standard_normal(n)
            b[n // 3] = bad
            s.set(rhs, b)
            s.set(sol, np.zeros(n))
            with pytest.raises(cb.CuibmError) as e:
                s.run(op)
            assert e.value.status == cb.ERR_NAN, system
            check(s, rng.standard_normal(n), np.zeros(n), system)
