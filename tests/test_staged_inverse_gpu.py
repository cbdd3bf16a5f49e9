"""Persistent solves that keep the coarsest inverse in shared memory, with the block and thread
counts a case may ask for (-solverBlocks, -solverThreads, option solver_blocks): every grid
that fits the SMs without it still launches, and the solution meets its residual bound (the
tolerance, and 40 eps of |A| |x| + |b| for the rounding of x and of five terms a row)."""
import numpy as np
import pytest

cb = pytest.importorskip("cuibm_gb300")
sp = pytest.importorskip("scipy.sparse")
from cuibm_gb300 import cases  # noqa: E402

pytestmark = pytest.mark.gpu
TOL = 1e-11


def case(folder, nx, ny, precision):
    sim = {"type": "simulation", "dt": 0.003, "nt": 10, "nsave": 10, "SolverType": "NAVIER_STOKES_SOLVER",
           "linearSolvers": cases.solvers("DIAGONAL", TOL, "SMOOTHED_AGGREGATION", TOL, pois_krylov="BICGSTAB",
                                          vel_krylov="BICGSTAB", precision=precision)}
    flow = [{"type": "flow", "nu": 0.01, "initialVelocity": [0.0, 0.0],
             "boundaryConditions": cases.bcs((0, 0), (0, 0), (0, 0), (1.0, 0))}]
    return cases.write_case(folder, [sim], flow, [cases.axis("x", 0.0, 0.01, [((nx + 0.5) * 0.01, 1.0)]),
                                                  cases.axis("y", 0.0, 0.01, [((ny + 0.5) * 0.01, 1.0)])], [])


def solve(s, rng):
    n = s.info.numP
    b = rng.standard_normal(n)
    s.set("rhs2", b)
    s.set("p", np.zeros(n))
    s.run("solve_poisson")
    x = s.get("p")
    r, c, v = s.matrix(2)
    A = sp.coo_matrix((v, (r, c)), shape=(n, n)).tocsr()
    floor = np.linalg.norm(abs(A) @ np.abs(x) + np.abs(b))
    assert np.linalg.norm(b - A @ x) <= TOL * np.linalg.norm(b) + 40 * np.finfo(float).eps * floor


# 38 x 39: one level of 1482 unknowns; 110 x 97: three levels
@pytest.mark.parametrize("nx,ny", [(38, 39), (110, 97)])
@pytest.mark.parametrize("precision", [None, "MIXED"])
@pytest.mark.parametrize("threads", [256, 512])
def test_block_and_thread_counts(tmp_path, nx, ny, precision, threads):
    f, rng = case(str(tmp_path / "c"), nx, ny, precision), np.random.default_rng(threads)
    args = ["-separable", "0", "-solverThreads", str(threads)]
    for blocks in (1, 160, 304):
        with cb.NavierStokesSolver(f, args + ["-solverBlocks", str(blocks)]) as s:
            s.set_option("write_output", 0)
            s.initialise()
            solve(s, rng)
    with cb.NavierStokesSolver(f, args) as s:
        s.set_option("write_output", 0)
        s.initialise()
        for blocks in (0, 153, 20, 170):
            s.set_option("solver_blocks", blocks)
            solve(s, rng)
            s.stepTime(1)
