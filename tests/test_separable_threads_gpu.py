"""Contexts of different sizes set up by several threads at once: a kernel's shared-memory limit
belongs to the process, so no context may lower what another one is about to launch with
(the set-up's rotations ask for 64 bytes a place: more than the 48 KB default from 769 on)."""
import threading

import numpy as np
import pytest

cb = pytest.importorskip("cuibm_gb300")
from cuibm_gb300 import cases  # noqa: E402

pytestmark = pytest.mark.gpu


def case(folder, nx, ny):
    sim = {"type": "simulation", "dt": 0.003, "nt": 10, "nsave": 10, "SolverType": "NAVIER_STOKES_SOLVER",
           "linearSolvers": cases.solvers("DIAGONAL", 1e-10, "SMOOTHED_AGGREGATION", 1e-10, pois_krylov="BICGSTAB",
                                          vel_krylov="BICGSTAB")}
    flow = [{"type": "flow", "nu": 0.01, "initialVelocity": [0.0, 0.0],
             "boundaryConditions": cases.bcs((0, 0), (0, 0), (0, 0), (1.0, 0))}]
    return cases.write_case(folder, [sim], flow, [cases.axis("x", 0.0, 0.01, [((nx + 0.5) * 0.01, 1.0)]),
                                                  cases.axis("y", 0.0, 0.01, [((ny + 0.5) * 0.01, 1.0)])], [])


def pressure(folder):
    with cb.NavierStokesSolver(folder, ["-separable", "1"]) as s:
        s.set_option("write_output", 0)
        s.initialise()
        s.stepTime(2)
        return s.get("p")


def test_set_ups_side_by_side(tmp_path):
    folders = [case(str(tmp_path / ("c%d" % n)), n, n + 10) for n in (790, 60, 850, 75)]
    alone = [pressure(f) for f in folders]
    failures = []

    def work(k):
        try:
            for _ in range(3 if k % 2 == 0 else 25):
                assert np.array_equal(pressure(folders[k]), alone[k])
        except Exception as e:  # noqa: BLE001  (reported by the test's thread)
            failures.append((k, repr(e)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(folders))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures


def test_bodies_side_by_side(tmp_path):
    """Contexts with bodies come and go in several threads; each keeps its own body's lists."""
    def cylinder(k):
        return cases.cylinder(str(tmp_path / ("b%d" % k)), h=0.05, ratio=1.1, extent=3.0, core=0.6, points=40 + 9 * k,
                              nu=0.025, dt=0.01, nt=10, vel_tol=1e-10, pois_tol=1e-10,
                              method=("LUO", "FADLUN", "OSC_CYLINDER", "LUO")[k])

    def run(folder):
        with cb.NavierStokesSolver(folder) as s:
            s.set_option("write_output", 0)
            s.initialise()
            s.stepTime(2)
            return s.get("u"), s.get("ghost_tags_uv"), np.array(s.forces())

    folders = [cylinder(k) for k in range(4)]
    alone, failures = [run(f) for f in folders], []

    def work(k):
        try:
            for _ in range(6):
                assert all(np.array_equal(a, b) for a, b in zip(run(folders[k]), alone[k]))
        except Exception as e:  # noqa: BLE001  (reported by the test's thread)
            failures.append((k, repr(e)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures
