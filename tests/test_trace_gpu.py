"""The solve trace (option trace_solve, python -m cuibm_gb300.trace): a step's persistent and
separable solves leave stamps in time order whose sites are lines that stamp, without a change
to any bit of the solution; a solve launched phase by phase leaves none, not another's."""
import numpy as np
import pytest

cb = pytest.importorskip("cuibm_gb300")
from cuibm_gb300 import cases, trace  # noqa: E402

pytestmark = pytest.mark.gpu


def case(tmp_path, kind):
    if kind == "cavity":  # CG by rows
        return cases.cavity(str(tmp_path / "c"), n=64, nu=0.01, dt=0.01, nt=100, vel_tol=1e-10, pois_tol=1e-10)
    if kind == "mixed":  # BiCGSTAB, flat kernels
        return cases.cavity(str(tmp_path / "c"), n=420, nu=0.01, dt=0.0005, nt=100, vel_tol=1e-10, pois_tol=1e-10,
                            pois_krylov="BICGSTAB", vel_krylov="BICGSTAB", precision="MIXED")
    return cases.cylinder(str(tmp_path / "c"), h=0.05, ratio=1.1, extent=3.0, core=0.6, points=48, nu=0.025, dt=0.01,
                          nt=100, vel_tol=1e-10, pois_tol=1e-10, method=kind)


def solver(f, separable, graph):
    s = cb.NavierStokesSolver(f, ["-separable", separable])
    s.set_option("write_output", 0)
    s.set_option("use_graph", graph)
    s.initialise()
    return s


@pytest.mark.parametrize("graph", [1, 0])
@pytest.mark.parametrize("separable", ["1", "0"])
@pytest.mark.parametrize("kind", ["cavity", "mixed", "LUO", "FADLUN", "OSC_CYLINDER"])
def test_stamps(tmp_path, kind, separable, graph):
    f = case(tmp_path, kind)
    with solver(f, separable, graph) as s:
        s.stepTime(3)
        ref = s.get("u"), s.get("p")
    with solver(f, separable, graph) as s:
        s.stepTime(1)
        s.set_option("trace_solve", 1)
        s.stepTime(1)
        t = s.get("solve_trace")
        s.set_option("trace_solve", 0)
        s.stepTime(1)
        assert np.array_equal(s.get("solve_trace"), t)  # off again
        assert np.array_equal(s.get("u"), ref[0]) and np.array_equal(s.get("p"), ref[1])
    for system, half in (("velocity", t[:len(t) // 2]), ("poisson", t[len(t) // 2:])):
        ph = trace.phases(half)
        assert len(ph) >= 4, system
        assert all(0 <= us < 1e5 for _, us in ph), system
        own = separable == "1" and not (system == "velocity" and kind == "OSC_CYLINDER")
        for site, _ in ph:
            at, text = trace.site_text(site)
            assert at.startswith("separable.cu" if own else "fused_kernels.cuh")
            assert ("stamp(c);" in text) if own else text


def test_no_stamps_of_phase_by_phase_solves(tmp_path):
    with solver(case(tmp_path, "LUO"), "0", 1) as s:
        s.set_option("trace_solve", 1)
        s.stepTime(1)
        assert s.get("solve_trace")[0] > 0
        s.set_option("fused_solve", 0)
        s.set_option("trace_solve", 1)
        s.stepTime(1)
        t = s.get("solve_trace")
        assert t[0] == 0 and t[len(t) // 2] == 0
