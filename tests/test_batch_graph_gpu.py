"""A batch step as one graph (CUIBM_BATCH_GRAPH=1): every instance's step is a branch of it,
whatever solver the instance takes - the separable one, whose step graph has conditional nodes,
a persistent smoothed-aggregation one, a strongly coupled body's loop - and ends with the bits of
the step launched on the instance's own stream.  An instance that needs host work between its
steps leaves the batch on its streams."""
import numpy as np
import pytest

cb = pytest.importorskip("cuibm_gb300")
from cuibm_gb300 import cases  # noqa: E402

pytestmark = pytest.mark.gpu


def cylinder(folder, method, extent=3.0, **kw):
    return cases.cylinder(folder, h=0.05, ratio=1.1, extent=extent, core=0.6, points=48, nu=0.025, dt=0.01, nt=100,
                          vel_tol=1e-10, pois_tol=1e-10, method=method, **kw)


def members(tmp_path):
    """Separable cavities (CG, by rows; BiCGSTAB in mixed precision), a one-level cavity, and each body method."""
    c = [dict(n=96), dict(n=64, precision="MIXED", pois_krylov="BICGSTAB"), dict(n=24)]
    out = [cases.cavity(str(tmp_path / ("cav%d" % k)), nu=0.01, dt=0.004, nt=100, vel_tol=1e-10, pois_tol=1e-10, **kw)
           for k, kw in enumerate(c)]
    return out + [cylinder(str(tmp_path / m), m) for m in ("LUO", "FADLUN", "OSC_CYLINDER")] + \
        [cylinder(str(tmp_path / "viv"), "LUO", 5.0, extra={"VIV": 2, "Ured": 5})]


def run(folders, graph, monkeypatch):
    monkeypatch.setenv("CUIBM_BATCH_GRAPH", "1" if graph else "0")
    with cb.Batch(folders) as b:
        for s in b.instances:
            s.set_option("write_output", 0)
        b.initialise()
        b.stepTime(3)
        b.instances[0].set_option("force_method", 0)  # (a call between steps)
        b.instances[3].set_option("solver_blocks", 20)  # another step graph
        b.stepTime(4)
        assert all(s.timeStep == 7 for s in b.instances)
        return b.graph_steps(), [(s.get("u"), s.get("p"), s.iterations()) for s in b.instances]


def test_one_graph_a_step(tmp_path, monkeypatch):
    folders = members(tmp_path)
    (n0, ref), (n1, got) = run(folders, False, monkeypatch), run(folders, True, monkeypatch)
    assert (n0, n1) == (0, 7)
    for k, (a, b) in enumerate(zip(ref, got)):
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1]) and a[2] == b[2], k


def test_host_work_between_steps_keeps_the_streams(tmp_path, monkeypatch):
    motion = {"xCoefficient": 0.05, "uCoefficient": 0.05 * 2 * np.pi, "xfrequency": 1.0, "xPhase": 0.0, "uPhase": 0.0}
    folders = members(tmp_path)[:4] + [cylinder(str(tmp_path / "moving"), "OSC_CYLINDER", motion=motion)]
    assert run(folders, True, monkeypatch)[0] == 0
