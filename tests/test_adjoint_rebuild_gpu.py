"""Gradients after the forward hierarchy or the separable plan was rebuilt on the same solver.

A transposed solve is a captured graph whose nodes hold the preconditioner's device
pointers; the option sa_body_free and a moving body's steps with it off free those tables
and build others, whose host objects may get the freed ones' addresses.  The gradient after
each such sequence is that of a solver that rebuilt nothing else before it.  The two runs'
preconditioners differ, so their solves stop at different places: forward and transposed
solves to a relative residual of 1e-12 leave up to 1e-9 of a field (the embedded method's
bound for u at this tolerance), six steps of them 1e-8 of the largest component."""
import numpy as np
import pytest

cb = pytest.importorskip("cuibm_gb300")
from cuibm_gb300 import cases  # noqa: E402

pytestmark = pytest.mark.gpu
NT = 6
SNAPSHOTS = 4


def case(folder):
    """The body moves 0.1, two of its cells of 0.05, in six steps."""
    motion = {"xCoefficient": 0.4, "uCoefficient": 0.4 * 4 * np.pi, "xfrequency": 2.0, "xPhase": -np.pi / 2,
              "uPhase": -np.pi / 2}
    return cases.cylinder(folder, h=0.05, ratio=1.1, extent=4.0, core=1.2, points=48, nu=0.05, dt=0.01, nt=3 * NT,
                          method="OSC_CYLINDER", quiescent=True, motion=motion, vel_tol=1e-12, pois_tol=1e-12)


def solver(folder, *args):
    s = cb.NavierStokesSolver(folder, list(args))
    s.set_option("write_output", 0)
    s.set_option("adjoint_tolerance", 1e-12)
    s.initialise()
    return s


def gradient(s, n):
    return s.adjoint(n, 2.0 / NT, snapshots=SNAPSHOTS)[1]


# what is done to the solver before its last gradient, over NT steps: an option, or a gradient
SEQUENCES = {"rebuilt by the longer forward sweep": [("free", 0), 3],
             "the plan freed and built again": [NT, ("free", 0), ("free", 1)],
             "the plan freed": [NT, ("free", 0)]}


@pytest.mark.parametrize("name,separable", [(n, "-1") for n in SEQUENCES] + [("the plan freed and built again", "0")])
def test_gradients_after_a_rebuild(tmp_path, name, separable):
    sequence = SEQUENCES[name]
    f = case(str(tmp_path / "c"))
    body_free = [a[1] for a in sequence if isinstance(a, tuple)][-1]
    with solver(f, "-separable", separable) as s:
        if not body_free:
            s.set_option("sa_body_free", 0)
        ref = gradient(s, NT)
        if not body_free:
            assert s.get_info().sa_rebuilds > 0
    with solver(f, "-separable", separable) as s:
        for act in sequence:
            if isinstance(act, tuple):
                s.set_option("sa_body_free", act[1])
            else:
                gradient(s, act)
        got = gradient(s, NT)
    assert np.all(np.isfinite(got)) and np.max(np.abs(got)) > 0
    assert np.max(np.abs(got - ref)) <= 1e-8 * np.max(np.abs(ref))
