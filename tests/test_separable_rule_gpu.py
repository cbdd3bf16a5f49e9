"""cuibm_separable reports the rule's choice (the bench labels its solves by it)."""
import pytest

cb = pytest.importorskip("cuibm_gb300")
from cuibm_gb300 import cases  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flag,expected", [("-1", (False, True)), ("0", (False, False)), ("1", (True, True))])
def test_choice_is_reported(tmp_path, flag, expected):
    f = cases.cylinder(str(tmp_path / "c"), h=0.05, ratio=1.1, extent=3.0, core=0.6, points=48, nu=0.025, dt=0.01, nt=5)
    with cb.NavierStokesSolver(f, ["-separable", flag]) as s:
        assert (s.separable(1), s.separable(2)) == expected and not s.separable(3)
