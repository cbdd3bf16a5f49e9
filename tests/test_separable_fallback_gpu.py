"""A case whose separable tables cannot be formed is set up with its other preconditioner instead
of being refused.  A time step of 1e-314 is one: the pressure operator's entries are then
denormal and the pinned cells' 1 / diagonal overflows."""
import numpy as np
import pytest

cb = pytest.importorskip("cuibm_gb300")
from cuibm_gb300 import cases  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("krylov", ["BICGSTAB", "CG"])
def test_singular_pinned_cells(tmp_path, krylov):
    f = cases.cavity(str(tmp_path / "c"), n=64, nu=0.01, dt=1e-314, nt=10, pois_krylov=krylov)
    out = []
    for flag in ("0", "-1", "1"):
        with cb.NavierStokesSolver(f, ["-separable", flag]) as s:
            s.set_option("write_output", 0)
            s.initialise()
            out.append((s.info.nx, s.get("u"), s.get("p")))
    for nx, u, p in out:
        assert nx == 64 and np.array_equal(u, out[0][1]) and np.array_equal(p, out[0][2])
