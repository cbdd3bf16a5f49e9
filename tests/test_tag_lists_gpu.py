"""The lists of crossing segments that the tagging walks (csrc/ib_kernels.cu k_tag_lines) are
sized for the body's shape: a body of very many points needs no more room than its perimeter
and its points ask for, and a body whose points are written anew (CUIBM_F_BODY_X, _Y) and
cross more lines than that is tagged all the same.  Tags, distances, intercepts and image
points equal the oracle's, bit for bit."""
import numpy as np
import pytest

import oracle

cb = pytest.importorskip("cuibm_gb300")
from cuibm_gb300 import cases  # noqa: E402

pytestmark = pytest.mark.gpu
FIELDS = (("ghost_tags_uv", "ghostTagsUV"), ("hybrid_tags_uv", "hybridTagsUV"), ("hybrid_tags_uv2", "hybridTagsUV2"),
          ("ghost_tags_p", "ghostTagsP"), ("hybrid_tags_p", "hybridTagsP"), ("dist_node", "dist_node"),
          ("dist_between", "dist_between"), ("uv_body", "uv"))


def solver(folder, points):
    s = cb.NavierStokesSolver(cases.cylinder(folder, h=0.05, ratio=1.1, extent=3.0, core=0.6, points=points, nu=0.025,
                                             dt=0.01, nt=5))
    s.set_option("write_output", 0)
    s.initialise()
    return s


def check(s, centre_y):
    g = oracle.Grid.from_arrays(s.get("x"), s.get("dx"), s.get("xu"), s.get("y"), s.get("dy"), s.get("yv"))
    i = s.info
    T = oracle.tag_points(g, s.get("body_x"), s.get("body_y"), s.get("body_uB"), s.get("body_vB"),
                          (i.bb_start_i, i.bb_start_j, i.bb_ncx, i.bb_ncy), 0.0, centre_y)
    for mine, ref in FIELDS:
        assert np.array_equal(s.get(mine), getattr(T, ref)), mine
    return T


@pytest.mark.parametrize("points", [20000, 60000])
def test_bodies_of_many_points(tmp_path, points):
    with solver(str(tmp_path / "c"), points) as s:
        T = check(s, sum(float(v) for v in s.get("body_y")) / points)
        assert (T.ghostTagsP > 0).sum() > 20


@pytest.mark.parametrize("points", [31, 64, 200])
@pytest.mark.parametrize("reach", [0.3, 0.5])
def test_points_written_anew(tmp_path, points, reach):
    """Every segment of the new body spans it: a star, then the circle once more."""
    with solver(str(tmp_path / "c"), points) as s:
        x, y = s.get("body_x"), s.get("body_y")
        mid = sum(float(v) for v in y) / points
        first = check(s, mid)
        a = np.arange(points) * (np.pi - 2 * np.pi / points) + 0.1
        s.set("body_x", reach * np.cos(a))
        s.set("body_y", reach * np.sin(a))
        s.run("tag_points")
        star = check(s, mid)
        assert not np.array_equal(star.ghostTagsUV, first.ghostTagsUV)
        s.set("body_x", x)
        s.set("body_y", y)
        s.run("tag_points")
        check(s, mid)
