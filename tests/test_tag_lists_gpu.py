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


@pytest.mark.parametrize("columns,wide", [(12000, False), (12600, True)])
def test_boxes_wider_than_shared_memory_holds(tmp_path, columns, wide):
    """A thin body across a box of about `columns` columns (rows of up to 12287 nodes are walked in
    shared memory, longer ones in place)."""
    h = 1.0 / 64
    a = columns * h / 4  # the box is twice the body
    t = np.arange(256) * 2 * np.pi / 256
    dirs = tmp_path / "c" / "bodyFiles"
    dirs.mkdir(parents=True)
    (dirs / "thin").write_text("256\n" + "\n".join("%r %r" % (float(a * np.cos(v)), float(0.1 * np.sin(v)))
                                                  for v in t) + "\n")
    sim = {"type": "simulation", "dt": 0.001, "nt": 5, "nsave": 5, "SolverType": "LUO",
           "linearSolvers": cases.solvers("DIAGONAL", 1e-5, "DIAGONAL", 1e-5, vel_krylov="BICGSTAB",
                                          pois_krylov="BICGSTAB")}
    flow = [{"type": "flow", "nu": 0.01, "initialVelocity": [1.0, 0.0],
             "boundaryConditions": cases.bcs((1, 0), (1, 0), (1, 0), (1, 0), xp_type="CONVECTIVE")}]
    half = 2 * a + 20 * h
    f = cases.write_case(str(tmp_path / "c"), [sim], flow,
                         [cases.axis("x", -half, h, [(half, 1.0)]), cases.axis("y", -0.5, h, [(0.5, 1.0)])],
                         [{"type": "points", "pointsFile": "thin"}])
    with cb.NavierStokesSolver(f) as s:
        s.set_option("write_output", 0)
        s.initialise()
        assert (s.info.bb_ncx + 1 > 12288) == wide
        T = check(s, sum(float(v) for v in s.get("body_y")) / 256)
        assert (T.ghostTagsP > 0).sum() > 1000 and (T.ghostTagsP == 0).sum() > 1000
