"""Tagging by the segments that cross each row and column (csrc/ib_kernels.cu k_tag_lines):
tags, distances, intercepts and image points equal the oracle's, bit for bit, for bodies
whose point counts fall on and beside the 32 segments a warp scans at a time, with points
on grid lines (a radius and centre on the nodes) and few points (long segments that cross
many lines)."""
import numpy as np
import pytest

import oracle

cb = pytest.importorskip("cuibm_gb300")
from cuibm_gb300 import cases  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("points,radius,h", [(8, 0.5, 0.05), (31, 0.5, 0.05), (32, 0.45, 0.05), (33, 0.5, 0.04),
                                             (64, 0.475, 0.05), (65, 0.31, 0.03), (128, 0.5, 0.025)])
def test_tags_equal_the_oracles(tmp_path, points, radius, h):
    f = cases.cylinder(str(tmp_path / "c"), h=h, ratio=1.1, extent=3.0, core=0.6, points=points, radius=radius, nu=0.025,
                       dt=0.01, nt=5)
    with cb.NavierStokesSolver(f) as s:
        s.set_option("write_output", 0)
        s.initialise()
        g = oracle.Grid.from_arrays(s.get("x"), s.get("dx"), s.get("xu"), s.get("y"), s.get("dy"), s.get("yv"))
        i = s.info
        bx, by = s.get("body_x"), s.get("body_y")
        T = oracle.tag_points(g, bx, by, s.get("body_uB"), s.get("body_vB"),
                              (i.bb_start_i, i.bb_start_j, i.bb_ncx, i.bb_ncy), 0.0,
                              sum(float(v) for v in by) / len(by))
        for mine, ref in (("ghost_tags_uv", T.ghostTagsUV), ("hybrid_tags_uv", T.hybridTagsUV),
                          ("hybrid_tags_uv2", T.hybridTagsUV2), ("ghost_tags_p", T.ghostTagsP),
                          ("hybrid_tags_p", T.hybridTagsP), ("dist_node", T.dist_node),
                          ("dist_between", T.dist_between), ("uv_body", T.uv)):
            assert np.array_equal(s.get(mine), ref), mine
