"""The benchmark names the kernels that a plan's FP32 f+K sweep runs (CPU), and scales captured
traffic only for the kernels that were captured."""
from __future__ import annotations

import os
import sys

import pytest

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))

import bench  # noqa: E402
from psierra_b200 import meshgen  # noqa: E402
from psierra_b200.pattern import MeshPattern  # noqa: E402


@pytest.mark.parametrize("points,queued,split,name", [
    (3, False, True, "tet4_points_kernel"), (1, False, True, "tet4_tiles_kernel"), (0, True, True, "tet4_split_kernel"),
    (0, True, False, "tet4_persistent_kernel")])
def test_kernel_of_the_plan(points, queued, split, name):
    m = meshgen.box_tet4(1.0, 1.0, 1.0, 2, 2, 2)
    p = MeshPattern(m.elements, m.n_nodes)
    plan = p.device("cpu")["plan"]
    if queued:
        p.set_queue(lag=8)
    plan.two_pass_p = points  # 3 above POINT_ELEMENTS_FP32 elements, 1 up to there
    kernel, captured = bench.fk_sweep(plan, split)
    assert kernel.startswith(name) and captured == (name == "tet4_points_kernel")
