"""Blocks per SM chosen alone (CPU): a limit on the launch holds for every sweep, so they all run
their queues; tuning one kind of sweep leaves the other kind's way as it was."""
from __future__ import annotations

import types

import pytest

from psierra_b200 import autotune, meshgen
from psierra_b200.pattern import MeshPattern


@pytest.fixture(params=[False, True], ids=["tet4", "tet10"])
def plan(request):
    m = meshgen.box_tet4(1.0, 1.0, 1.0, 3, 3, 3)
    m = meshgen.tet4_to_tet10(m) if request.param else m
    p = MeshPattern(m.elements, m.n_nodes)
    st = p.device("cpu")["plan"]
    return p, lambda: (st.two_pass, st.two_pass_k, st.blocks_per_sm)


def test_blocks_per_sm_selects_the_queues(plan):
    p, way = plan
    p.set_queue(blocks_per_sm=0)  # the default launch
    assert way() == (1, 1, 0)
    p.set_queue(blocks_per_sm=1)
    assert way() == (0, 0, 1) and p.point_precisions == 0
    p.set_queue(blocks_per_sm=0)
    assert way() == (0, 0, 0)
    p.set_two_pass()
    assert way() == (1, 1, 0)
    # before the plan is on a device
    q = MeshPattern(p.conn, p.n_nodes)
    q.set_queue(blocks_per_sm=2)
    st = q.device("cpu")["plan"]
    assert (st.two_pass, st.two_pass_k, st.blocks_per_sm) == (0, 0, 2)


def test_tuning_one_kind_of_sweep_keeps_the_other(plan):
    p, way = plan
    asm = types.SimpleNamespace(pattern=p, set_queue=p.set_queue, set_two_pass=p.set_two_pass)
    autotune._apply(asm, True, 8, 2, 6, None)
    assert way() == (1, 0, 2)
    p.set_two_pass()
    autotune._apply(asm, False, 8, 2, 6)
    assert way() == (0, 1, 2)
    autotune._apply(asm, True, 8, 2, 6, None)
    assert way() == (0, 0, 2)
