"""Which way the sweeps run (CPU): two passes by default, the queued kernels once a shape
of their queue is chosen or its waits are limited, and for tangents of large meshes."""
from __future__ import annotations

from psierra_b200 import meshgen
from psierra_b200.pattern import MeshPattern


def test_choices():
    m = meshgen.box_tet4(1.0, 1.0, 1.0, 3, 3, 3)
    p = MeshPattern(m.elements, m.n_nodes)
    st = p.device("cpu")["plan"]
    way = lambda: (st.two_pass, st.two_pass_k)  # noqa: E731
    assert way() == (1, 1)
    p.set_wait_limit(100)
    assert way() == (0, 0)
    p.set_wait_limit(0)
    p.set_queue(ring_slack=12)  # no lag, no kernel: nothing chosen
    assert way() == (1, 1)
    p.set_queue(lag_f=3)
    assert way() == (0, 1)
    p.set_queue(lag=3)
    assert way() == (0, 0)
    p.set_two_pass(k=False)
    assert way() == (1, 0)
    p.set_two_pass()
    assert way() == (1, 1)
    p.set_queue(split=False)
    assert way() == (1, 0)
    p.TWO_PASS_K_ELEMENTS = m.n_elements - 1
    p.set_two_pass()
    assert way() == (1, 0)
    t10 = meshgen.tet4_to_tet10(m)
    p = MeshPattern(t10.elements, t10.n_nodes)
    st = p.device("cpu")["plan"]
    assert way() == (1, 1)
    p.set_queue(lag=3)
    assert way() == (1, 0)
    p.set_queue(lag_f=3)
    assert way() == (0, 0)
