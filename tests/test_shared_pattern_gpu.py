"""Two assemblers of one pattern (GPU): a queue, a wait limit or the passes chosen through one of
them sizes the other's workspace too."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from psierra_b200 import meshgen
from psierra_b200.assembler import GPUAssembler
from psierra_b200.material import NeoHookeanField
from psierra_b200.pattern import MeshPattern

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32-mixed"])
@pytest.mark.parametrize("tet10", [False, True])
def test_workspaces_follow_the_pattern(tet10, precision):
    m = meshgen.box_tet4(1.0, 1.0, 1.0, 8, 8, 8)
    m = meshgen.tet4_to_tet10(m) if tet10 else m
    mu = np.full(m.n_elements, 1e3)
    p = MeshPattern(m.elements, m.n_nodes)
    a, b = (GPUAssembler(m.nodes, m.elements, NeoHookeanField(mu, 20.0 * mu), precision=precision, pattern=p)
            for _ in range(2))
    u = torch.from_numpy(1e-3 * np.sin(5.0 * m.nodes[:, [1, 2, 0]]).reshape(-1)).cuda()
    (f, k), f_alone = b.assemble(u), b.assemble(u, want_k=False)[0]
    for change in (lambda: a.set_wait_limit(1 << 22), lambda: a.set_wait_limit(0), lambda: a.set_queue(split=False),
                   lambda: a.set_queue(lag=2, lag_f=2), lambda: a.set_queue(lag=40, lag_f=40, ring_slack=40),
                   lambda: a.set_two_pass(k=False), a.set_two_pass, lambda: p.set_queue(lag=3, lag_f=3)):
        change()
        for s in (b, a):
            g, l = s.assemble(u)
            assert torch.equal(f, g) and torch.equal(k, l)
            assert torch.equal(s.assemble(u, want_k=False)[0], f_alone)
