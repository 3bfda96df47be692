"""Linear and mass matrices of Tet4 (GPU), which run the queue whatever the passes of the other
sweeps: on the queue's ring, not on records of the whole mesh, with the same bits either way."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest
import torch

from psierra_b200 import _lib, meshgen
from psierra_b200.assembler import GPUAssembler
from psierra_b200.material import NeoHookeanField

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32-mixed"])
@pytest.mark.parametrize("cells", [1, 9, 40])  # one granule; a ring wider than the mesh; a ring that wraps
def test_ring_beside_two_pass_records(cells, precision):
    m = meshgen.box_tet4(1.0, 1.0, 1.0, cells, cells, cells)
    mu = np.random.default_rng(2).uniform(1e3, 2e3, m.n_elements)
    a, b = (GPUAssembler(m.nodes, m.elements, NeoHookeanField(mu, 20.0 * mu, mass_density=900.0), precision=precision)
            for _ in range(2))
    b.set_queue(lag=b.pattern.lag, lag_f=b.pattern.lag_f)
    assert (a.dev["plan"].two_pass_k, b.dev["plan"].two_pass_k) == (1, 0)
    u = torch.zeros(3 * m.n_nodes, dtype=torch.float64, device="cuda")
    for kind in ("linear", "mass"):
        ka = a.assemble(None, **{kind: True})[1]
        a.assemble(u)  # the other sweeps' records share the workspace
        assert torch.equal(ka, a.assemble(None, **{kind: True})[1])
        assert torch.equal(ka, b.assemble(None, **{kind: True})[1])


def test_records_stay_on_the_ring():
    m = meshgen.box_tet4(1.0, 1.0, 1.0, 40, 40, 40)  # 94 granules, a ring of 64
    mu = np.full(m.n_elements, 1e3)
    a, b = (GPUAssembler(m.nodes, m.elements, NeoHookeanField(mu, 20.0 * mu, mass_density=900.0), precision="fp32-mixed")
            for _ in range(2))
    b.set_queue(lag=b.pattern.lag, lag_f=b.pattern.lag_f)
    ring = b.workspace("fp32-mixed").numel()
    work = a.workspace("fp32-mixed")
    assert work.numel() > ring
    for kind in ("linear", "mass"):
        work.fill_(0xA5)
        a.assemble(None, **{kind: True})
        assert bool((work[ring:] == 0xA5).all()), kind


def test_the_workspace_covers_every_sweep():
    # 4,097 elements: two granules, so the ring of the queue is larger than the records of the mesh
    m = meshgen.box_tet4(1.0, 1.0, 1.0, 9, 9, 9)
    used, local = np.unique(m.elements[:4097], return_inverse=True)
    m = meshgen.TetMesh(m.nodes[used], local.reshape(-1, 4))
    mu = np.full(m.n_elements, 1e3)
    a = GPUAssembler(m.nodes, m.elements, NeoHookeanField(mu, 20.0 * mu, mass_density=900.0), precision="fp32-mixed")
    ring, size = ctypes.c_int64(), ctypes.c_int64()
    _lib.check(_lib.lib().psx_work_bytes(ctypes.byref(a.dev["plan"]), _lib.PSX_FP32_MIXED, ctypes.byref(ring),
                                         ctypes.byref(size)), "psx_work_bytes")
    assert ring.value == 8192 and a.workspace("fp32-mixed").numel() == size.value
    assert size.value >= 8192 // 32 * (9 * 4 + 6 * 4) * 4
    a.assemble(None, linear=True)
    a.assemble(torch.zeros(3 * m.n_nodes, dtype=torch.float64, device="cuda"))
