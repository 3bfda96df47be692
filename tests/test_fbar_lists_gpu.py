"""Tet4Fbar passes at the edges of their warps (GPU): one element, entry lists longer and
shorter than a warp's threshold, runs that start inside a warp, more than one block of
entries.  Against the oracle; f, K_dev + K_vol within 1e-12 of
their largest entry (FP64, the closed form against the reference's dense products)."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import tet4fbar
from psierra_b200 import meshgen
from psierra_b200.fbar import FbarAssembler
from psierra_b200.material import IsotropicElasticParameters, NeoHookean

pytestmark = pytest.mark.gpu


def _fan(n):
    """n tetrahedra around one edge: two nodes whose lists have n terms."""
    a = np.linspace(0.0, 2 * np.pi, n, endpoint=False)
    ring = np.stack([np.cos(a), np.sin(a), 0.05 * np.sin(3 * a)], axis=1)
    nodes = np.vstack([[0.0, 0.0, -0.5], [0.0, 0.0, 0.5], ring])
    k = np.arange(n)
    return meshgen.TetMesh(nodes, np.stack([0 * k, 2 + k, 2 + (k + 1) % n, 0 * k + 1], axis=1))


MESHES = {
    "one element": lambda: meshgen.TetMesh(np.vstack([np.zeros(3), np.eye(3)]), np.array([[0, 1, 2, 3]])),
    "fan of 40": lambda: _fan(40),
    "fan of 7": lambda: _fan(7),
    "box": lambda: meshgen.box_tet4(1.0, 0.7, 0.4, 5, 4, 2),
    "two boxes": lambda: meshgen.concat_meshes([meshgen.box_tet4(1.0, 1.0, 1.0, 2, 1, 1), meshgen.box_tet4(1, 1, 1, 1, 1, 1)])[0],
}


@pytest.mark.parametrize("name", list(MESHES))
def test_fbar_matches_the_oracle(name):
    m = MESHES[name]()
    p = IsotropicElasticParameters()
    p.set_from_youngs_poisson(youngs_modulus=2e3, poissons_ratio=0.49, mass_density=1000.0)
    X = m.nodes
    u = 0.05 * (X[:, [1, 2, 0]] - X.mean(axis=0)) + 0.01 * np.sin(5.0 * X)
    a = FbarAssembler(m.nodes, m.elements, NeoHookean(p))
    ud = torch.from_numpy(u.reshape(-1)).cuda()
    f, k = a.assemble(ud)
    f_ref = tet4fbar.internal_forces(m.nodes, m.elements, u, p.shear_modulus, p.bulk_modulus)
    K_ref = tet4fbar.tangent(m.nodes, m.elements, u, p.shear_modulus, p.bulk_modulus)
    assert np.abs(f.cpu().numpy() - f_ref).max() <= 1e-12 * np.abs(f_ref).max()
    D = abs(a.csr(k) - K_ref)
    assert (D.max() if D.nnz else 0.0) <= 1e-12 * abs(K_ref).max()
    f2, k2 = a.assemble(ud)
    assert torch.equal(f, f2) and torch.equal(k, k2)
    f3, _ = a.assemble(ud, want_k=False)
    assert torch.equal(f, f3)
    _, k4 = a.assemble(ud, want_f=False)
    assert torch.equal(k, k4)
