"""FP32 tangents from point records (GPU) below the size where they are the default: the package's
bar of 1e-6 of K's norm against the FP64 sweep, and the extreme element states (det F 0.35 to 2.5,
nu to 0.4999, strains of 1e-7) at the bars that the other FP32 kernels are held to there."""
from __future__ import annotations

import pytest

from conftest import block_diagonal_blocks, disjoint_mesh, golden, rel_max
from psierra_b200.element import Tet4TotalLagrangian
from psierra_b200.material import NeoHookeanField
from psierra_b200.pattern import MeshPattern
from test_two_pass_gpu import MESHES, _pair

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def all_sizes(monkeypatch):
    monkeypatch.setattr(MeshPattern, "POINT_ELEMENTS_FP32", 0)


@pytest.mark.parametrize("name", list(MESHES))
def test_norm_error(name):
    a, _, u, _ = _pair(MESHES[name](), "fp32-mixed")
    assert a.dev["plan"].two_pass_p == 3
    k64 = a.assemble(u, precision="fp64")[1]
    assert float((a.assemble(u)[1].double() - k64).norm()) <= 1e-6 * float(k64.norm())


def test_extreme_states():
    g = golden("element_extreme_tet4")
    n = len(g["X"])
    el = Tet4TotalLagrangian(NeoHookeanField(g["mu"], g["kappa"]), precision="fp32-mixed")
    f, K = el.assemble_force_and_tangent(disjoint_mesh(g["X"]), g["u"].reshape(-1, 3))
    kb, fb = block_diagonal_blocks(K, n, 12), f.reshape(n, 12)
    for i in range(n):
        assert rel_max(kb[i], g["k"][i]) < 2e-6, (i, rel_max(kb[i], g["k"][i]))
        assert rel_max(fb[i], g["f"][i]) < (2e-7 if i % 4 == 3 else 1e-11), (i, rel_max(fb[i], g["f"][i]))
