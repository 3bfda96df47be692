"""Sweeps in two passes against the queued kernels (GPU).

Same element code, tile records and association: f, K.v, dynamic relaxation, the adjoint and
the FP32 tangents must be equal bit for bit.  Meshes at the edges of the tiles: one element, a last tile of
one element, ragged boxes, shuffled numbering (wide spans, many nodes per tile), disjoint
unions, a mesh of many granules.
"""
from __future__ import annotations

import numpy as np
import pytest
import torch

from psierra_b200 import meshgen
from psierra_b200.assembler import GPUAssembler
from psierra_b200.material import NeoHookeanField

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda")


def _shuffled(mesh, seed):
    rng = np.random.default_rng(seed)
    new = rng.permutation(mesh.n_nodes)
    nodes = np.empty_like(mesh.nodes)
    nodes[new] = mesh.nodes
    return meshgen.TetMesh(nodes, new[mesh.elements][rng.permutation(mesh.n_elements)])


def _cut(mesh, n):
    el = mesh.elements[:n]
    used, local = np.unique(el, return_inverse=True)
    return meshgen.TetMesh(mesh.nodes[used], local.reshape(el.shape))


MESHES = {
    "one element": lambda: meshgen.TetMesh(np.vstack([np.zeros(3), np.eye(3)]), np.array([[0, 1, 2, 3]])),
    "33 elements": lambda: _cut(meshgen.box_tet4(1.0, 1.0, 1.0, 2, 2, 2), 33),
    "ragged box": lambda: meshgen.box_tet4(1.0, 0.3, 0.5, 7, 3, 5),
    "shuffled box": lambda: _shuffled(meshgen.box_tet4(1.0, 1.0, 1.0, 11, 12, 13), 3),
    "uneven beams": lambda: meshgen.concat_meshes([c.mesh for c in meshgen.beam_batch(n=12, target_tets=60000, seed=3)])[0],
    "cube 34": lambda: meshgen.box_tet4(1.0, 1.0, 1.0, 34, 34, 34),
}


def _pair(mesh, precision):
    mu = np.random.default_rng(4).uniform(1e3, 5e3, mesh.n_elements)
    field = NeoHookeanField(mu, 20.0 * mu, mass_density=900.0)
    a, b = (GPUAssembler(mesh.nodes, mesh.elements, field, precision=precision) for _ in range(2))
    b.set_queue(lag=b.pattern.lag, lag_f=b.pattern.lag_f, split=True)
    way = lambda s: (s.dev["plan"].two_pass, s.dev["plan"].two_pass_k)  # noqa: E731
    assert way(a) == (1, 1) and way(b) == (0, 0)
    X = mesh.nodes
    ext = float(np.ptp(X, axis=0).max())
    u = 0.03 * (X[:, [1, 2, 0]] - X.mean(axis=0)) + 0.002 * ext * np.sin(6.0 * X / ext)
    v = np.random.default_rng(5).normal(size=3 * mesh.n_nodes)
    return a, b, torch.from_numpy(u.reshape(-1)).to(DEV), torch.from_numpy(v).to(DEV)


@pytest.mark.parametrize("precision", ["fp64", "fp32-mixed"])
@pytest.mark.parametrize("name", list(MESHES))
def test_two_pass_sweeps_equal_the_queued_kernels(name, precision):
    a, b, u, v = _pair(MESHES[name](), precision)

    def sweeps(s):
        yield "f", s.assemble(u, want_k=False)[0]
        yield "K.v", s.kv(u, v)
        yield from zip(("f of f+K", "K of f+K"), s.assemble(u))
        yield "K", s.assemble(u, want_f=False)[1]
        yield from zip(("f of effective", "effective"), s.assemble_effective(u, 0.9, 37.0, 0.02))
        yield "effective without f", s.assemble_effective(u, 0.9, 37.0, 0.02, want_f=False)[1]
        yield "mass", s.assemble(None, mass=True)[1]
        yield "linear", s.assemble(None, linear=True)[1]
        yield from zip(("X", "mu", "kappa"), s.adjoint(u, v))
        x, vel, r = torch.zeros_like(v), torch.zeros_like(v), torch.empty_like(v)
        for _ in range(3):
            s.dr_step(u, v, torch.full_like(v, 1e-6), x, vel, 0.9, 1.9, 1.0, r_out=r)
        yield from (("x", x), ("vel", vel), ("r", r))

    for (what, x), (_, y) in zip(sweeps(a), sweeps(b)):
        assert torch.equal(x, y), what
    assert a.status_counts() == (0, 0, -1, 0)


@pytest.mark.parametrize("precision", ["fp64", "fp32-mixed"])
@pytest.mark.parametrize("name", ["one element", "33 elements", "ragged box", "shuffled box"])
def test_tet10_two_pass_sweeps_equal_the_queued_kernel(name, precision):
    # tiles of 8 elements: 1, 4 x 8 + 1, ...; every sum has the same terms in the same order
    mesh = meshgen.tet4_to_tet10(MESHES[name]())
    a, b, u, v = _pair(mesh, precision)

    def sweeps(s):
        yield "f", s.assemble(u, want_k=False)[0]
        yield from zip(("f of f+K", "K of f+K"), s.assemble(u))
        yield "K", s.assemble(u, want_f=False)[1]
        yield "mass", s.assemble(None, mass=True)[1]
        yield "linear", s.assemble(None, linear=True)[1]

    for (what, x), (_, y) in zip(sweeps(a), sweeps(b)):
        assert torch.equal(x, y), what
    assert a.status_counts() == (0, 0, -1, 0)


def test_workspace_follows_the_way_the_sweeps_run():
    a, b, u, v = _pair(MESHES["cube 34"](), "fp64")
    y = a.kv(u, v).clone()
    a.set_queue(lag_f=2, ring_slack=6)
    assert torch.equal(a.kv(u, v), y)
    a.set_two_pass()
    assert torch.equal(a.kv(u, v), y)
    a.set_wait_limit(1 << 22)
    assert a.dev["plan"].two_pass == 0 and torch.equal(a.kv(u, v), y)


def test_larger_meshes_queue_their_fp32_tangent(monkeypatch):
    from psierra_b200.pattern import MeshPattern

    monkeypatch.setattr(MeshPattern, "TWO_PASS_K_ELEMENTS", 1000)
    m = meshgen.box_tet4(1.0, 1.0, 1.0, 6, 6, 6)
    mu = np.full(m.n_elements, 1e3)
    a = GPUAssembler(m.nodes, m.elements, NeoHookeanField(mu, 20.0 * mu), precision="fp32-mixed")
    assert a.dev["plan"].two_pass == 1 and a.dev["plan"].two_pass_k == 0
    u = torch.zeros(3 * m.n_nodes, dtype=torch.float64, device=DEV)
    k = a.assemble(u)[1]
    monkeypatch.undo()
    b = GPUAssembler(m.nodes, m.elements, NeoHookeanField(mu, 20.0 * mu), precision="fp32-mixed")
    assert b.dev["plan"].two_pass_k == 1 and torch.equal(b.assemble(u)[1], k)


@pytest.mark.parametrize("name", list(MESHES))
def test_fp32_point_records(name, monkeypatch):
    # f: the tile records' bits.  K: factors rounded once to FP32, about 12 roundings of terms
    # that sum to a few times the largest entry: 5e-6 of it
    from psierra_b200.pattern import MeshPattern

    monkeypatch.setattr(MeshPattern, "POINT_ELEMENTS_FP32", 0)
    a, b, u, v = _pair(MESHES[name](), "fp32-mixed")
    assert a.dev["plan"].two_pass_p == 3 and b.dev["plan"].two_pass_p == 0
    f, k = a.assemble(u)
    assert torch.equal(f, b.assemble(u)[0])
    k64 = b.assemble(u, precision="fp64")[1]
    assert float((k.double() - k64).abs().max()) <= 5e-6 * float(k64.abs().max())
    assert torch.equal(a.assemble(u, want_f=False)[1], k)
    assert torch.equal(a.assemble(u, precision="fp64")[1], k64)
    assert a.status_counts() == (0, 0, -1, 0)


def test_point_records_report_bad_elements():
    a, b, u, v = _pair(MESHES["ragged box"](), "fp64")
    x = u.view(-1, 3).clone()
    x[5] -= 40.0  # inverts elements around the node
    for s in (a, b):
        with pytest.raises(ValueError, match="inversion"):
            s.assemble(x)
    assert a.status_counts() == b.status_counts()


def test_lists_that_would_be_mostly_padding_stay_queued():
    # fans: two nodes in all 120 elements, so the 32 lists beside them would be padded to that
    n = 120
    ang = np.linspace(0.0, 6.0, n + 1)
    rim = np.stack([np.cos(ang), np.sin(ang), 0.0 * ang], axis=1)
    fan = np.vstack([[0.0, 0.0, 0.0], [0.0, 0.0, 1.0], rim])
    el = np.array([[0, 2 + i, 3 + i, 1] for i in range(n)])
    nodes = np.vstack([fan + [3.0 * j, 0.0, 0.0] for j in range(6)])
    el = np.vstack([el + j * len(fan) for j in range(6)])
    mu = np.full(len(el), 1e3)
    a = GPUAssembler(nodes, el, NeoHookeanField(mu, 20.0 * mu))
    b = GPUAssembler(nodes, el, NeoHookeanField(mu, 20.0 * mu))
    b.set_queue(lag=b.pattern.lag)
    assert a.dev["plan"].two_pass_p == 0
    u = torch.from_numpy(1e-3 * nodes[:, [1, 2, 0]].reshape(-1)).to(DEV)
    assert torch.equal(a.assemble(u)[1], b.assemble(u)[1])


def test_captured_in_a_graph():
    a, b, u, v = _pair(MESHES["ragged box"](), "fp64")
    y, k = b.kv(u, v), b.assemble(u)[1]
    out, k_out = torch.empty_like(y), torch.empty_like(k)

    def sweeps():
        a.kv(u, v, y_out=out, check_status=False)
        a.assemble(u, want_f=False, k_out=k_out, check_status=False)

    sweeps()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        sweeps()
    out.zero_()
    k_out.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, y) and torch.equal(k_out, k)
