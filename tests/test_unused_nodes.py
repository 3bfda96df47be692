"""Meshes with nodes that no element has: first, last, scattered and in long runs.

The plan has no pairs for them (CPU).  Every sweep must give the used nodes and the CSR values the
bits it gives the same mesh without them, and the unused nodes f = 0 (GPU): elements, relative
node order and so every sum are the same.
"""
from __future__ import annotations

import numpy as np
import pytest
import torch

from psierra_b200 import meshgen
from psierra_b200.material import IsotropicElasticParameters, NeoHookean
from psierra_b200.pattern import MeshPattern

GAPS = {  # unused nodes before these nodes
    "first": [0], "last three": [480, 480, 480], "scattered": list(range(0, 480, 3)) + [480] * 40,
    "run of 500": [200] * 500,
}


def _meshes(gaps, tet10=False):
    m = meshgen.box_tet4(1.0, 0.8, 0.5, 9, 7, 5)  # 480 nodes
    m = meshgen.tet4_to_tet10(m) if tet10 else m
    g = np.sort(np.array(gaps))
    new = np.arange(m.n_nodes) + np.searchsorted(g, np.arange(m.n_nodes), side="right")
    nodes = np.full((m.n_nodes + g.size, 3), 0.123)
    nodes[new] = m.nodes
    return m, meshgen.TetMesh(nodes, new[m.elements]), new


@pytest.mark.parametrize("tet10", [False, True])
@pytest.mark.parametrize("name", list(GAPS))
def test_plan(name, tet10):
    m, wide, new = _meshes(GAPS[name], tet10)
    a, b = MeshPattern(m.elements, m.n_nodes), MeshPattern(wide.elements, wide.n_nodes)
    # counted before anything is filled
    el = m.elements
    i, j = (el[:, :, None] + 0 * el[:, None, :]).ravel(), (el[:, None, :] + 0 * el[:, :, None]).ravel()
    pairs = np.unique((i * m.n_nodes + j)[i < j]).size
    from psierra_b200 import _lib

    n, s = np.zeros(1, dtype=np.int64), np.zeros(1, dtype=np.int64)
    _lib.check(_lib.lib().psx_plan_count(_lib.ptr(b.conn), b.n_elements, b.npe, b.n_nodes, _lib.ptr(b.nbr_ptr), _lib.ptr(n),
                                         _lib.ptr(s)), "psx_plan_count")
    assert int(n[0]) == pairs
    ha, hb = a.plan_host(), b.plan_host()
    for k in ("pair_info", "pair_ptr", "pair_src", "node_src"):
        assert np.array_equal(ha[k], hb[k]), k
    ia, ib = ha["node_info"].reshape(-1, 4), hb["node_info"].reshape(-1, 4)
    used = ib[:, 1] > 0
    assert used.sum() == m.n_nodes and np.array_equal(ib[used][:, 2], new[ia[:, 2]])
    assert np.array_equal(np.diff(hb["node_ptr"])[used], np.diff(ha["node_ptr"])) and not np.diff(hb["node_ptr"])[~used].any()


def _material():
    p = IsotropicElasticParameters()
    p.set_from_youngs_poisson(youngs_modulus=3e3, poissons_ratio=0.45, mass_density=1000.0)
    return NeoHookean(p)


def _u(m, wide, new):
    u = 0.05 * np.sin(5.0 * m.nodes[:, [1, 2, 0]])
    w = np.zeros((wide.n_nodes, 3))
    w[new] = u
    t = lambda x: torch.from_numpy(x.reshape(-1)).cuda()  # noqa: E731
    return t(u), t(w)


def _same_nodes(f, g, new):
    g = g.view(-1, 3).cpu().numpy()
    rest = np.delete(g, new, axis=0)
    return np.array_equal(f.view(-1, 3).cpu().numpy(), g[new]) and not rest.any()


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "fp32-mixed"])
@pytest.mark.parametrize("name", list(GAPS))
def test_sweeps(name, precision, monkeypatch):
    from psierra_b200.assembler import GPUAssembler

    for tet10, points in ((False, False), (False, True), (True, False)):
        m, wide, new = _meshes(GAPS[name], tet10)
        if points:
            monkeypatch.setattr(MeshPattern, "POINT_ELEMENTS_FP32", 0)
        a, b = (GPUAssembler(x.nodes, x.elements, _material(), precision=precision) for x in (m, wide))
        u, w = _u(m, wide, new)
        for queued in (False, True):
            if queued:
                b.set_queue(lag=b.pattern.lag, lag_f=b.pattern.lag_f)
                a.set_queue(lag=a.pattern.lag, lag_f=a.pattern.lag_f)
            (fa, ka), (fb, kb) = a.assemble(u), b.assemble(w)
            assert torch.equal(ka, kb) and _same_nodes(fa, fb, new)
            assert torch.equal(a.assemble(None, mass=True)[1], b.assemble(None, mass=True)[1])
            assert _same_nodes(a.assemble(u, want_k=False)[0], b.assemble(w, want_k=False)[0], new)
            if not tet10:
                assert _same_nodes(a.kv(u, u), b.kv(w, w), new)


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(GAPS))
def test_fbar(name):
    from psierra_b200.fbar import FbarAssembler

    m, wide, new = _meshes(GAPS[name])
    a, b = (FbarAssembler(x.nodes, x.elements, _material()) for x in (m, wide))
    u, w = _u(m, wide, new)
    (fa, ka), (fb, kb) = a.assemble(u), b.assemble(w)
    assert torch.isfinite(kb).all() and _same_nodes(fa, fb, new)
    # entries that start elsewhere in their warp are summed as before: per entry, in a fixed order
    assert torch.equal(ka, kb)
