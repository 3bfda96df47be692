"""ECSW evaluation at the edges of its tiles (GPU): one element, one mode, modes around the
32-wide result tiles, more runs than elements.  Against the reference formula with the
oracle's batched element function; FP64, 1e-12 of the largest entry (the summation order
differs, sums of up to 12 n terms of one sign pattern)."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import vectorized
from psierra_b200 import meshgen
from psierra_b200.ecsw import ECSWEvaluator
from psierra_b200.material import NeoHookeanField

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,r", [(1, 1), (1, 33), (3, 31), (5, 32), (130, 33), (700, 64), (257, 100)])
def test_ecsw_tiles(n, r):
    m = meshgen.box_tet4(1.0, 0.4, 0.3, 9, 5, 5)
    rng = np.random.default_rng(100 * n + r)
    Phi, _ = np.linalg.qr(rng.normal(size=(m.n_dofs, r)))
    idx = np.sort(rng.choice(m.n_elements, size=n, replace=False))
    w = rng.uniform(0.5, 3.0, size=n)
    u_r = 0.02 * rng.normal(size=r)
    mu = 3e3 * np.exp(0.2 * rng.normal(size=m.n_elements))
    kappa = 30.0 * mu
    ev = ECSWEvaluator(m.nodes, m.elements, NeoHookeanField(mu, kappa), Phi, idx, w)
    f, K = ev.evaluate_forces_and_stiffness(u_r)
    u = Phi @ u_r
    k, fe = vectorized.element_force_and_tangent(m.nodes, m.elements[idx], u.reshape(-1, 3), mu[idx], kappa[idx])
    P = Phi[(3 * m.elements[idx][:, :, None] + np.arange(3)).reshape(n, 12)]
    Kr = np.einsum("eai,eab,ebj->ij", P, w[:, None, None] * k.reshape(n, 12, 12), P, optimize=True)
    fr = np.einsum("eai,ea->i", P, w[:, None] * fe.reshape(n, 12))
    assert np.abs(K - 0.5 * (Kr + Kr.T)).max() <= 1e-12 * np.abs(Kr).max()
    assert np.abs(f - fr).max() <= 1e-11 * np.abs(fr).max()  # the oracle's f rounds at 1e-12
    assert np.array_equal(K, K.T)
    f2, K2 = ev.evaluate_forces_and_stiffness(u_r)
    assert np.array_equal(f, f2) and np.array_equal(K, K2)
