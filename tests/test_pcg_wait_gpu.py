"""The bounded wait of the one-launch CG (GPU): with a limit of one poll some block gives up at the
first meetings, the kernel ends by itself, and the caller is told so, apart from a breakdown; the
next solve in the same context has the bits of an untouched one."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from psierra_b200 import meshgen
from psierra_b200.solver import ConjugateGradientSolver

pytestmark = pytest.mark.gpu


def _system(n):
    """A tridiagonal system of condition below 3, and its right-hand side, on the device."""
    i = np.arange(n)
    cols = np.stack([i - 1, i, i + 1], axis=1)
    vals = np.where(cols == i[:, None], 4.0, -1.0)
    keep = (cols >= 0) & (cols < n)
    t = lambda a, d: torch.from_numpy(np.ascontiguousarray(a, dtype=d)).cuda()  # noqa: E731
    return (t(np.concatenate([[0], np.cumsum(keep.sum(axis=1))]), np.int32), t(cols[keep], np.int32),
            t(vals[keep], np.float64), t(np.sin(i), np.float64))


@pytest.mark.parametrize("n", [6147, 300000])
def test_a_wait_that_runs_out_is_not_a_breakdown(n):
    d = _system(n)
    solve = lambda s: (lambda x: (s.solve_device(*d, x), x))(torch.zeros_like(d[3]))  # noqa: E731
    ref, want = solve(ConjugateGradientSolver(tolerance=1e-10))
    s = ConjugateGradientSolver(tolerance=1e-10)
    s.set_wait_limit(1)
    with pytest.raises(RuntimeError, match="bounded wait"):
        solve(s)
    assert s.last.flags == 1 and not s.last.converged
    torch.cuda.synchronize()  # the launch returned: the context is usable
    s.set_wait_limit(0)
    r, x = solve(s)
    assert r.converged and r.iterations == ref.iterations and torch.equal(x, want)
    with pytest.raises(ValueError):
        s.set_wait_limit(-1)


def test_batched_newton_raises():
    from psierra_b200.batched import BatchedNewton, MeshBatch

    meshes = [meshgen.box_tet4(1.0 + 0.1 * i, 0.1, 0.1, 60, 5, 5) for i in range(2)]  # 13,176 unknowns
    mu, _, kappa = meshgen.lame_from_young_poisson(1e5, 0.3)
    fixed = [np.concatenate([3 * meshgen.nodes_on_plane(m, 0, "min") + c for c in range(3)]) for m in meshes]
    batch = MeshBatch(meshes, [mu, mu], [kappa, kappa], precision="fp64")
    solver = BatchedNewton(batch, fixed, pcg_iterations=20, per_instance_cg=False)
    solver.pcg_wait_spins = 1
    with pytest.raises(RuntimeError, match="bounded wait in the CG"):
        solver.solve(batch.concat([meshgen.traction_nodal_forces(m, 0, "max", [50.0, 0.0, -10.0]) for m in meshes]),
                     n_steps=1, nr_iterations=2)
    torch.cuda.synchronize()
