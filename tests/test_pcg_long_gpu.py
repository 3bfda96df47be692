"""One-launch CG beyond short, well-conditioned solves (GPU): a slender cantilever's tangent, whose
solve takes hundreds of iterations, in the cluster and the grid form, and solves on two streams
at once."""
from __future__ import annotations

import threading

import numpy as np
import pytest
import scipy.sparse as spsp
import torch

from psierra_b200 import meshgen
from psierra_b200.assembler import GPUAssembler
from psierra_b200.material import NeoHookeanField
from psierra_b200.solver import ConjugateGradientSolver

pytestmark = pytest.mark.gpu


def _cantilever(nx, ny):
    """The cantilever's eliminated tangent at u = 0, a tip load, and both on the device."""
    m = meshgen.box_tet4(1.0, 0.1, 0.1, nx, ny, ny)
    mu, _, kappa = meshgen.lame_from_young_poisson(1e5, 0.3)
    asm = GPUAssembler(m.nodes, m.elements, NeoHookeanField(np.full(m.n_elements, mu), np.full(m.n_elements, kappa)))
    K = asm.assemble(torch.zeros(m.n_dofs, dtype=torch.float64, device="cuda"), want_f=False)[1].cpu().numpy()
    p = asm.pattern
    free = np.ones(m.n_dofs)
    clamp = meshgen.nodes_on_plane(m, 0, "min")
    free[np.concatenate([3 * clamp + c for c in range(3)])] = 0.0
    rows = np.repeat(np.arange(m.n_dofs), np.diff(p.indptr))
    vals = K * free[rows] * free[p.indices] + (rows == p.indices) * (1.0 - free[rows])
    A = spsp.csr_matrix((vals, p.indices, p.indptr), shape=(m.n_dofs, m.n_dofs))
    b = meshgen.traction_nodal_forces(m, 0, "max", [50.0, 0.0, -10.0]) * free
    t = lambda a, d: torch.from_numpy(np.ascontiguousarray(a, dtype=d)).cuda()  # noqa: E731
    return A, b, (t(p.indptr, np.int32), t(p.indices, np.int32), t(vals, np.float64), t(b, np.float64))


def _solve(d):
    s = ConjugateGradientSolver(tolerance=1e-10, max_iterations=5000, preconditioner="block-jacobi")
    x = torch.zeros_like(d[3])
    return s.solve_device(*d, x, nodal=True), x


@pytest.mark.parametrize("nx,ny", [(40, 4), (120, 6), (160, 12)])  # 3,075, 17,787 and 81,627 unknowns
def test_long_solves_reach_their_residual(nx, ny):
    A, b, d = _cantilever(nx, ny)
    r, x = _solve(d)
    assert r.converged and r.iterations >= 200
    x = x.cpu().numpy()
    # the recurrence's residual is under 1e-10 ||b||; the true one strays from it by at most a few
    # roundings of A x per iteration, m entries per row: (m + 4) eps ||A|| ||x|| each
    m = np.diff(A.indptr).max()
    stray = r.iterations * (m + 4) * 2.0 ** -53 * np.abs(A).sum(axis=1).max() * np.linalg.norm(x)
    assert np.linalg.norm(b - A @ x) <= 1e-10 * np.linalg.norm(b) + stray
    r2, x2 = _solve(d)
    assert r2.iterations == r.iterations and np.array_equal(x2.cpu().numpy(), x)


@pytest.mark.parametrize("shapes", [((120, 6), (160, 12)), ((40, 4), (120, 6))])  # grid and grid, cluster and grid
def test_two_solves_on_two_streams(shapes):
    systems = [_cantilever(*s)[2] for s in shapes]
    want = [_solve(d) for d in systems]
    torch.cuda.synchronize()
    got = [[], []]

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(5):
                r, x = _solve(systems[i])
                got[i].append(r.iterations == want[i][0].iterations and torch.equal(x, want[i][1]))

    threads = [threading.Thread(target=work, args=(i,)) for i in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert got == [[True] * 5] * 2
