"""CG in one launch (GPU) at the edges of its forms: one row, systems smaller than the
cluster's blocks, the last rows of the cluster form and the first of the grid form, ragged
shares, systems past the shared memory (three launches per iteration), every preconditioner
and value type, node-blocked or not.

The systems are diagonally dominant (condition below 10), so an iterate with a recurrence
residual under rtol = 1e-10 has a true residual within rounding of it: ||b - A x|| <= 1.01e-10
||b||, and CG needs no more than 60 iterations.
"""
from __future__ import annotations

import numpy as np
import pytest
import scipy.sparse as spsp
import torch

from psierra_b200.solver import ConjugateGradientSolver

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda")


def _system(n, nodal, seed=0):
    """Random symmetric pattern over nodes (3 x 3 blocks, nodal) or rows, made dominant."""
    rng = np.random.default_rng(seed)
    units = n // 3 if nodal else n
    per = 3 if nodal else 1
    i = np.repeat(np.arange(units), 4)
    j = np.clip(i + rng.integers(-40, 41, i.size), 0, units - 1)
    i, j = np.concatenate([i, j, np.arange(units)]), np.concatenate([j, i, np.arange(units)])
    blk = rng.uniform(-1.0, 1.0, (i.size, per, per))
    rows = (per * i[:, None, None] + np.arange(per)[:, None]) + 0 * blk.astype(int)
    cols = (per * j[:, None, None] + np.arange(per)[None, :]) + 0 * blk.astype(int)
    A = spsp.coo_matrix((blk.ravel(), (rows.ravel(), cols.ravel())), shape=(n, n)).tocsr()
    pattern = A.copy()
    pattern.data[:] = 0.0
    A = 0.5 * (A + A.T)
    A = (A + spsp.diags(2.0 * np.asarray(np.abs(A).sum(axis=1)).ravel() + 1.0) + pattern).tocsr()
    A.sort_indices()
    return A, rng.normal(size=n)


def _solve(A, b, precond, nodal, dtype=np.float64, **kw):
    s = ConjugateGradientSolver(tolerance=1e-10, max_iterations=kw.pop("maxiter", 500), preconditioner=precond)
    t = lambda a, d: torch.from_numpy(np.ascontiguousarray(a, dtype=d)).to(DEV)  # noqa: E731
    x = torch.zeros(len(b), dtype=torch.float64, device=DEV) if "x0" not in kw else t(kw["x0"], np.float64)
    r = s.solve_device(t(A.indptr, np.int32), t(A.indices, np.int32), t(A.data, dtype), t(b, np.float64), x, nodal=nodal)
    return x.cpu().numpy(), r


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("nodal,precond", [(True, "block-jacobi"), (True, "jacobi"), (True, None), (False, "block-jacobi"),
                                           (False, "jacobi"), (False, None)])
@pytest.mark.parametrize("n", [3, 27, 99, 6144, 6147, 60000])
def test_forms(n, nodal, precond, dtype):
    A, b = _system(n, nodal, seed=n)
    if dtype == np.float32:
        A.data = A.data.astype(np.float32).astype(np.float64)
        A = (0.5 * (A + A.T)).tocsr()
        A.sort_indices()
        A.data = A.data.astype(np.float32).astype(np.float64)
    x, r = _solve(A, b, precond, nodal, dtype)
    assert r.converged and r.iterations <= 60
    assert np.linalg.norm(b - A @ x) <= 1.01e-10 * np.linalg.norm(b)
    y, q = _solve(A, b, precond, nodal, dtype)
    assert np.array_equal(x, y) and q.iterations == r.iterations  # reproducible


@pytest.mark.parametrize("n,nodal,precond", [(1, False, "jacobi"), (2, False, "jacobi"), (5000, False, "jacobi"),
                                             (900000, False, "jacobi"), (600000, True, "block-jacobi")])
def test_row_forms_and_systems_past_the_shared_memory(n, nodal, precond):
    A, b = _system(n, nodal, seed=1)
    x, r = _solve(A, b, precond, nodal)
    assert r.converged and np.linalg.norm(b - A @ x) <= 1.01e-10 * np.linalg.norm(b)


@pytest.mark.parametrize("n", [300, 30000])
def test_status_of_zero_load_limits_and_starts(n):
    A, b = _system(n, True, seed=2)
    x, r = _solve(A, 0.0 * b, "block-jacobi", True)
    assert r.converged and r.iterations == 0 and not x.any()
    _, r = _solve(A, b, "block-jacobi", True, maxiter=3)
    assert r.flags == 2 and r.iterations == 3
    _, r = _solve(A, b, "block-jacobi", True, maxiter=0)
    assert r.flags == 4 and r.iterations == 0
    x, full = _solve(A, b, "block-jacobi", True)
    y, r = _solve(A, b, "block-jacobi", True, x0=x)
    assert r.converged and r.iterations <= 1
    z = b.copy()
    z[7] = np.nan
    _, r = _solve(A, z, "block-jacobi", True)
    assert not r.converged


@pytest.mark.parametrize("n", [300, 30000])
def test_enqueued_in_a_graph(n):
    from psierra_b200 import _lib

    A, b = _system(n, True, seed=2)
    want, r = _solve(A, b, "block-jacobi", True)
    t = lambda a, d: torch.from_numpy(np.ascontiguousarray(a, dtype=d)).to(DEV)  # noqa: E731
    ip, ix, v, bd = t(A.indptr, np.int32), t(A.indices, np.int32), t(A.data, np.float64), t(b, np.float64)
    x, st = torch.zeros(n, dtype=torch.float64, device=DEV), torch.zeros(8, dtype=torch.int32, device=DEV)
    precond = _lib.PSX_PRECOND_BJACOBI | _lib.PSX_PCG_NODAL
    work = ConjugateGradientSolver(preconditioner="block-jacobi")._workspace(n, precond)

    def solve():
        x.zero_()
        _lib.check(_lib.lib().psx_pcg_enqueue(n, ip.data_ptr(), ix.data_ptr(), v.data_ptr(), _lib.PSX_FP64, bd.data_ptr(),
                                              x.data_ptr(), 1e-10, 0.0, 500, precond, work.data_ptr(), work.numel(),
                                              st.data_ptr(), _lib.current_stream()), "psx_pcg_enqueue")

    solve()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        solve()
    for _ in range(2):
        x.fill_(7.0)
        g.replay()
        torch.cuda.synchronize()
        assert np.array_equal(x.cpu().numpy(), want) and int(st[4]) == r.iterations and int(st[5]) == 0
