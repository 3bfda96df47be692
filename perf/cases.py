"""What a user of this framework has it do, as cases that can be timed.

Each case is one call (or one short sequence of calls) through the public entry points, on
inputs made from a seed: a mesh whose nodes are moved a little off their grid, a smooth
displacement with some noise, moduli where the call takes one per element.  The meshes are
the generators' boxes (cantilevers, cubes) and the clipped ellipsoid, from a few hundred
elements (one small specimen, where launches and latency count) to the 3,072,000 elements
of the 80^3 cube.

``exact`` evaluates the same quantities in float64 with plain torch: closed-form
NeoHookean force and tangent, sums over node pairs, plain conjugate gradients.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from psierra_b200 import meshgen
from psierra_b200.adjoint import internal_force
from psierra_b200.assembler import GPUAssembler
from psierra_b200.ecsw import ECSWEvaluator
from psierra_b200.fbar import FbarAssembler
from psierra_b200.material import IsotropicElasticParameters, NeoHookean, NeoHookeanField
from psierra_b200.newton import DeviceNewton
from psierra_b200.solver import ConjugateGradientSolver

KINDS = ("f_k", "f", "kv", "effective", "adjoint", "tet10", "pcg", "newton", "fbar", "ecsw")


def _case(name, kind, shape, nx, ny=0, nz=0, precision="fp64", field=False, r=0, n=0):
    """``shape``: "beam" (long box), "cube" (unit box) of nx x ny x nz cells, or
    "ellipsoid" (80 x 60 x 70 mm semi-axes, nx cells along the longest one).  ``field``:
    moduli per element.  ``r``, ``n``: modes and sampled elements of the reduced model."""
    return {"name": name, "kind": kind, "shape": shape, "nx": nx, "ny": ny, "nz": nz, "precision": precision,
            "field": field, "r": r, "n": n}


def listed():
    return [
        # one Newton iteration's sweep of a small cantilever: launches and latency count
        _case("beam_f_k_fp64", "f_k", "beam", 40, 4, 4),
        # the same sweep at the size the headline metric is quoted on
        _case("cube80_f_k_mixed", "f_k", "cube", 80, 80, 80, "fp32-mixed"),
        # one million elements of an organ-like body with a modulus per element, FP64
        _case("ellipsoid_f_k_fp64", "f_k", "ellipsoid", 80, field=True),
        # f alone, as every trial of a line search asks for it; odd cell counts
        _case("cube_f_fp64", "f", "cube", 37, 41, 43),
        # matrix-free K_T(u) v, one product of a matrix-free iteration
        _case("cube56_kv_mixed", "kv", "cube", 56, 56, 56, "fp32-mixed"),
        # effective tangent of a generalized-alpha step of a large beam
        _case("beam_effective_mixed", "effective", "beam", 120, 10, 10, "fp32-mixed"),
        # f and its gradients (coordinates, displacement, moduli): parameter identification
        _case("ellipsoid_adjoint_fp64", "adjoint", "ellipsoid", 40, field=True),
        # quadratic elements, the sweep of a compression test's Newton iteration
        _case("cube30_tet10_fp64", "tet10", "cube", 30, 30, 30),
        # one linear step of Newton: block-Jacobi conjugate gradients on the FP32 tangent
        _case("cube40_pcg_mixed", "pcg", "cube", 40, 40, 40, "fp32-mixed"),
        # a whole static solve of a cantilever
        _case("beam_newton_mixed", "newton", "beam", 30, 5, 5, "fp32-mixed"),
        # nodal F-bar for a nearly incompressible body
        _case("cube30_fbar_fp64", "fbar", "cube", 30, 30, 30),
        # hyper-reduced evaluation of an online simulation
        _case("ecsw_fp64", "ecsw", "beam", 60, 8, 8, r=30, n=1500),
    ]


def draw(rng):
    kind = rng.choice(KINDS)
    log = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))  # noqa: E731
    precision = rng.choice(("fp64", "fp32-mixed"))
    field = rng.random() < 0.4
    if kind == "ecsw":
        return _case(None, kind, "beam", log(30, 90), log(4, 10), log(4, 10), "fp64", field, r=log(8, 60), n=log(100, 1900)) \
            | {"name": ""}
    # target element counts of each kind, the upper ends well inside the listed ones
    lo, hi = {"tet10": (300, 160_000), "fbar": (300, 160_000), "newton": (400, 6_000), "pcg": (2_000, 380_000),
              "adjoint": (500, 500_000)}.get(kind, (300, 2_500_000))
    e = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    if kind in ("newton",):
        shape = "beam"
    elif kind in ("pcg", "fbar", "tet10"):
        shape = "cube"
    else:
        shape = rng.choice(("beam", "cube", "ellipsoid"))
    if shape == "ellipsoid":
        # 6 tetrahedra per cell, pi/6 of the box of 1 x 3/4 x 7/8 of nx^3 cells
        nx = max(8, int(round((e / (6 * 0.42)) ** (1 / 3))))
        c = _case("", kind, shape, min(nx, 96), precision=precision, field=field)
    else:
        c3 = (e / 6) ** (1 / 3)
        if shape == "beam":
            ny, nz = (max(2, int(round(c3 * rng.uniform(0.3, 0.5)))) for _ in range(2))
            nx = max(6, int(round(e / 6 / (ny * nz))))
            if kind == "newton":
                # stocky cantilevers (the line search stalls on slender ones)
                ny, nz = min(ny, 6), min(nz, 6)
                nx = min(nx, 6 * min(ny, nz))
        else:
            nx, ny = (max(2, int(round(c3 * rng.uniform(0.8, 1.25)))) for _ in range(2))
            nz = max(2, int(round(e / 6 / (nx * ny))))
        c = _case("", kind, shape, nx, ny, nz, precision, field)
    if kind in ("fbar", "adjoint"):
        c["precision"] = "fp64"
    if kind == "adjoint":
        c["field"] = True
    if kind in ("fbar", "pcg"):
        c["field"] = False
    return c


# ---------------------------------------------------------------------------- inputs
def _mesh(case):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if case["shape"] == "ellipsoid":
        return meshgen.ellipsoid_tet4(0.08, 0.06, 0.07, 0.16 / nx), 0.16 / nx
    if case["shape"] == "beam":
        m = meshgen.box_tet4(0.02 * nx, 0.02 * ny, 0.02 * nz, nx, ny, nz)
        return m, 0.02
    return meshgen.box_tet4(1.0, 1.0, 1.0, nx, ny, nz), 1.0 / max(nx, ny, nz)


def _inputs(case, seed):
    """Mesh (nodes off their grid by up to 6% of a cell), displacement (smooth, strains of a
    few percent, plus noise) and moduli; numpy arrays."""
    rng = np.random.default_rng([7, seed])
    m, h = _mesh(case)
    lo, hi = m.nodes.min(axis=0), m.nodes.max(axis=0)
    inner = ((m.nodes > lo + 1e-9) & (m.nodes < hi - 1e-9))  # boxes keep their faces
    m = meshgen.TetMesh(m.nodes + rng.uniform(-0.06, 0.06, m.nodes.shape) * h * inner, m.elements)
    if case["kind"] == "tet10":
        m = meshgen.tet4_to_tet10(m)
    ext = float((hi - lo).max())
    s = (m.nodes - lo) / ext
    a = 0.03 * ext * rng.uniform(0.5, 1.5, 3)
    ph = rng.uniform(0.0, 6.28, 3)
    u = np.stack([a[i] * np.sin(2.1 * s[:, (i + 1) % 3] + ph[i]) * (0.4 + s[:, (i + 2) % 3]) for i in range(3)], axis=1)
    u += rng.uniform(-0.002, 0.002, u.shape) * h
    E, nu = rng.uniform(2e3, 4e3), rng.uniform(0.40, 0.46)
    if case["kind"] == "fbar":
        nu = rng.uniform(0.48, 0.495)
    mu, kappa = E / (2 * (1 + nu)), E / (3 * (1 - 2 * nu))
    if case["field"]:
        mu_e = mu * np.exp(0.3 * rng.normal(size=m.n_elements))
        mu, kappa = mu_e, kappa / mu * mu_e
    return m, u, mu, kappa, rng


def _material(mu, kappa):
    if np.ndim(mu):
        return NeoHookeanField(mu, kappa)
    p = IsotropicElasticParameters()
    p.set_from_bulk_shear(kappa, mu, 1000.0)
    return NeoHookean(p)


def _dev(a, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dtype, device=_device())


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _effective_coefficients():
    """c_t, c_m, c_0 of generalized-alpha with rho_inf = 0.8, dt = 1e-2, Rayleigh damping 0.5 / 1e-4."""
    rho, dt, alpha_r, beta_r = 0.8, 1e-2, 0.5, 1e-4
    am, af = (2 * rho - 1) / (rho + 1), rho / (rho + 1)
    gamma = 0.5 - am + af
    beta = 0.25 * (1 - am + af) ** 2
    a0, a1 = 1 / (beta * dt * dt), gamma / (beta * dt)
    return 1 - af, (1 - am) * a0 + (1 - af) * a1 * alpha_r, (1 - af) * a1 * beta_r


def _linear_system(case, m, u, mu, kappa, rng):
    """Tangent of the cube clamped at z = 0 as node-blocked CSR (float32 values for the mixed
    precision) and a load on the free DOFs, by plain torch, so that the system itself does not
    depend on the code that solves it."""
    _, K, indptr, indices, _ = _tet4_assemble(m, u, mu, kappa)
    n = m.n_dofs
    fixed = torch.zeros(n, dtype=torch.bool, device=K.device)
    fixed[_dev(3 * np.flatnonzero(m.nodes[:, 2] < 1e-9), torch.int64)[:, None] + torch.arange(3, device=K.device)] = True
    rows = torch.repeat_interleave(torch.arange(n, device=K.device), indptr.diff())
    K = torch.where(fixed[rows] | fixed[indices], (rows == indices).double(), K)
    if case["precision"] != "fp64":
        K = K.float()
    b = _dev(rng.uniform(-1.0, 1.0, n) + np.tile([0.3, 0.0, -1.0], m.n_nodes))
    b[fixed] = 0.0
    return indptr.int(), indices.int(), K, b


def _cantilever(m, rng):
    """Clamp at x = 0 and a tip load that bends the beam by about 0.3% of its length."""
    lo, hi = m.nodes[:, 0].min(), m.nodes[:, 0].max()
    clamp = np.flatnonzero(m.nodes[:, 0] < lo + 1e-9)
    tip = np.flatnonzero(m.nodes[:, 0] > hi - 1e-9)
    fixed = (3 * clamp[:, None] + np.arange(3)).ravel()
    f = np.zeros((m.n_nodes, 3))
    size = m.nodes.max(axis=0) - m.nodes.min(axis=0)
    stiff = 3 * 3e3 * size[1] * size[2] ** 3 / 12 / size[0] ** 3  # tip force per tip displacement
    f[tip] = np.array([0.0, 0.0, -0.0025 * size[0] * stiff * rng.uniform(0.8, 1.2)]) / tip.size
    return fixed, f.ravel()


def prepare(case, seed):
    kind = case["kind"]
    m, u, mu, kappa, rng = _inputs(case, seed)
    st = {"case": case}
    if kind == "pcg":
        st["indptr"], st["indices"], st["K"], st["b"] = _linear_system(case, m, u, mu, kappa, rng)
        st["solver"] = ConjugateGradientSolver(tolerance=1e-12, max_iterations=20000, preconditioner="block-jacobi")
        return st
    if kind == "ecsw":
        Phi, idx, w, u_r = _reduced(case, m, rng)
        st["ev"] = ECSWEvaluator(m.nodes, m.elements, _material(mu, kappa), Phi, idx, w)
        st["u_r"] = _dev(u_r)
        return st
    if kind == "fbar":
        st["asm"], st["u"] = FbarAssembler(m.nodes, m.elements, _material(mu, kappa)), _dev(u.ravel())
        return st
    asm = GPUAssembler(m.nodes, m.elements, _material(mu, kappa), precision=case["precision"])
    st["asm"] = asm
    if kind == "newton":
        fixed, f = _cantilever(m, rng)
        st["solver"] = DeviceNewton(asm, fixed)
        st["f_ext"] = _dev(f)
        return st
    st["u"] = _dev(u.ravel())
    if kind in ("f_k", "tet10", "effective"):
        st["f"], st["k"] = asm.new_f(), asm.new_k()
    elif kind == "f":
        st["f"] = asm.new_f()
    elif kind == "kv":
        st["v"], st["y"] = _dev(rng.normal(size=m.n_dofs)), asm.new_f()
    elif kind == "adjoint":
        st["leaves"] = [_dev(a).requires_grad_(True) for a in (m.nodes, u, mu, kappa)]
        st["w"] = _dev(rng.normal(size=m.n_dofs))
    return st


def _reduced(case, m, rng):
    """Smooth modes, sampled elements and their weights."""
    r, n = case["r"], min(case["n"], m.n_elements)
    s = m.nodes / m.nodes.max()
    Phi = np.zeros((m.n_dofs, r))
    for j in range(r):
        k = rng.uniform(0.5, 4.0, (3, 3))
        Phi[:, j] = np.stack([np.sin(s @ k[i] + rng.uniform(0, 6.28)) for i in range(3)], axis=1).ravel()
    Phi = np.linalg.qr(Phi)[0]
    idx = np.sort(rng.choice(m.n_elements, size=n, replace=False))
    w = rng.uniform(0.5, 2.0, n) * m.n_elements / n
    return Phi, idx, w, 0.01 * m.nodes.max() * rng.normal(size=r)


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "pcg":
        x = torch.zeros_like(state["b"])
        state["solver"].solve_device(state["indptr"], state["indices"], state["K"], state["b"], x, nodal=True)
        return x
    if kind == "ecsw":
        f, K = state["ev"].evaluate_device(state["u_r"])
        return {"f": f, "k": K}
    asm = state["asm"]
    if kind == "fbar":
        f, k = asm.assemble(state["u"])
        return {"f": f, "k": k}
    if kind == "newton":
        return state["solver"].solve(state["f_ext"], n_steps=2).u
    if kind in ("f_k", "tet10"):
        f, k = asm.assemble(state["u"], f_out=state["f"], k_out=state["k"])
        return {"f": f, "k": k}
    if kind == "f":
        return asm.assemble(state["u"], want_k=False, f_out=state["f"])[0]
    if kind == "kv":
        return asm.kv(state["u"], state["v"], y_out=state["y"])
    if kind == "effective":
        f, k = asm.assemble_effective(state["u"], *_effective_coefficients(), f_out=state["f"], k_out=state["k"])
        return {"f": f, "k": k}
    f = internal_force(asm, *state["leaves"])
    gX, gu, gm, gk = torch.autograd.grad(f, state["leaves"], state["w"])
    return {"f": f.detach(), "X": gX, "u": gu, "mu": gm, "kappa": gk}


def work(case):
    kind = case["kind"]
    if kind == "ecsw":
        n, r = case["n"], case["r"]
        return {"bytes": 8 * n * (12 * r + 12 + 1) + 8 * (r * r + 2 * r), "flops": n * (1500 + 24 * r + 2 * 144 * r + 12 * r * r)}
    m = _mesh(case)[0]
    if kind == "tet10":
        m = meshgen.tet4_to_tet10(m)
    el, N = m.elements, m.n_nodes
    E, npe = el.shape
    a, b = np.triu_indices(npe, 1)
    pairs = np.unique(np.minimum(el[:, a], el[:, b]) * N + np.maximum(el[:, a], el[:, b])).size
    nnz = 9 * (N + 2 * pairs)
    s_k = 8 if case["precision"] == "fp64" else 4
    mesh = 4 * npe * E + 24 * N + (16 * E if case["field"] else 0)  # connectivity, coordinates, moduli
    f_flops = 600 * E if npe == 4 else 4 * 1700 * E
    k_flops = 10 * 60 * E if npe == 4 else 4 * 55 * 60 * E
    if kind == "pcg":
        # one iteration's reads and writes (values, one column index per 3x3 block, x, r, z, p, q and the
        # block-Jacobi inverse) for about as many iterations as the condition of the cube asks for
        its = 6 * max(case["nx"], case["ny"], case["nz"])
        return {"bytes": its * (s_k * nnz + 4 * nnz // 9 + 8 * 3 * N * 13), "flops": its * (2 * nnz + 50 * N)}
    if kind == "newton":
        its = 8 * 6 * case["nx"]  # about eight linear steps
        return {"bytes": its * (s_k * nnz + 4 * nnz // 9 + 8 * 3 * N * 13), "flops": its * (2 * nnz + 50 * N)}
    if kind == "f":
        return {"bytes": mesh + 48 * N, "flops": f_flops}
    if kind == "kv":
        return {"bytes": mesh + 72 * N, "flops": f_flops + 200 * E}
    if kind == "adjoint":
        return {"bytes": mesh + 24 * N * 5 + 16 * E, "flops": 2 * f_flops + 600 * E}
    if kind == "fbar":
        # the two-ring matrix: about 65 nodes in a node's two-ring inside a Kuhn box
        cells = np.array([case["nx"], case["ny"], case["nz"]]) + 1.0
        nnz = int(9 * 65 * N * np.prod(1.0 - 1.0 / cells))
        return {"bytes": mesh + 48 * N + 8 * nnz, "flops": 2 * f_flops + k_flops + nnz * 20}
    return {"bytes": mesh + 48 * N + s_k * nnz, "flops": f_flops + k_flops}


# ---------------------------------------------------------------------------- plain float64 evaluation
def _blocks(elements, N):
    """Node-block pattern of ``elements`` (E, npe): sorted pair keys, per node the first block, and the
    block of every (element, a, b)."""
    el = _dev(elements, torch.int64)
    keys, inv = torch.unique((el[:, :, None] * N + el[:, None, :]).reshape(-1), return_inverse=True)
    row = torch.div(keys, N, rounding_mode="floor")
    ptr = torch.zeros(N + 1, dtype=torch.int64, device=el.device)
    ptr[1:] = torch.cumsum(torch.bincount(row, minlength=N), 0)
    return keys, ptr, inv.view(el.shape[0], el.shape[1], el.shape[1])


def _csr_order(blocks, keys, ptr, N):
    """(3 N rows) CSR values, row pointers and columns of 3x3 blocks in the order of ``keys``."""
    row, col = torch.div(keys, N, rounding_mode="floor"), keys % N
    deg = ptr.diff()
    at = 9 * ptr[row] + 3 * (torch.arange(keys.numel(), device=keys.device) - ptr[row])
    out = torch.empty(9 * keys.numel(), dtype=blocks.dtype, device=blocks.device)
    indices = torch.empty_like(out, dtype=torch.int32)
    for k in range(3):
        for j in range(3):
            p = at + 3 * deg[row] * k + j
            out[p] = blocks[:, 3 * k + j]
            indices[p] = (3 * col + j).int()
    indptr = torch.zeros(3 * N + 1, dtype=torch.int64, device=keys.device)
    indptr[1:] = torch.cumsum(torch.repeat_interleave(3 * deg, 3), 0)
    return out, indptr, indices


def _point(l, mu, kappa):
    """P, F, F^-1 and the scalars of the NeoHookean law at displacement gradients ``l``, without
    the cancellation of F^T F - I at small strain."""
    I = torch.eye(3, dtype=l.dtype, device=l.device)
    tr = l.diagonal(dim1=-2, dim2=-1).sum(-1)
    jm1 = tr + 0.5 * (tr * tr - torch.einsum("...ij,...ji->...", l, l)) + torch.linalg.det(l)
    lnj = torch.log1p(jm1)
    phi, beta = mu * torch.exp(-2.0 / 3.0 * lnj), kappa * lnj
    F = I + l
    Fi = torch.linalg.inv(F)
    E = 0.5 * (l + l.transpose(-1, -2) + l.transpose(-1, -2) @ l)
    trE = E.diagonal(dim1=-2, dim2=-1).sum(-1)
    T = 2.0 * phi[..., None, None] * (E - trE[..., None, None] / 3.0 * I) + beta[..., None, None] * I
    return Fi.transpose(-1, -2) @ T, F, Fi, phi, beta, 3.0 + 2.0 * trE


def _shape(X):
    """Gradients (n, 4, 3) and volumes of linear tetrahedra with corners X (n, 4, 3)."""
    D = (X[:, 1:] - X[:, :1]).transpose(1, 2)
    Di = torch.linalg.inv(D)
    return torch.cat([-Di.sum(1, keepdim=True), Di], 1), torch.linalg.det(D) / 6.0


def _k_ab(p, q, g, a, b, A, hb, c, phi):
    """The (a, b) blocks (n, 9): A p_a p_b + hb p_b p_a + c (p_a q_b + q_a p_b) + phi g_a.g_b I."""
    out = (A[:, None, None] * p[:, a, :, None] * p[:, b, None, :] + hb[:, None, None] * p[:, b, :, None] * p[:, a, None, :]
           + c[:, None, None] * (p[:, a, :, None] * q[:, b, None, :] + q[:, a, :, None] * p[:, b, None, :]))
    out.diagonal(dim1=1, dim2=2).add_((phi * (g[:, a] * g[:, b]).sum(-1))[:, None])
    return out.reshape(-1, 9)


def _add(acc, at, v):
    # sort-based accumulation: the same bits for the same inputs
    acc.index_put_((at,), v, accumulate=True)


def _tet4_assemble(m, u, mu, kappa, c_t=1.0, c_m=0.0, c_0=0.0, want_k=True, step=400_000):
    N, E = m.n_nodes, m.n_elements
    X, U, el = _dev(m.nodes), _dev(u), _dev(m.elements, torch.int64)
    mu_t, ka_t = (_dev(a) if np.ndim(a) else torch.full((E,), float(a), dtype=torch.float64, device=X.device) for a in (mu, kappa))
    f = torch.zeros(N, 3, dtype=torch.float64, device=X.device)
    keys = ptr = None
    if want_k:
        keys, ptr, inv = _blocks(m.elements, N)
        K = torch.zeros(keys.numel(), 9, dtype=torch.float64, device=X.device)
    for e0 in range(0, E, step):
        e = slice(e0, min(E, e0 + step))
        g, V = _shape(X[el[e]])
        Ue = U[el[e]]
        l = torch.einsum("nbi,nbj->nij", Ue[:, 1:] - Ue[:, :1], g[:, 1:])
        P, F, Fi, phi, beta, I1 = _point(l, mu_t[e], ka_t[e])
        for a in range(4):
            _add(f, el[e, a], V[:, None] * torch.einsum("nij,nj->ni", P, g[:, a]))
        if not want_k:
            continue
        p = torch.einsum("nji,naj->nai", Fi, g)
        q = torch.einsum("nij,naj->nai", F, g)
        w = c_t * V
        coef = (w * (ka_t[e] + 2.0 / 9.0 * phi * I1), w * (phi * I1 / 3.0 - beta), -2.0 / 3.0 * w * phi, w * phi)
        zero = torch.zeros_like(V)
        lin = (c_0 * V * (ka_t[e] - 2.0 / 3.0 * mu_t[e]), c_0 * V * mu_t[e], zero, c_0 * V * mu_t[e])
        for a in range(4):
            for b in range(4):
                v = _k_ab(p, q, g, a, b, *coef)
                if c_0:
                    v = v + _k_ab(g, g, g, a, b, *lin)
                if c_m:
                    v[:, 0::4] += (c_m * 1000.0 * V.abs() / 20.0 * (2.0 if a == b else 1.0))[:, None]
                _add(K, inv[e, a, b], v)
    if not want_k:
        return f.reshape(-1), None, None, None, None
    k, indptr, indices = _csr_order(K, keys, ptr, N)
    return f.reshape(-1), k, indptr, indices.long(), (keys, ptr)


def _tet4_kv(m, u, v, mu, kappa, step=400_000):
    N, E = m.n_nodes, m.n_elements
    X, U, el, Vv = _dev(m.nodes), _dev(u), _dev(m.elements, torch.int64), _dev(v).view(-1, 3)
    mu_t, ka_t = (_dev(a) if np.ndim(a) else torch.full((E,), float(a), dtype=torch.float64, device=X.device) for a in (mu, kappa))
    y = torch.zeros(N, 3, dtype=torch.float64, device=X.device)
    for e0 in range(0, E, step):
        e = slice(e0, min(E, e0 + step))
        g, V = _shape(X[el[e]])
        Ue, Ve = U[el[e]], Vv[el[e]]
        l = torch.einsum("nbi,nbj->nij", Ue[:, 1:] - Ue[:, :1], g[:, 1:])
        _, F, Fi, phi, beta, I1 = _point(l, mu_t[e], ka_t[e])
        p, q = torch.einsum("nji,naj->nai", Fi, g), torch.einsum("nij,naj->nai", F, g)
        coef = (V * (ka_t[e] + 2.0 / 9.0 * phi * I1), V * (phi * I1 / 3.0 - beta), -2.0 / 3.0 * V * phi, V * phi)
        for a in range(4):
            t = sum(torch.einsum("nij,nj->ni", _k_ab(p, q, g, a, b, *coef).view(-1, 3, 3), Ve[:, b]) for b in range(4))
            _add(y, el[e, a], t)
    return y.reshape(-1)


def _tet10_assemble(m, u, mu, kappa, step=20_000):
    N, E = m.n_nodes, m.n_elements
    X, U, el = _dev(m.nodes), _dev(u), _dev(m.elements, torch.int64)
    mu_t, ka_t = (_dev(a) if np.ndim(a) else torch.full((E,), float(a), dtype=torch.float64, device=X.device) for a in (mu, kappa))
    keys, ptr, inv = _blocks(m.elements, N)
    K = torch.zeros(keys.numel(), 9, dtype=torch.float64, device=X.device)
    f = torch.zeros(N, 3, dtype=torch.float64, device=X.device)
    a5, b5 = (5 - math.sqrt(5.0)) / 20, (5 + 3 * math.sqrt(5.0)) / 20
    edges = ((0, 1), (1, 2), (2, 0), (0, 3), (1, 3), (2, 3))
    dL = np.array([[-1.0, -1, -1], [1, 0, 0], [0, 1, 0], [0, 0, 1]])
    rule = []
    for qp in range(4):
        L = np.full(4, a5)
        L[qp] = b5
        rule.append(_dev(np.concatenate([(4 * L - 1)[:, None] * dL, [4 * (L[i] * dL[j] + L[j] * dL[i]) for i, j in edges]])))
    for e0 in range(0, E, step):
        e = slice(e0, min(E, e0 + step))
        Xe, Ue = X[el[e]], U[el[e]]
        points = []
        for dN in rule:
            Jm = torch.einsum("nai,aj->nij", Xe, dN)
            g = torch.einsum("aj,njk->nak", dN, torch.linalg.inv(Jm))
            V = torch.linalg.det(Jm) / 24.0
            l = torch.einsum("nbi,nbj->nij", Ue[:, 1:] - Ue[:, :1], g[:, 1:])
            P, F, Fi, phi, beta, I1 = _point(l, mu_t[e], ka_t[e])
            p, q = torch.einsum("nji,naj->nai", Fi, g), torch.einsum("nij,naj->nai", F, g)
            points.append((p, q, g, V * (ka_t[e] + 2.0 / 9.0 * phi * I1), V * (phi * I1 / 3.0 - beta), -2.0 / 3.0 * V * phi,
                           V * phi, V[:, None, None] * P))
        for a in range(10):
            _add(f, el[e, a], sum(torch.einsum("nij,nj->ni", P, g[:, a]) for _, _, g, _, _, _, _, P in points))
            for b in range(10):
                _add(K, inv[e, a, b], sum(_k_ab(p, q, g, a, b, A, hb, c, ph) for p, q, g, A, hb, c, ph, _ in points))
    return f.reshape(-1), _csr_order(K, keys, ptr, N)[0]


def _cg(indptr, indices, K, b, free=None, tol=1e-15, most=6000):
    """Block-Jacobi conjugate gradients, then one step of refinement, in float64."""
    n = b.numel()
    K = K.double()
    A = torch.sparse_csr_tensor(indptr.long(), indices.long(), K, (n, n))
    rows = torch.repeat_interleave(torch.arange(n, device=b.device), indptr.long().diff())
    at = rows // 3 == indices // 3
    D = torch.zeros(n // 3, 3, 3, dtype=torch.float64, device=b.device)
    D[rows[at] // 3, rows[at] % 3, indices[at].long() % 3] = K[at]
    Di = torch.linalg.inv(D)
    prec = lambda r: torch.einsum("nij,nj->ni", Di, r.view(-1, 3)).reshape(-1)  # noqa: E731
    x = torch.zeros_like(b)
    for _ in range(2):
        r = b - A @ x
        z = prec(r)
        p, rz, stop = z.clone(), r @ z, tol * float(b.norm())
        for it in range(most):
            Ap = A @ p
            al = rz / (p @ Ap)
            x, r = x + al * p, r - al * Ap
            if it % 20 == 19 and float(r.norm()) < stop:
                break
            z = prec(r)
            rz, old = r @ z, rz
            p = z + (rz / old) * p
    return x


def _newton_exact(m, mu, kappa, fixed, f_ext):
    free = torch.ones(m.n_dofs, dtype=torch.bool, device=_device())
    free[_dev(fixed, torch.int64)] = False
    u = torch.zeros(m.n_dofs, dtype=torch.float64, device=_device())
    for lam in (0.5, 1.0):
        for _ in range(8):
            f, K, indptr, indices, _ = _tet4_assemble(m, u.view(-1, 3).cpu().numpy(), mu, kappa)
            r = torch.where(free, lam * _dev(f_ext) - f, torch.zeros_like(f))
            if float(r.norm()) < 1e-12 * float(np.linalg.norm(f_ext)):
                break
            rows = torch.repeat_interleave(torch.arange(m.n_dofs, device=K.device), indptr.diff())
            K = torch.where(free[rows] & free[indices], K, (rows == indices).double())
            u = u + _cg(indptr, indices, K, r, tol=1e-10, most=3000)
    return u


def _fbar_assemble(m, u, mu, kappa):
    """Nodal F-bar: f and K_dev + K_vol on the two-ring pattern."""
    N, E = m.n_nodes, m.n_elements
    X, U, el = _dev(m.nodes), _dev(u), _dev(m.elements, torch.int64)
    g, V = _shape(X[el])
    I = torch.eye(3, dtype=torch.float64, device=X.device)
    Ue = U[el]
    F = I + torch.einsum("nbi,nbj->nij", Ue[:, 1:] - Ue[:, :1], g[:, 1:])
    J = torch.linalg.det(F)
    v0, v = (torch.zeros(N, dtype=torch.float64, device=X.device) for _ in range(2))
    for a in range(4):
        _add(v0, el[:, a], 0.25 * V)
        _add(v, el[:, a], 0.25 * V * J)
    jbar = (v / v0)[el].mean(1)
    ratio = (jbar / J) ** (1.0 / 3.0)
    Fb = ratio[:, None, None] * F
    C = Fb.transpose(1, 2) @ Fb
    Ci = torch.linalg.inv(C)
    I1, lnj = C.diagonal(dim1=1, dim2=2).sum(1), torch.log(jbar)
    fac = mu * jbar ** (-2.0 / 3.0)
    S = fac[:, None, None] * (I - I1[:, None, None] / 3.0 * Ci) + (kappa * lnj)[:, None, None] * Ci
    # Voigt order xx yy zz xy yz zx
    vi, vj = [0, 1, 2, 0, 1, 2], [0, 1, 2, 1, 2, 0]
    one = torch.tensor([1.0, 1, 1, 0, 0, 0], dtype=torch.float64, device=X.device)
    cv = Ci[:, vi, vj]
    ii = 0.5 * (Ci[:, vi][:, :, vi] * Ci[:, vj][:, :, vj] + Ci[:, vi][:, :, vj] * Ci[:, vj][:, :, vi])
    oo = cv[:, :, None] * cv[:, None, :]
    Cv = (kappa * oo - (2.0 * kappa * lnj)[:, None, None] * ii + (2.0 / 9.0 * fac * I1)[:, None, None] * oo
          + (2.0 / 3.0 * fac * I1)[:, None, None] * ii
          - (2.0 / 3.0 * fac)[:, None, None] * (cv[:, :, None] * one + one[:, None] * cv[:, None, :]))
    Cd = Cv - kappa * one[:, None] * one
    B = torch.zeros(E, 6, 12, dtype=torch.float64, device=X.device)
    for b in range(4):
        for k in range(3):
            for s in range(6):
                i, j = vi[s], vj[s]
                B[:, s, 3 * b + k] = F[:, k, i] * g[:, b, j] if i == j else F[:, k, i] * g[:, b, j] + F[:, k, j] * g[:, b, i]
    div = B[:, 0] + B[:, 1] + B[:, 2]
    vol = one[:, None] * div[:, None, :] / 3.0
    r2 = (ratio ** 2)[:, None, None]
    Bd = r2 * (B - vol)
    fe = V[:, None] * torch.einsum("nsa,ns->na", Bd + vol, S[:, vi, vj])
    Ke = V[:, None, None] * (Bd.transpose(1, 2) @ Cd @ Bd)
    geo = V[:, None, None] * (g @ S @ g.transpose(1, 2))
    f = torch.zeros(N, 3, dtype=torch.float64, device=X.device)
    # one-ring vectors g_a[b]
    keys1, ptr1, inv1 = _blocks(m.elements, N)
    ga = torch.zeros(keys1.numel(), 3, dtype=torch.float64, device=X.device)
    for a in range(4):
        _add(f, el[:, a], fe[:, 3 * a:3 * a + 3])
        w = 0.25 * V * J / v0[el[:, a]]
        for b in range(4):
            _add(ga, inv1[:, a, b], w[:, None] * div[:, 3 * b:3 * b + 3])
    # every two nodes b, c of a node's star
    deg, node = ptr1.diff(), torch.div(keys1, N, rounding_mode="floor")
    first = torch.repeat_interleave(torch.arange(keys1.numel(), device=X.device), deg[node])
    second = torch.arange(first.numel(), device=X.device) - torch.repeat_interleave(
        torch.cumsum(deg[node], 0) - deg[node], deg[node]) + ptr1[node[first]]
    keys2, inv2 = torch.unique((keys1[first] % N) * N + keys1[second] % N, return_inverse=True)
    K = torch.zeros(keys2.numel(), 9, dtype=torch.float64, device=X.device)
    _add(K, inv2, ((kappa * v0[node[first]])[:, None, None] * ga[first][:, :, None] * ga[second][:, None, :]).reshape(-1, 9))
    for a in range(4):
        for b in range(4):
            v9 = Ke[:, 3 * a:3 * a + 3, 3 * b:3 * b + 3] + geo[:, a, b, None, None] * I
            _add(K, torch.searchsorted(keys2, el[:, a] * N + el[:, b]), v9.reshape(-1, 9))
    ptr2 = torch.zeros(N + 1, dtype=torch.int64, device=X.device)
    ptr2[1:] = torch.cumsum(torch.bincount(torch.div(keys2, N, rounding_mode="floor"), minlength=N), 0)
    return f.reshape(-1), _csr_order(K, keys2, ptr2, N)[0]


def _adjoint_exact(m, u, mu, kappa, w):
    """f and the gradients of w.f by automatic differentiation."""
    leaves = [_dev(a).requires_grad_(True) for a in (m.nodes, u, mu, kappa)]
    X, U, mu_t, ka_t = leaves
    el = _dev(m.elements, torch.int64)
    g, V = _shape(X[el])
    Ue = U[el]
    P = _point(torch.einsum("nbi,nbj->nij", Ue[:, 1:] - Ue[:, :1], g[:, 1:]), mu_t, ka_t)[0]
    fe = V[:, None, None] * torch.einsum("nij,naj->nai", P, g)
    f = torch.zeros_like(X).index_put((el.reshape(-1),), fe.reshape(-1, 3), accumulate=True).reshape(-1)
    gX, gu, gm, gk = torch.autograd.grad(f, leaves, _dev(w))
    return {"f": f.detach(), "X": gX, "u": gu, "mu": gm, "kappa": gk}


def _ecsw_exact(m, mu, kappa, Phi, idx, w, u_r):
    el = m.elements[idx]
    n, r = el.shape[0], Phi.shape[1]
    P = _dev(Phi[(3 * el[:, :, None] + np.arange(3)).reshape(n, 12)])
    mu_t, ka_t = (_dev(a[idx]) if np.ndim(a) else torch.full((n,), float(a), dtype=torch.float64, device=P.device)
                  for a in (mu, kappa))
    g, V = _shape(_dev(m.nodes[el]))
    Ue = (P @ _dev(u_r)).view(n, 4, 3)
    Pk, F, Fi, phi, beta, I1 = _point(torch.einsum("nbi,nbj->nij", Ue[:, 1:] - Ue[:, :1], g[:, 1:]), mu_t, ka_t)
    p, q = torch.einsum("nji,naj->nai", Fi, g), torch.einsum("nij,naj->nai", F, g)
    coef = (V * (ka_t + 2.0 / 9.0 * phi * I1), V * (phi * I1 / 3.0 - beta), -2.0 / 3.0 * V * phi, V * phi)
    Ke = torch.zeros(n, 12, 12, dtype=torch.float64, device=P.device)
    for a in range(4):
        for b in range(4):
            Ke[:, 3 * a:3 * a + 3, 3 * b:3 * b + 3] = _k_ab(p, q, g, a, b, *coef).view(n, 3, 3)
    fe = (V[:, None, None] * torch.einsum("nij,naj->nai", Pk, g)).view(n, 12)
    wt = _dev(w)
    K = torch.einsum("nai,naj->ij", P, wt[:, None, None] * (Ke @ P))
    return {"f": torch.einsum("nai,na->i", P, wt[:, None] * fe), "k": 0.5 * (K + K.T)}


def exact(case, seed):
    kind = case["kind"]
    m, u, mu, kappa, rng = _inputs(case, seed)
    if kind == "pcg":
        return _cg(*_linear_system(case, m, u, mu, kappa, rng))
    if kind == "ecsw":
        return _ecsw_exact(m, mu, kappa, *_reduced(case, m, rng))
    if kind == "fbar":
        f, k = _fbar_assemble(m, u, mu, kappa)
        return {"f": f, "k": k}
    if kind == "newton":
        return _newton_exact(m, mu, kappa, *_cantilever(m, rng))
    if kind == "kv":
        return _tet4_kv(m, u, rng.normal(size=m.n_dofs), mu, kappa)
    if kind == "adjoint":
        return _adjoint_exact(m, u, mu, kappa, rng.normal(size=m.n_dofs))
    if kind == "tet10":
        f, k = _tet10_assemble(m, u, mu, kappa)
        return {"f": f, "k": k}
    if kind == "f":
        return _tet4_assemble(m, u, mu, kappa, want_k=False)[0]
    c = _effective_coefficients() if kind == "effective" else (1.0, 0.0, 0.0)
    f, k, _, _, _ = _tet4_assemble(m, u, mu, kappa, *c)
    return {"f": f, "k": k}
