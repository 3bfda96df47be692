"""One-launch CG solves that the device refuses (GPU): the next form solves them.

A small library in front of libcudart (LD_PRELOAD, in a child process) answers chosen calls with
an error code and passes every other call on, so nothing that is refused runs.
"""
from __future__ import annotations

import os
import subprocess
import sys
import textwrap

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

FRONT = r"""
#include <cuda_runtime_api.h>
#include <dlfcn.h>
extern "C" {
int front_refuse = 0;   // bit 0: cooperative launches, bit 1: cluster launches
int front_refused = 0;  // how many were
int front_coop = 0;     // cooperative launches
int front_grid = 0;     // blocks of the last cluster launch
int front_narrow = 0;   // the n-th kernel asked for its clusters has none of 16 blocks
static cudaError_t pending = cudaSuccess;
static void* real(const char* name) {
  static void* h = dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD);
  return dlsym(h, name);
}
static cudaError_t refuse() { ++front_refused; return pending = cudaErrorCooperativeLaunchTooLarge; }
cudaError_t cudaLaunchCooperativeKernel(const void* f, dim3 g, dim3 b, void** a, size_t m, cudaStream_t s) {
  if (front_refuse & 1) return refuse();
  ++front_coop;
  return ((cudaError_t(*)(const void*, dim3, dim3, void**, size_t, cudaStream_t))real("cudaLaunchCooperativeKernel"))(f, g, b, a, m, s);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** a) {
  if (c->numAttrs == 1 && c->attrs[0].id == cudaLaunchAttributeClusterDimension) {
    if (front_refuse & 2) return refuse();
    front_grid = c->gridDim.x;
  }
  return ((cudaError_t(*)(const cudaLaunchConfig_t*, const void*, void**))real("cudaLaunchKernelExC"))(c, f, a);
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void* f, const cudaLaunchConfig_t* c) {
  static const void* asked[64];
  int k = 0;
  while (k < 63 && asked[k] && asked[k] != f) ++k;
  asked[k] = f;
  if (k + 1 == front_narrow && c->gridDim.x == 16) { *n = 0; return cudaSuccess; }
  return ((cudaError_t(*)(int*, const void*, const cudaLaunchConfig_t*))real("cudaOccupancyMaxActiveClusters"))(n, f, c);
}
cudaError_t cudaGetLastError(void) {
  cudaError_t e = pending;
  pending = cudaSuccess;
  return e != cudaSuccess ? e : ((cudaError_t(*)(void))real("cudaGetLastError"))();
}
}
"""

CHILD = """
    import ctypes, sys
    import numpy as np, torch
    sys.path[:0] = [{root!r}, {root!r} + "/tests"]
    from test_pcg_resident_gpu import _solve, _system
    front = ctypes.CDLL({front!r})
    word = lambda name: ctypes.c_int.in_dll(front, name)

    def solve(n, dtype=np.float64):
        A, b = _system(n, True, seed=n)
        A.data = A.data.astype(np.float32).astype(np.float64)
        x, r = _solve(A, b, "block-jacobi", True, dtype)
        assert r.converged and r.iterations <= 60
        assert np.linalg.norm(b - A @ x) <= 1.01e-10 * np.linalg.norm(b)
        return x
"""


def _child(tmp_path, body):
    front = tmp_path / "front.so"
    (tmp_path / "front.cpp").write_text(FRONT)
    subprocess.run(["g++", "-shared", "-fPIC", "-O1", "-I/usr/local/cuda/include", "-o", str(front),
                    str(tmp_path / "front.cpp"), "-ldl"], check=True)
    code = textwrap.dedent(CHILD).format(root=ROOT, front=str(front)) + textwrap.dedent(body)
    r = subprocess.run([sys.executable, "-c", code], env={**os.environ, "LD_PRELOAD": str(front)}, cwd=ROOT,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]


def test_the_next_form_solves_what_is_refused(tmp_path):
    _child(tmp_path, """
    for n in (3000, 30000):  # cluster form, grid form
        want = solve(n)
        for bits, times in ((1, n > 6144), (2, n <= 6144), (3, 1 + (n <= 6144))):
            word("front_refuse").value = bits
            word("front_refused").value = 0
            x = solve(n)
            word("front_refuse").value = 0
            assert word("front_refused").value == times, (n, bits, word("front_refused").value)
            # two residuals of 1.01e-10 ||b||, condition below 10
            assert np.linalg.norm(x - want) <= 2.1e-9 * np.linalg.norm(want)
        assert np.array_equal(solve(n), want)
    """)


def test_each_kernel_keeps_its_own_cluster_size(tmp_path):
    _child(tmp_path, """
    word("front_narrow").value = 2  # the second kernel, FP32 values, gets 8 blocks
    for dtype, blocks in ((np.float64, 16), (np.float32, 8), (np.float64, 16), (np.float32, 8)):
        solve(3000, dtype)
        assert word("front_grid").value == blocks, (dtype, word("front_grid").value)
    """)


@pytest.mark.parametrize("precond,unit", [("block-jacobi", 176), ("jacobi", 128)])
def test_large_systems_leave_the_gathers_their_cache(tmp_path, precond, unit):
    # one block per SM, 194 KB of state: the last system that one launch takes and the next one
    _child(tmp_path, f"""
    from psierra_b200.solver import ConjugateGradientSolver
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    last = 3 * sms * (194 * 1024 // {unit})
    for n, launches in ((last, 1), (last + 3, 0)):
        # 3 x 3 blocks 4 I and nothing else: solved in one iteration
        t = lambda a, d: torch.from_numpy(np.ascontiguousarray(a, dtype=d)).cuda()
        rows = np.arange(n)
        indices = 3 * (rows // 3)[:, None] + np.arange(3)
        values = 4.0 * (indices == rows[:, None])
        b, x = torch.ones(n, dtype=torch.float64, device="cuda"), torch.zeros(n, dtype=torch.float64, device="cuda")
        word("front_coop").value = 0
        r = ConjugateGradientSolver(tolerance=1e-10, preconditioner="{precond}").solve_device(
            t(3 * np.arange(n + 1), np.int32), t(indices, np.int32), t(values, np.float64), b, x, nodal=True)
        assert r.converged and torch.equal(x, 0.25 * b)
        assert word("front_coop").value == launches, (n, word("front_coop").value)
    """)
